"""The kernels that take a Gauss point per lane (damage system, degraded
stiffness, post-processing) against the oracle on every element they serve:
one element alone, blocks and warps with a remainder of elements, distorted
elements, with and without a committed History field."""

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from helpers import row_scaled_err
from oracle import fem
from oracle.simulate import OracleMesh, PhaseFieldOracle

pytestmark = pytest.mark.gpu

ELEMENTS = {"TRI3": 2, "QUAD4": 2, "QUAD9": 2, "TRI6": 2, "QUAD8": 2, "TRI10": 2,
            "HEXA8": 3, "TETRA4": 3, "TETRA10": 3, "PRISM6": 3}


def make_mesh(elem, counts, rng):
    from easyfea_gb300 import mesh as gmesh

    dim = ELEMENTS[elem]
    if dim == 2:
        m = gmesh.Mesh_Rect(gmesh.ElemType(elem), 3.0, 1.0, *counts[:2])
    else:
        m = gmesh.Mesh_Box(gmesh.ElemType(elem), 3.0, 1.0, 1.5, *counts)
    h = min(3.0 / counts[0], 1.0 / counts[1])
    m.coord[:, :dim] += rng.uniform(-0.03, 0.03, (m.Nn, dim)) * h
    return m


def state(m, scale):
    """A displacement whose strain has distinct principal values everywhere
    (a spectral split is ill conditioned where two of them meet): a constant
    gradient and a smooth tenth of it."""
    dim = m.dim
    G = np.array([[1.0, 0.2, -0.1], [0.3, -0.7, 0.15], [0.1, -0.05, 0.3]])[:dim, :dim]
    x = m.coord[:, :dim]
    return (scale * (x @ G.T + 0.03 * np.sin(x @ G.T + 0.4))).ravel()


@pytest.mark.parametrize("elem", sorted(ELEMENTS))
@pytest.mark.parametrize("counts", [(1, 1, 1), (7, 3, 3)])
@pytest.mark.parametrize("split, regu", [("Amor", "AT1"), ("Miehe", "AT2")])
def test_phase_field_systems(elem, counts, split, regu):
    from easyfea_gb300 import Models
    from easyfea_gb300 import simulations as Simulations

    rng = np.random.default_rng(len(elem) + counts[0])
    m = make_mesh(elem, counts, rng)
    dim = m.dim
    mat = Models.Elastic.Isotropic(dim, E=210e3, v=0.3, planeStress=False, thickness=0.7)
    simu = Simulations.PhaseField(m, Models.PhaseField(mat, split, regu, 2.7, 0.2))
    pf = PhaseFieldOracle(OracleMesh.from_mesh(m), 210e3, 0.3, False, 0.7, split, regu, 2.7, 0.2)
    pf.d = rng.uniform(0.0, 0.9, m.Nn)
    for scale in (2e-3, 1.5e-3):  # the second state lies under the committed History
        pf.u = state(m, scale)
        simu.u_device.copy_(torch.as_tensor(pf.u))
        simu.d_device.copy_(torch.as_tensor(pf.d))
        simu.Need_Update()
        pf.damage_system()
        pf.elastic_system()
        Kd, _, _, Fd = simu.Get_K_C_M_F("damage")
        assert row_scaled_err(sp.csr_matrix(Kd), sp.csr_matrix(pf.Kd)) <= 1e-12
        F = np.asarray(pf.Fd).ravel()
        np.testing.assert_allclose(np.asarray(Fd.todense()).ravel(), F, rtol=1e-10, atol=1e-12 * np.abs(F).max())
        H = simu.psiP_device.cpu().numpy().reshape(pf.psiP.shape)
        np.testing.assert_allclose(H, pf.psiP, rtol=1e-10, atol=1e-12 * np.abs(pf.psiP).max())
        Ku = simu.Get_K_C_M_F("elastic")[0]
        # the 3D spectral projectors round with the inverse of the eigenvalue gaps
        assert row_scaled_err(sp.csr_matrix(Ku), sp.csr_matrix(pf.Ku)) <= (5e-12 if dim == 3 else 1e-12)
        simu.Save_Iter()
        pf.H_old = pf.psiP


@pytest.mark.parametrize("elem", sorted(ELEMENTS))
@pytest.mark.parametrize("counts", [(1, 1, 1), (7, 3, 3)])
def test_elastic_fields(elem, counts):
    from easyfea_gb300 import Models
    from easyfea_gb300 import simulations as Simulations

    rng = np.random.default_rng(len(elem) + counts[0])
    m = make_mesh(elem, counts, rng)
    simu = Simulations.Elastic(m, Models.Elastic.Isotropic(m.dim, E=70000.0, v=0.33, planeStress=True, thickness=0.5))
    u = 1e-3 * rng.standard_normal(m.Nn * m.dim)
    simu._Set_solutions("elastic", u)
    C = fem.isotropic_C(70000.0, 0.33, m.dim, True)
    g = m.groupElem
    for r, nv in (("Svm", True), ("Strain", False), ("Stress", True), ("Wdef_e", False)):
        thickness = 0.5 if m.dim == 2 else 1.0  # a 3D law has none
        ref = np.asarray(fem.elastic_result(elem, m.coord, g.connect, u, C, r, thickness, nv), float)
        out = np.asarray(simu.Result(r, nodeValues=nv), float)
        # means of Gauss-point values in another summation order: a few ulps of the largest
        assert np.abs(out - ref).max() <= 1e-12 * np.abs(ref).max(), r
