"""The isotropic FP64 stiffness kernel (Gauss points per lane) against the
general Kelvin-Mandel kernel on every element it serves: warps with a
remainder of elements, one element alone, distorted elements, homogeneous and
per-element moduli."""

import numpy as np
import pytest

from helpers import row_scaled_err
from test_gpu_isotropic import assemble

pytestmark = pytest.mark.gpu

ELEMENTS = {"TRI3": 2, "QUAD4": 2, "QUAD9": 2, "TRI6": 2, "QUAD8": 2, "TRI10": 2,
            "HEXA8": 3, "TETRA4": 3, "TETRA10": 3, "PRISM6": 3}


@pytest.mark.parametrize("elem", sorted(ELEMENTS))
@pytest.mark.parametrize("counts", [(1, 1, 1), (7, 3, 3)])
@pytest.mark.parametrize("hetero", [False, True])
def test_equals_the_general_kernel(elem, counts, hetero):
    import scipy.sparse as sp
    import torch

    from easyfea_gb300 import Models
    from easyfea_gb300 import mesh as gmesh
    from easyfea_gb300 import simulations as Simulations

    dim = ELEMENTS[elem]
    rng = np.random.default_rng(len(elem) + counts[0])
    if dim == 2:
        m = gmesh.Mesh_Rect(gmesh.ElemType(elem), 12.0, 4.0, *counts[:2])
        h = min(12.0 / counts[0], 4.0 / counts[1])
    else:
        m = gmesh.Mesh_Box(gmesh.ElemType(elem), 12.0, 4.0, 5.0, *counts)
        h = min(12.0 / counts[0], 4.0 / counts[1])
    m.coord[:, :dim] += rng.uniform(-0.04, 0.04, (m.Nn, dim)) * h
    law = dict(v=0.3, planeStress=dim == 2)
    E = rng.uniform(0.5, 2.0, m.Ne) * 210000.0 if hetero else 210000.0
    simu = Simulations.Elastic(m, Models.Elastic.Isotropic(dim, E=E, **law))
    dev = torch.device("cuda", 0)
    ref = np.ascontiguousarray(Models.Elastic.Isotropic(dim, E=1.0 if hetero else E, **law).C)
    lame = Simulations.isotropic_lame(ref)
    if hetero:
        general = assemble(simu, torch.as_tensor(np.concatenate([ref.ravel(), E]), device=dev), 2)
        iso = assemble(simu, torch.as_tensor(np.concatenate([lame, E]), device=dev), 4)
    else:
        general = assemble(simu, torch.as_tensor(ref, device=dev), 0)
        iso = assemble(simu, torch.as_tensor(lame, device=dev), 3)
    indptr, indices = (t.cpu().numpy() for t in simu.dmesh.pattern(dim))
    K = [sp.csr_matrix((v, indices, indptr), shape=(dim * m.Nn,) * 2) for v in (general, iso)]
    # the sums of both kernels, re-associated: a few dozen FP64 roundings per entry
    assert row_scaled_err(K[1], K[0]) <= 1e-13
    assert abs(K[1] - K[1].T).max() <= 1e-13 * abs(K[1]).max()
