"""Resident solves of quadratic 3D elements: rows of up to 125 neighbours, the
longest first in the numbering, in shared memory, partly there and read from
global memory with and without a halo (few CTAs), against the reference's
displacements."""

import pytest

from test_gpu_coarse import elastic, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["el_hexa20", "el_hexa27", "el_prism18", "el_tetra10"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ctas", [1, 2, 5, 152])
def test_matches_reference(golden, monkeypatch, case, precision, ctas):
    monkeypatch.setenv("GFEA_RESIDENT_CTAS", str(ctas))
    g = golden(case)
    simu = elastic(g, precision=precision)
    u = simu.Solve()
    assert simu.last_solve.status == 0
    assert simu.last_solve.rel_residual <= max(1e-12, simu.last_solve.floor_rel)
    assert rel_err(u, g["u"]) <= 1e-8


@pytest.mark.parametrize("precision,ctas", [("fp64", 5), ("fp64", 40), ("mixed", 3)])
def test_rows_and_halo_beyond_shared_memory(monkeypatch, precision, ctas):
    """The corner nodes' CTAs hold neither their rows nor the part of p that
    they read: the same solution as with everything in shared memory."""
    import numpy as np

    from easyfea_gb300 import Models
    from easyfea_gb300 import mesh as gmesh
    from easyfea_gb300 import simulations as Simulations

    m = gmesh.Mesh_Box(gmesh.ElemType.HEXA27, 100.0, 20.0, 20.0, 12, 4, 4)
    out = []
    for c in (ctas, 152):
        monkeypatch.setenv("GFEA_RESIDENT_CTAS", str(c))
        simu = Simulations.Elastic(m, Models.Elastic.Isotropic(3, E=210000.0, v=0.3))
        simu.precision = precision
        simu.add_dirichlet(m.Nodes_Conditions(lambda x, y, z: x == 0), [0.0] * 3, ["x", "y", "z"])
        simu.add_dirichlet(np.arange(7, m.Nn, 97), [0.01], ["y"])
        simu.add_surfLoad(m.Nodes_Conditions(lambda x, y, z: x == 100.0), [-1.0], ["z"])
        out.append(simu.Solve())
        assert simu.last_solve.status == 0
    assert np.abs(out[0] - out[1]).max() <= 1e-9 * np.abs(out[1]).max()
