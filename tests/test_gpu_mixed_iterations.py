"""The FP32 iteration keeps the conjugacy of its directions over the reliable
updates: it needs about as many iterations as the FP64 one, whose residual
never drifts.  Systems whose first update finds a drift as large as the
iterated residual itself."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elem,counts", [("TETRA10", (12, 4, 4)), ("HEXA27", (15, 5, 5)), ("HEXA8", (50, 15, 15)),
                                         ("QUAD8", (20, 6))])
def test_mixed_iterations_stay_near_fp64(elem, counts):
    from easyfea_gb300 import Models
    from easyfea_gb300 import mesh as gmesh
    from easyfea_gb300 import simulations as Simulations

    dim = len(counts)
    make = gmesh.Mesh_Rect if dim == 2 else gmesh.Mesh_Box
    m = make(gmesh.ElemType(elem), *((100.0, 20.0, 20.0)[:dim]), *counts)
    unknowns = ["x", "y", "z"][:dim]
    its = {}
    for precision in ("fp64", "mixed"):
        simu = Simulations.Elastic(m, Models.Elastic.Isotropic(dim, E=210000.0, v=0.3))
        simu.precision = precision
        simu.add_dirichlet(m.Nodes_Conditions(lambda x, y, z: x == 0), [0.0] * dim, unknowns)
        simu.add_surfLoad(m.Nodes_Conditions(lambda x, y, z: x == 100.0), [-1.0], [unknowns[-1]])
        simu.Solve()
        assert simu.last_solve.status == 0
        its[precision] = simu.last_solve.iterations
    # each of five updates costs the FP32 iteration a few directions at most
    assert its["mixed"] <= 1.25 * its["fp64"], its
