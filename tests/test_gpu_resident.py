"""The resident PCG (one cooperative launch for a whole solve) against direct
solves and the reference's displacements, over its branches: one CTA, few,
more than a warp's worth and one per SM; rows of the operator in shared
memory, partly there and read from global memory; halos of neighbours and
neighbours read one by one; ragged node degrees; with and without the coarse
level; known DOFs everywhere in a CTA's range.  GFEA_RESIDENT_CTAS bounds the
number of CTAs, so that small systems give large ones."""

import ctypes

import numpy as np
import pytest

from test_gpu_coarse import elastic, rel_err
from test_gpu_staged import hub_graph, solve, spd_values

pytestmark = pytest.mark.gpu


def direct(A, b, known, xk):
    import scipy.sparse.linalg as spla

    u = ~known
    rhs = b[u] - A[u][:, known] @ xk[known]
    Auu = A[u][:, u].tocsc()
    return u, rhs, Auu, spla.spsolve(Auu, rhs)


@pytest.mark.parametrize("ctas", [1, 2, 33, 152])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("D", [1, 2, 3])
def test_ragged_graph(monkeypatch, D, precision, ctas):
    """Hub nodes next to nodes of five neighbours; at 1 and 2 CTAs part of the
    values stays in global memory."""
    monkeypatch.setenv("GFEA_RESIDENT_CTAS", str(ctas))
    Nn = 1511
    node_ptr, nbr = hub_graph(Nn, hubs=12, hub_deg=300, seed=D)
    vals, A = spd_values(node_ptr, nbr, D, seed=10 + D)
    rng = np.random.default_rng(5)
    known = rng.random(Nn * D) < 0.03
    xk, b = rng.normal(size=Nn * D), rng.normal(size=Nn * D)
    x, res = solve(node_ptr, nbr, vals, D, known, xk, b, precision)
    u, rhs, Auu, ref = direct(A, b, known, xk)
    assert res.status == 0 and res.iterations > 0
    assert np.array_equal(x[known], xk[known])
    # the stopping rule's residual, and its error at a condition number ~1e4
    assert np.linalg.norm(rhs - Auu @ x[u]) <= 1e-10 * np.linalg.norm(rhs)
    assert np.abs(x[u] - ref).max() <= 1e-7 * np.abs(ref).max()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_neighbours_without_a_halo(monkeypatch, precision):
    """A random graph: a CTA's distinct neighbours do not fit in shared memory."""
    import scipy.sparse as sp

    monkeypatch.setenv("GFEA_RESIDENT_CTAS", "20")
    Nn = 30011
    rng = np.random.default_rng(3)
    i, j = rng.integers(0, Nn, (2, 10 * Nn))
    W = sp.csr_matrix((rng.uniform(0.5, 1.5, i.size), (i, j)), shape=(Nn, Nn))
    W = (W + W.T).tolil()
    W.setdiag(0)
    W = W.tocsr()
    W.eliminate_zeros()
    A = (sp.diags(np.asarray(W.sum(axis=1)).ravel() + 0.5) - W).tocsr()
    A.sort_indices()
    known = rng.random(Nn) < 0.02
    xk, b = rng.normal(size=Nn), rng.normal(size=Nn)
    x, res = solve(A.indptr.astype(np.int32), A.indices.astype(np.int32), A.data, 1, known, xk, b, precision)
    assert res.status == 0
    r = (b - A @ x)[~known]
    ref = (b - A[:, known] @ xk[known])[~known]
    assert np.linalg.norm(r) <= 1e-10 * np.linalg.norm(ref)


@pytest.mark.parametrize("case", ["el_quad4", "el_quad9", "el_hexa8", "el_cantilever_240x26"])
@pytest.mark.parametrize("ctas", [1, 5, 40, 152])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_two_level_matches_reference(golden, monkeypatch, case, ctas, precision):
    monkeypatch.setenv("GFEA_RESIDENT_CTAS", str(ctas))
    g = golden(case)
    simu = elastic(g, precision=precision)
    for _ in range(2):  # new workspace, then kept aggregation and stale packets
        simu.Need_Update()
        u = simu.Solve()
        assert simu.last_solve.status == 0
        assert simu.last_solve.rel_residual <= max(1e-12, simu.last_solve.floor_rel)
        assert rel_err(u, g["u"]) <= 1e-8


@pytest.mark.parametrize("precision,ctas", [("mixed", 6), ("fp64", 9)])
def test_partly_resident_rows_with_known_dofs(monkeypatch, precision, ctas):
    """Lane groups whose nodes are half in shared memory, with scattered known
    DOFs: the same solution as with everything resident."""
    from easyfea_gb300 import Models
    from easyfea_gb300 import mesh as gmesh
    from easyfea_gb300 import simulations as Simulations

    m = gmesh.Mesh_Quad9_Rect(120.0, 13.0, 75, 15)
    out = []
    for c in (ctas, 152):
        monkeypatch.setenv("GFEA_RESIDENT_CTAS", str(c))
        simu = Simulations.Elastic(m, Models.Elastic.Isotropic(2, E=210000.0, v=0.3, planeStress=True, thickness=13.0))
        simu.precision = precision
        simu.add_dirichlet(m.Nodes_Conditions(lambda x, y, z: x == 0), [0.0, 0.0], ["x", "y"])
        simu.add_dirichlet(np.arange(7, m.Nn, 97), [0.01], ["y"])
        simu.add_surfLoad(m.Nodes_Conditions(lambda x, y, z: x == 120.0), [-800 / 13**2], ["y"])
        out.append(simu.Solve())
        assert simu.last_solve.status == 0
    assert np.abs(out[0] - out[1]).max() <= 1e-9 * np.abs(out[1]).max()


def test_stops_at_max_iters_and_reports_singular_blocks():
    from easyfea_gb300 import _lib

    node_ptr, nbr = hub_graph(600, hubs=3, hub_deg=100, seed=1)
    vals, _ = spd_values(node_ptr, nbr, 2, seed=2)
    known = np.zeros(1200, bool)
    known[:3] = True
    import test_gpu_staged as staged

    class Few(_lib.PcgOpts):
        def __init__(self, *a):
            super().__init__(*a)
            self.max_iters = 3

    keep = _lib.PcgOpts
    try:
        _lib.PcgOpts = Few
        with pytest.raises(_lib.GfeaError) as e:
            staged.solve(node_ptr, nbr, vals, 2, known, np.zeros(1200), np.ones(1200), "fp64")
        assert e.value.status == _lib.ERR_NOT_CONVERGED
    finally:
        _lib.PcgOpts = keep
    with pytest.raises(_lib.GfeaError) as e:
        staged.solve(node_ptr, nbr, vals * 0, 2, known, np.zeros(1200), np.ones(1200), "fp64")
    assert e.value.status not in (_lib.OK, _lib.ERR_TIMEOUT)
    assert ctypes.c_int(e.value.status).value > 0
