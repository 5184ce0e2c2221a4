"""The coarse matrix's inverse (one cooperative launch): A_c^-1 A_c = I for
scalar graph Laplacians, where A_c is the sum of the entries between
aggregates, at the edges of the pivot blocks and of the tiles (one CTA up to 48
unknowns, then tiles of 16 x 16, 32 x 16 ... and a padded last block)."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def coarse_inverse(nx, ny, target, precision, seed):
    import scipy.sparse as sp
    import torch

    from easyfea_gb300 import _lib

    L = _lib.load()
    rng = np.random.default_rng(seed)
    Nn = nx * ny
    X, Y = np.meshgrid(np.arange(nx, dtype=float), np.arange(ny, dtype=float))
    coord = np.stack([X.ravel(), Y.ravel(), np.zeros(Nn)], axis=1)
    ident = lambda n: sp.identity(n, format="csr")  # noqa: E731
    path = lambda n: sp.diags([np.ones(n - 1)], [1], shape=(n, n))  # noqa: E731
    W = (sp.kron(ident(ny), path(nx)) + sp.kron(path(ny), ident(nx))).tocsr()
    W.data = rng.uniform(0.5, 1.5, W.nnz)
    W = W + W.T
    A = (sp.diags(np.asarray(W.sum(axis=1)).ravel() + 0.05) - W).tocsr()
    A.sort_indices()
    if precision == _lib.F32:
        A.data = A.data.astype(np.float32).astype(np.float64)
    d = {k: torch.as_tensor(v, device="cuda") for k, v in
         {"ptr": A.indptr.astype(np.int32), "nbr": A.indices.astype(np.int32), "v64": A.data,
          "v32": A.data.astype(np.float32), "known": np.zeros(Nn, np.uint8), "coord": coord}.items()}
    s = _lib.System(_lib.ABI_VERSION, 1, Nn, A.nnz, _lib.ptr(d["ptr"]), _lib.ptr(d["nbr"]), _lib.ptr(d["v64"]),
                    _lib.ptr(d["v32"]), _lib.ptr(d["known"]), 0, 0, _lib.ptr(d["coord"]))
    o = _lib.PcgOpts(_lib.ABI_VERSION, precision, 0, 0, 0.0, 0.0, 0, 0, target, 0)
    nb = ctypes.c_size_t()
    _lib.check(L.gfea_coarse_workspace_size(ctypes.byref(s), ctypes.byref(o), ctypes.byref(nb)), "size")
    work = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    lv = _lib.CoarseLevel()
    _lib.check(L.gfea_coarse_setup(ctypes.byref(s), ctypes.byref(o), 0, _lib.ptr(work), work.numel(),
                                   ctypes.byref(lv), _lib.stream()), "setup")
    torch.cuda.synchronize()

    def read(ptr, n, dtype):
        off = ptr - work.data_ptr()
        return work[off:off + n * np.dtype(dtype).itemsize].cpu().numpy().view(dtype)

    nc = lv.nc
    agg = read(lv.agg, Nn, np.int32)
    R = sp.csr_matrix((np.ones(Nn), (np.arange(Nn), agg)), shape=(Nn, nc))
    return nc, (R.T @ A @ R).toarray(), read(lv.inv, nc * nc, np.float64).reshape(nc, nc)


@pytest.mark.parametrize("target", [1, 2, 15, 16, 17, 48, 49, 64, 97, 192, 208, 300, 429, 512])
@pytest.mark.parametrize("precision", [0, 1])
def test_inverse_of_the_coarse_matrix(target, precision):
    nc, Ac, inv = coarse_inverse(61, 53, target, precision, seed=target)
    assert 1 <= nc <= target
    shift = 1e-6 if precision else 1e-8  # of the largest diagonal entry, added to the diagonal
    Ac = Ac + shift * np.abs(np.diag(Ac)).max() * np.eye(nc)
    # float-float pairs carry 2^-44; FP32 values add their matrix's own sums (2^-24 per entry)
    cond = np.linalg.cond(Ac)
    tol = cond * (2.0**-40 if precision == 0 else 2.0**-20)
    assert np.abs(inv @ Ac - np.eye(nc)).max() <= tol
    assert np.abs(inv - inv.T).max() <= tol * np.abs(inv).max()


@pytest.mark.parametrize("elem,counts", [("QUAD4", (23, 7)), ("TRI6", (9, 5)), ("HEXA8", (11, 4, 3)), ("TETRA4", (7, 3, 3))])
@pytest.mark.parametrize("target", [1, 5, 9])
def test_rigid_body_modes_of_an_elastic_operator(elem, counts, target):
    """A_c = R^T K R with translations and rotations of every aggregate, known
    DOFs masked: neighbours in several aggregates, whole aggregates inside."""
    import torch

    from easyfea_gb300 import Models, _lib
    from easyfea_gb300 import mesh as gmesh
    from easyfea_gb300 import simulations as Simulations

    dim = len(counts)
    make = gmesh.Mesh_Rect if dim == 2 else gmesh.Mesh_Box
    m = make(gmesh.ElemType(elem), *((30.0, 8.0, 6.0)[:dim]), *counts)
    simu = Simulations.Elastic(m, Models.Elastic.Isotropic(dim, E=210000.0, v=0.3, planeStress=dim == 2))
    op = simu.K_device
    known = np.zeros(m.Nn * dim, np.uint8)
    left = m.Nodes_Conditions(lambda x, y, z: x == 0)
    for k in range(dim):
        known[left * dim + k] = 1
    known[5] = 1
    kd = torch.as_tensor(known, device="cuda")
    s = op.system(kd)
    o = _lib.PcgOpts(_lib.ABI_VERSION, _lib.F64, 0, 0, 0.0, 0.0, 0, 0, target, 0)
    L = _lib.load()
    nb = ctypes.c_size_t()
    _lib.check(L.gfea_coarse_workspace_size(ctypes.byref(s), ctypes.byref(o), ctypes.byref(nb)), "size")
    work = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    lv = _lib.CoarseLevel()
    _lib.check(L.gfea_coarse_setup(ctypes.byref(s), ctypes.byref(o), 0, _lib.ptr(work), work.numel(),
                                   ctypes.byref(lv), _lib.stream()), "setup")
    torch.cuda.synchronize()

    def read(ptr, n, dtype):
        off = ptr - work.data_ptr()
        return work[off:off + n * np.dtype(dtype).itemsize].cpu().numpy().view(dtype)

    agg = read(lv.agg, m.Nn, np.int32)
    off = read(lv.off, 4 * m.Nn, np.float32).reshape(-1, 4).astype(np.float64)
    nc, nr = lv.nc, lv.nr
    R = np.zeros((m.Nn * dim, nc))
    for a in range(m.Nn):
        x, y, z = off[a, :3]
        modes = (np.array([[1, 0, -y], [0, 1, x]]) if dim == 2 else
                 np.array([[1, 0, 0, 0, z, -y], [0, 1, 0, -z, 0, x], [0, 0, 1, y, -x, 0]]))
        R[a * dim:(a + 1) * dim, agg[a] * nr:(agg[a] + 1) * nr] = modes
    R[known.astype(bool)] = 0
    Ac = R.T @ (op.to_scipy() @ R)
    d = np.diag(Ac).copy()
    np.fill_diagonal(Ac, np.where(d > 1e-14 * d.max(), d + 1e-8 * d.max(), d.max()))
    inv = read(lv.inv, nc * nc, np.float64).reshape(nc, nc)
    assert np.abs(inv @ Ac - np.eye(nc)).max() <= np.linalg.cond(Ac) * 2.0**-40
