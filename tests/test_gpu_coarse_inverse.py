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
