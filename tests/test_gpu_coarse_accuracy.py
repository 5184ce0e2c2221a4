"""Accuracy of the coarse matrix's inverse where the matrix is hardest: the
rotations of aggregates of one or two nodes leave pivots at the level of the
regularising shift (condition numbers of a few 1e8).  Compared with an inverse
in extended precision."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHIFT = 1e-8  # of the largest diagonal entry, FP64 values


def coarse_level(m, target):
    """(A_c with its regularisation, the device's inverse) of an elastic
    operator clamped at its left end, FP64."""
    import torch

    from easyfea_gb300 import Models, _lib
    from easyfea_gb300 import simulations as Simulations

    dim = m.dim
    simu = Simulations.Elastic(m, Models.Elastic.Isotropic(dim, E=210000.0, v=0.3))
    op = simu.K_device
    known = np.zeros(m.Nn * dim, np.uint8)
    left = np.flatnonzero(m.coord[:, 0] == m.coord[:, 0].min())
    for k in range(dim):
        known[left * dim + k] = 1
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
        R[a * dim:(a + 1) * dim, agg[a] * nr:(agg[a] + 1) * nr] = np.array(
            [[1, 0, 0, 0, z, -y], [0, 1, 0, -z, 0, x], [0, 0, 1, y, -x, 0]])
    R[known.astype(bool)] = 0
    Ac = R.T @ (op.to_scipy() @ R)
    d = np.diag(Ac).copy()
    np.fill_diagonal(Ac, np.where(d > 1e-14 * d.max(), d + SHIFT * d.max(), d.max()))
    return Ac, read(lv.inv, nc * nc, np.float64).reshape(nc, nc)


def extended_inverse(A):
    """Gauss-Jordan without pivoting (A is SPD) in extended precision."""
    M = A.astype(np.longdouble)
    for p in range(len(M)):
        row = M[p] / M[p, p]
        row[p] = 1 / M[p, p]
        col = M[:, p].copy()
        M[:, p] = 0
        M -= np.outer(col, row)
        M[p] = row
    return M.astype(np.float64)


@pytest.mark.parametrize("elem,counts,target", [("HEXA8", (8, 3, 2), 64), ("TETRA4", (6, 2, 2), 40)])
def test_aggregates_of_one_and_two_nodes(elem, counts, target):
    from easyfea_gb300 import mesh as gmesh

    m = gmesh.Mesh_Box(gmesh.ElemType(elem), 100.0, 20.0, 20.0, *counts)
    Ac, inv = coarse_level(m, target)
    n, cond = len(Ac), np.linalg.cond(Ac)
    assert cond > 1e8  # the hard case
    ref = extended_inverse(Ac)
    # n products in pairs of 2^-45, on the condition number
    assert np.linalg.norm(inv - ref) <= n * 2.0**-45 * cond * np.linalg.norm(ref)
    assert np.linalg.eigvalsh((inv + inv.T) / 2).min() > 0
