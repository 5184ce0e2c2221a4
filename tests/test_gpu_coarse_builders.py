"""gfea_coarse_setup and gfea_coarse_batch_build build the same level: the same
regularisation and, to rounding, the same inverse, positive definite also where
aggregates have one or two nodes."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("elem,counts,target", [("HEXA8", (24, 7, 6), 60), ("HEXA8", (8, 3, 2), 64), ("QUAD4", (60, 8), 90),
                                                ("TETRA4", (6, 2, 2), 40)])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_single_and_batched_inverse_agree(elem, counts, target, precision):
    import torch

    from easyfea_gb300 import Models, _lib
    from easyfea_gb300 import mesh as gmesh
    from easyfea_gb300 import simulations as Simulations

    dim = len(counts)
    make = gmesh.Mesh_Rect if dim == 2 else gmesh.Mesh_Box
    m = make(gmesh.ElemType(elem), *((100.0, 20.0, 20.0)[:dim]), *counts)
    simu = Simulations.Elastic(m, Models.Elastic.Isotropic(dim, E=210000.0, v=0.3))
    op = simu.K_device
    op.ensure_f32()
    known = np.zeros(m.Nn * dim, np.uint8)
    left = np.flatnonzero(m.coord[:, 0] == 0)
    for k in range(dim):
        known[left * dim + k] = 1
    kd = torch.as_tensor(known, device="cuda")
    prec = _lib.F64 if precision == "fp64" else _lib.F32
    s = op.system(kd)
    o = _lib.PcgOpts(_lib.ABI_VERSION, prec, 0, 0, 0.0, 0.0, 0, 0, target, 0)
    L = _lib.load()
    nb = ctypes.c_size_t()
    _lib.check(L.gfea_coarse_workspace_size(ctypes.byref(s), ctypes.byref(o), ctypes.byref(nb)), "size")
    work = torch.empty(nb.value, dtype=torch.uint8, device="cuda")
    lv = (_lib.CoarseLevel * 1)()
    _lib.check(L.gfea_coarse_setup(ctypes.byref(s), ctypes.byref(o), 0, _lib.ptr(work), work.numel(), lv, _lib.stream()),
               "setup")
    torch.cuda.synchronize()

    def inverse():
        off = lv[0].inv - work.data_ptr()
        return work[off:off + 8 * lv[0].nc**2].cpu().numpy().view(np.float64).reshape(lv[0].nc, -1).copy()

    one = inverse()
    scratch = torch.empty(int(L.gfea_coarse_batch_scratch_size(1)), dtype=torch.uint8, device="cuda")
    systems, works = (_lib.System * 1)(s), (ctypes.c_void_p * 1)(work.data_ptr())
    _lib.check(L.gfea_coarse_batch_prepare(systems, ctypes.byref(o), 1, works, lv, _lib.ptr(scratch), scratch.numel(),
                                           _lib.stream()), "prepare")
    first = (ctypes.c_int32 * 4)(*[0 if d < dim else 1 for d in range(4)])
    _lib.check(L.gfea_coarse_batch_build(_lib.ptr(scratch), 1, first, lv[0].nc, prec, _lib.stream()), "build")
    torch.cuda.synchronize()
    batch = inverse()
    # n products in pairs of 2^-45 on the condition number, either side; FP32
    # values: the matrix's own sums (2^-24 an entry)
    cond = np.linalg.cond(one)
    tol = 2 * len(one) * 2.0**-45 * cond + (cond * 2.0**-20 if precision == "mixed" else 0)
    assert np.linalg.norm(one - batch) <= tol * np.linalg.norm(one)
    for inv in (one, batch):
        assert np.linalg.eigvalsh((inv + inv.T) / 2).min() > 0
