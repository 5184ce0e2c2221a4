"""Batched PCG with systems on both sides of the wide-cluster limit (400 000
stored values): solutions against single FP64 solves, and bit-equality alone
(wide) and in company (wide, or narrow in a batch that fills the GPU)."""

import numpy as np
import pytest

from easyfea_gb300 import mesh as gmesh
from test_gpu_batch import elastic_system

pytestmark = pytest.mark.gpu

MESHES = {  # stored values: dof_n^2 times the node pairs
    "wide2d": lambda: gmesh.Mesh_Quad4_Rect(120.0, 13.0, 240, 52),
    "wide3d": lambda: gmesh.Mesh_Hexa8_Box(60.0, 10.0, 10.0, 40, 8, 8),
    "narrow2d": lambda: gmesh.Mesh_Quad4_Rect(120.0, 13.0, 60, 7),
    "narrow3d": lambda: gmesh.Mesh_Hexa8_Box(60.0, 10.0, 10.0, 13, 3, 3),
    "one": lambda: gmesh.Mesh_Quad4_Rect(120.0, 13.0, 1, 1),
}


@pytest.mark.parametrize("names", [("wide2d",), ("wide2d", "wide3d"), ("one",), ("narrow3d", "wide3d", "one", "wide2d", "narrow2d")])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_widths(precision, names):
    from easyfea_gb300.batching import solve_batch
    from easyfea_gb300.device import pcg

    systems = [elastic_system(MESHES[k](), 210000.0)[1] for k in names]
    for k, s in zip(names, systems):
        assert (s.op.dof_n**2 * s.op.dmesh.n_pairs >= 400000) == k.startswith("wide")
    x0 = [s.x.clone() for s in systems]
    for coarse in (-1, 0):
        for s, x in zip(systems, x0):
            s.x.copy_(x)
        infos = solve_batch(systems, precision=precision, coarse=coarse)
        for s, x, info in zip(systems, x0, infos):
            assert info.status == 0
            assert info.rel_residual <= max(1e-10, info.floor_rel)
            xs = x.clone()
            pcg(s.op, s.b, xs, s.known, rtol=1e-12, precision="fp64")
            ref = xs.cpu().numpy()
            # both residuals at 1e-10 and 1e-12: the distance of test_gpu_batch
            assert np.abs(s.x.cpu().numpy() - ref).max() <= 1e-7 * np.abs(ref).max()
    mixed = [s.x.cpu().numpy() for s in systems]  # block-Jacobi: no atomics before the solve
    for s, x, m in zip(systems, x0, mixed):
        s.x.copy_(x)
        solve_batch([s], precision=precision, coarse=0)
        assert np.array_equal(s.x.cpu().numpy(), m)


@pytest.mark.parametrize("name", ["wide2d", "wide3d"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_same_bits_at_either_width(precision, name):
    from easyfea_gb300.batching import solve_batch

    systems = [elastic_system(MESHES[name](), 210000.0)[1] for _ in range(24)]  # 38 largest > 2 x 24: no
    x0 = systems[0].x.clone()
    solve_batch(systems, precision=precision, coarse=0)
    narrow = systems[0].x.cpu().numpy()  # (each system's K has its own rounding: atomics)
    systems[0].x.copy_(x0)
    solve_batch(systems[:1], precision=precision, coarse=0)
    assert np.array_equal(systems[0].x.cpu().numpy(), narrow)
