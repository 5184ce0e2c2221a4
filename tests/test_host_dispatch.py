"""Which kernels a solve launches, and with what grids and shared memory, on
devices this machine does not have: a fake CUDA runtime records the launches of
the built library and refuses what the real one would refuse."""

import json
import os
import subprocess
import sys

import pytest

from easyfea_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    _build.build()
    d = tmp_path_factory.mktemp("fake")
    script = d / "fake.map"
    script.write_text("libcudart.so.13 { global: *; };\n")
    so = str(d / "libcudart.so.13")
    inc = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(_build.nvcc_path()))), "include")
    r = subprocess.run(["g++", "-shared", "-fPIC", "-O1", "-std=c++17", "-I", inc, "-Wl,-soname,libcudart.so.13",
                        f"-Wl,--version-script={script}", "-o", so, os.path.join(HERE, "fake_cudart.cpp")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def go(*steps, env=None):
        r = subprocess.run([sys.executable, os.path.join(HERE, "host_dispatch.py"), so, json.dumps(steps)],
                           capture_output=True, text=True, timeout=120, env={**os.environ, **(env or {})})
        assert r.returncode == 0, r.stderr[-2000:]
        return json.loads(r.stdout.strip().splitlines()[-1])

    return go


def names(step):
    return [line.split()[0] for line in step["launches"]]


def refused(step):
    return [line for line in step["launches"] if line.endswith("refused")]


BOX = {"D": 3, "nodes": 13104, "degree": 24, "precision": "fp64"}


@pytest.mark.parametrize("case,kernel", [
    ({**BOX}, "resident_kernel"),
    ({**BOX, "precision": "mixed"}, "resident_kernel"),
    ({"D": 2, "nodes": 2106, "degree": 7, "precision": "mixed"}, "resident_kernel"),  # 40 to 48 KB
    ({**BOX, "nodes": 100000, "coarse": 250}, "coarse_inverse"),
    ({**BOX, "precision": "mixed", "coarse": 0, "check_every": 4, "env": {"GFEA_STAGE_MIN_BYTES": "0"}},
     "apply_staged_kernel"),
])
def test_shared_memory_is_opted_into_on_every_device(run, case, kernel):
    """The attribute belongs to the device that was current when it was set: a
    second device of the same process has to get it too."""
    out = run({**case, "device": 0}, {**case, "device": 1})
    for s in out:
        assert any(n.startswith(kernel) for n in names(s)), names(s)
        assert not refused(s)
    assert names(out[0]) == names(out[1])


@pytest.mark.parametrize("sms", [152, 100, 16])
@pytest.mark.parametrize("aggregates", [40, 250])
def test_coarse_inverse_needs_no_co_resident_grid(run, sms, aggregates):
    """240 and 1,500 coarse unknowns on a device or an MPS share of fewer SMs."""
    (s,) = run({**BOX, "nodes": 100000, "coarse": aggregates, "sms": sms})
    inverse = [line for line in s["launches"] if line.startswith("coarse_inverse")]
    assert inverse and not any("cooperative" in line or "refused" in line for line in inverse)


def resident_ctas(step):
    return [int(line.split()[2]) for line in step["launches"] if line.startswith("resident_kernel")]


@pytest.mark.parametrize("sms", [152, 100, 16])
def test_resident_grid_fits_the_device(run, sms):
    (s,) = run({**BOX, "nodes": 5000, "sms": sms})
    assert s["status"] in (0, 5) and not refused(s)
    assert resident_ctas(s) and max(resident_ctas(s)) <= sms or "apply_kernel" in names(s)


def test_refused_cooperative_launch_leaves_the_multi_kernel_iteration(run):
    """A context of fewer SMs than the device reports (a green context)."""
    (s,) = run({**BOX, "coop_limit": 60})
    assert s["status"] == 5 == s["result"]  # the recorded iteration stops at once
    assert [line.split()[0] for line in refused(s)] == ["resident_kernel"]
    after = names(s)[names(s).index("resident_kernel") + 1:]
    assert "bjacobi_kernel" in after and any(n.startswith("apply") for n in after)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_wait_that_ran_out_leaves_the_multi_kernel_iteration(run, precision):
    (s,) = run({**BOX, "precision": precision, "timed_out": 1})
    assert s["status"] == 5 == s["result"]  # the recorded iteration stops at once; not GFEA_ERR_TIMEOUT
    after = names(s)[names(s).index("resident_kernel") + 1:]
    assert "bjacobi_kernel" in after and any(n.startswith("apply") for n in after)


@pytest.mark.parametrize("nodes,degree,precision,least", [(2025, 52, "fp64", 90), (2025, 52, "mixed", 90),
                                                          (600, 41, "fp64", 18), (2025, 24, "fp64", 40)])
def test_long_rows_spread_over_more_ctas(run, nodes, degree, precision, least):
    """A CTA's work goes by its stored values, and the longest rows come
    together (corner nodes first): about 10,240 values a CTA, with room for rows
    of three times the average length or all of the shared memory."""
    (s,) = run({**BOX, "nodes": nodes, "degree": degree, "precision": precision})
    (line,) = [line for line in s["launches"] if line.startswith("resident_kernel")]
    w = line.split()
    grid = int(w[w.index("grid") + 1])
    assert least <= grid <= 152
    values = nodes * degree * (9 * (8 if precision == "fp64" else 4) + 2) / grid
    assert int(w[w.index("smem") + 1]) >= min(3 * values, 200 * 1024)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_lanes_reach_the_product_they_schedule(run, precision):
    (s,) = run({**BOX, "precision": precision, "lanes": 16})
    assert "resident_kernel" not in names(s) and any(n.startswith("apply") for n in names(s))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_first_solve_tunes_the_product_and_is_resident(run, precision):
    first, second = run({**BOX, "precision": precision, "tune_mode": 2}, {**BOX, "precision": precision, "tune_mode": 2})
    n = names(first)
    assert any(k.startswith("apply") for k in n[:n.index("resident_kernel")])
    assert n[-1] == "resident_kernel" == names(second)[-1]
    assert not any(k.startswith("apply") for k in names(second))


@pytest.mark.parametrize("nodes,degree,precision,resident", [
    (13005, 57, "fp64", True), (26901, 59, "fp64", False), (69000, 64, "fp64", False), (38360, 53, "fp64", False),
    (20280, 52, "fp64", True), (22000, 58, "mixed", True), (60000, 60, "mixed", False), (2000, 8, "fp64", True)])
def test_operators_that_cannot_be_staged_are_resident_up_to_a_size(run, nodes, degree, precision, resident):
    """Tiles of long rows are too large to be staged at any size: that they are
    not staged does not mean that they stay in L2."""
    (s,) = run({**BOX, "nodes": nodes, "degree": degree, "precision": precision, "coarse": 0})
    assert ("resident_kernel" in names(s)) == resident
    assert resident or any(n.startswith("apply") for n in names(s))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_staged_operator_in_a_workspace_without_tiles_is_not_resident(run, precision):
    big = {**BOX, "nodes": 90000, "precision": precision, "coarse": 0}
    s, short = run(big, {**big, "work_without_tiles": 1})
    assert "apply_staged_kernel" in names(s)
    assert "resident_kernel" not in names(short) and "apply_kernel" in names(short)
