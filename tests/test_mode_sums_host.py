"""The restriction's sums in the FP32 solve: float pairs, whatever the number of
an aggregate's nodes that a lane adds up."""

import os
import subprocess

import pytest

from easyfea_gb300 import _build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("modes") / "mode_sums")
    # no contraction of products and sums: the pairs' error terms rely on each rounding
    r = subprocess.run([_build.nvcc_path(), *_build.ARCH, "-std=c++17", "-O1", "-Xcompiler", "-ffp-contract=off", "-I",
                        _build.CSRC, "-o", exe, os.path.join(HERE, "mode_sums.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("nodes", [1, 31, 33, 4000])
def test_sums_keep_the_bits_of_their_products(program, dim, nodes):
    err = float(subprocess.run([program, str(nodes), str(dim)], capture_output=True, text=True, check=True).stdout)
    # exact products; each addition's error is kept in a float: 2^-24 of 2^-24 a
    # term, and the reference's own 2^-53 a term
    assert err <= nodes * (2.0**-47 + 2.0**-52)
