"""The waits between the CTAs of a resident solve: a partner that takes part ends
them, one that is absent lets them run out after their limit, and the context
stays usable."""

import ctypes
import time

import pytest

pytestmark = pytest.mark.gpu


def test_wait_for_an_absent_cta_runs_out_and_the_context_survives():
    import torch

    from easyfea_gb300 import _lib

    L = _lib.load()

    def run(limit_us, present):
        st = ctypes.c_int32(99)
        _lib.check(L.gfea_selftest_exchange(limit_us, present, ctypes.byref(st), _lib.stream()), "selftest")
        return st.value

    assert run(200000, 1) == _lib.OK
    t0 = time.perf_counter()
    assert run(20000, 0) == _lib.ERR_TIMEOUT
    assert 0.015 <= time.perf_counter() - t0 < 5.0
    x = torch.arange(1000, dtype=torch.float64, device="cuda")
    assert float((x * 2).sum().item()) == 999000.0
    assert run(200000, 1) == _lib.OK
    with pytest.raises(_lib.GfeaError):
        run(0, 1)
