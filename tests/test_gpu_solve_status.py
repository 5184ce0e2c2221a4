"""The status of a solve that cannot end well: the same number from the resident
solve and from the multi-kernel iteration."""

import numpy as np
import pytest

from test_gpu_staged import hub_graph, solve, spd_values

pytestmark = pytest.mark.gpu

SINGULAR, BREAKDOWN, NAN = 4, 6, 7


@pytest.mark.parametrize("lanes", [0, 8])  # resident, multi-kernel
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("what,status", [("zero", SINGULAR), ("negative", BREAKDOWN), ("nan in b", NAN)])
def test_status(monkeypatch, what, status, precision, lanes):
    from easyfea_gb300 import _lib

    class Opts(_lib.PcgOpts):
        def __init__(self, *a):
            super().__init__(*a)
            self.lanes = lanes

    monkeypatch.setattr(_lib, "PcgOpts", Opts)
    node_ptr, nbr = hub_graph(600, hubs=3, hub_deg=100, seed=1)
    vals, _ = spd_values(node_ptr, nbr, 2, seed=2)
    known = np.zeros(1200, bool)
    known[:3] = True
    b = np.ones(1200)
    if what == "zero":
        vals = vals * 0
    elif what == "negative":
        vals = -vals
    else:
        b[700] = np.nan
    with pytest.raises(_lib.GfeaError) as e:
        solve(node_ptr, nbr, vals, 2, known, np.zeros(1200), b, precision)
    assert e.value.status == status
