"""The multi-kernel PCG (host checks requested, or staged operators): r.z from
r.y + rc.ec, the direction formed from y and the coarse correction, and the
residual with a component per lane, against the reference's displacements and
against a direct solve of a scalar system."""

import numpy as np
import pytest

from test_gpu_coarse import elastic, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", ["el_quad4", "el_tri3", "el_quad9", "el_hexa8", "el_cantilever_240x26"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("coarse", [0, 7, -1])
@pytest.mark.parametrize("staged", [False, True])
def test_matches_reference(golden, monkeypatch, case, precision, coarse, staged):
    from easyfea_gb300.device import pcg

    if staged:
        monkeypatch.setenv("GFEA_STAGE_MIN_BYTES", "0")
    g = golden(case)
    simu = elastic(g, precision=precision)
    op, b = simu.K_device, simu._neumann_vec("elastic")
    known, x = simu._dirichlet_state("elastic", b)
    info = pcg(op, b, x, known, rtol=1e-12, precision=precision, coarse=coarse, check_every=0 if staged else 8)
    assert info.status == 0 and info.iterations > 0
    assert info.rel_residual <= max(1e-12, info.floor_rel)
    assert rel_err(x.cpu().numpy(), g["u"]) <= 1e-8


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_same_iterations_as_the_resident_solve(golden, precision):
    """Both run the same recurrence; only the order of sums differs."""
    from easyfea_gb300.device import pcg

    g = golden("el_hexa8")
    its = []
    for check in (0, 16):
        simu = elastic(g, precision=precision)
        op, b = simu.K_device, simu._neumann_vec("elastic")
        known, x = simu._dirichlet_state("elastic", b)
        its.append(pcg(op, b, x, known, rtol=1e-10, precision=precision, coarse=-1, check_every=check).iterations)
    assert abs(its[0] - its[1]) <= max(3, 0.1 * its[0]), its
