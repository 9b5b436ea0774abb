"""Gradient flow of a start with no gauge force (unit links, no scalar currents):
the reference returns at the first zero-force link, so every link keeps its value
in every step.  The links stay, in steps of either parity (two markers are used in
turn), and putting all of them back is work for the whole GPU: the flow takes no
longer than a few times that of a hot start, whose links all move."""
import time

import numpy as np
import pytest

from native import hot_fields
from su2higgs_gb300 import abi

pytestmark = pytest.mark.gpu


def lattice(p, f, unit):
    from su2higgs_gb300 import gpu
    link = np.array(f.link)
    if unit:
        link[:] = [1.0, 0.0, 0.0, 0.0]
    lat = gpu.Lattice(p, seed=1)
    lat.upload(link=link, d0=f.d0, trip=f.trip)
    return lat


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("L", [(2, 2, 2), (6, 10, 4), (20, 24, 22)])
def test_unit_links_stay(L, precision):
    p = abi.make_params("fund", L=L, precision=precision)
    rows = lattice(p, hot_fields(p, seed=3, phi_mean=0.5), True).grad_flow(0.045, 0.01, 1)
    assert len(rows) >= 6
    # the Wilson action of unit links is 0, and every row's sums are the first's
    assert np.array_equal(rows[:, 1:], np.broadcast_to(rows[0, 1:], rows[:, 1:].shape), equal_nan=True)


def test_unit_links_are_not_slow():
    p = abi.make_params("pure", L=(64, 64, 64), precision=32)
    f = hot_fields(p, seed=3)
    best = []
    for unit in (False, True):
        lat = lattice(p, f, unit)
        t = []
        for _ in range(4):
            t0 = time.perf_counter()
            lat.grad_flow(0.095, 0.01, 5)
            t.append(time.perf_counter() - t0)
        best.append(min(t))
    assert best[1] < 4 * best[0], best
