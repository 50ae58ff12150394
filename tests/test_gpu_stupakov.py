"""Stupakov's drift wake against the CPU restatement, bit for bit: the modes
of the drift, bin counts around a warp and at the ends of the range, and
bunches so short or long that the scan, the passes or neither solve for phi."""
import numpy as np
import pytest

from csr_cases import stupakov_cases
from elegant_b200 import Tracker, workloads as w
from reforacle import PortOracle, by_id

pytestmark = pytest.mark.gpu
P0 = 1000 / 0.51099895


def _check(lat, beam, passes):
    with Tracker(lat, P0, passes) as t:
        res = t.track(beam)
        wakes = t.csr_wakes(10_000_000)
    rows, nl, _, want = PortOracle("b2e").track(lat, beam.coords, beam.ids, P0, passes, capture_wakes=True)
    coords, ids, _ = by_id(rows)
    order = np.argsort(res.ids)
    assert res.n_left == nl and np.array_equal(res.ids[order], ids)
    assert np.array_equal(wakes, want) and wakes.size > 0
    assert np.array_equal(res.coords[order], coords)


@pytest.mark.parametrize("case", [c for c in stupakov_cases() if "mode0" not in c])
def test_modes(case):
    _check(stupakov_cases()[case], w.chicane_beam(5000, seed=31), 2 if case.endswith("2p") else 1)


@pytest.mark.parametrize("bins", [2, 31, 33, 1025, 4096])
@pytest.mark.parametrize("sigma_z", [2e-6, 1e-3, 0.3])
def test_bins_and_lengths(bins, sigma_z):
    lat = w.chicane(bins=bins, n_kicks=3, stupakov=True, drift={"N_KICKS": 3})
    _check(lat, w.chicane_beam(3000, seed=bins, sigma_z=sigma_z, chirp=0.0), 1)
