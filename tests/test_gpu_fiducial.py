"""RFCA fiducial times: the parallel exact sum of arrival times where they
share a binade, the serial Kahan sum where they do not, against the CPU
restatement's serial loop, bit for bit (the RF phase moves every coordinate
behind the cavity)."""
import numpy as np
import pytest

from elegant_b200 import Element, Lattice, Tracker, workloads as w
from elegant_b200.beam import Beam
from reforacle import PortOracle, by_id

pytestmark = pytest.mark.gpu

# a short line keeps the oracle quick; its cavity is at 20 m, or first
DRIFT = 20.0


def _lattice(first):
    rf = Element("RF", "RFCA", {"L": 0.0, "VOLT": 1e6, "FREQ": 500e6, "PHASE": 170.0})
    line = [Element("D", "DRIF", {"L": DRIFT})]
    return Lattice([rf] + line if first else line + [rf])


@pytest.mark.parametrize("n", [1, 2, 255, 257, 5000])
@pytest.mark.parametrize("where", ["one binade", "across a power of two", "at its top", "cavity first"])
def test_fiducial_time_is_the_serial_kahan_mean(n, where):
    """Arrival times t = s/(c beta) around 2^-24 s (17.87 m), wholly above it,
    on both sides of it, within n ulps of 2^-23 s, or of both signs."""
    rng = np.random.default_rng(n)
    c = np.zeros((n, 6))
    c[:, 1] = rng.normal(0, 1e-4, n)
    c[:, 4] = rng.normal(0, 3e-3, n)
    c[:, 5] = rng.normal(0, 1e-3, n)
    light = 2.99792458e8
    if where == "across a power of two":
        c[:, 4] += light * 2.0 ** -24 - DRIFT
    elif where == "at its top":
        c[:, 1:] = 0
        c[:, 4] = light * 2.0 ** -23 - DRIFT - 1.5e-7  # beta < 1 puts t about at the binade's end
        c[:, 4] += np.arange(n) * 2.0 ** -48
    lat = _lattice(where == "cavity first")
    beam = Beam(c, np.arange(1, n + 1))
    p = w.ring_p_central()
    with Tracker(lat, p, 2) as t:
        res = t.track(beam)
    rows, n_left, _ = PortOracle("b2e").track(lat, beam.coords, beam.ids, p, 2)
    ref, ids, loss = by_id(rows)
    assert n_left == res.n_left == n
    assert np.array_equal(res.ids, ids)
    assert np.array_equal(res.coords.view(np.int64), np.ascontiguousarray(ref).view(np.int64))
