"""RFCA fiducial times of ensembles, a warp per instance up to 64 rows on
average and blocks beyond, against the restatement's serial sum, bit for bit:
instances of none, one and many rows, lost rows, and arrival times on both
sides of a power of two (the serial sum, which is the restatement's where no
row is lost before the cavity)."""
import numpy as np
import pytest

from elegant_b200 import Beam, Element, Lattice, Tracker, workloads as w
from reforacle import PortOracle, by_id

pytestmark = pytest.mark.gpu
P = w.ring_p_central()
LIGHT = 2.99792458e8


def _lattice():
    return Lattice([Element("A", "MAXAMP", {"X_MAX": 0.01, "Y_MAX": 0.01}), Element("D", "DRIF", {"L": 20.0}),
                    Element("RF", "RFCA", {"L": 0.0, "VOLT": 1e6, "FREQ": 500e6, "PHASE": 170.0})])


@pytest.mark.parametrize("sizes", [[1, 0, 3, 32, 33], [64] * 4, [65] * 4, [0, 400, 1, 2] + [1] * 30, [1000, 3, 900]])
@pytest.mark.parametrize("across", [False, True])
def test_instances(sizes, across):
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(offsets[-1])
    rng = np.random.default_rng(n)
    c = np.zeros((n, 6))
    c[:, 1] = rng.normal(0, 1e-5, n)
    c[:, 4] = rng.normal(0, 3e-3, n) + (LIGHT * 2.0 ** -24 - 20.0 if across else 0)
    c[:, 5] = rng.normal(0, 1e-3, n)
    if not across:  # lost before the cavity; the order of a serial sum would be the restatement's own then
        c[rng.random(n) < 0.2, 0] = 0.02
    ids = np.arange(1, n + 1)
    lat = _lattice()
    with Tracker(lat, P, 2) as t:
        t.load_ensemble(offsets, [])
        res = t.track(Beam(c, ids))
    for k in range(len(sizes)):
        sl = slice(offsets[k], offsets[k + 1])
        if sizes[k] == 0:
            continue
        rows = PortOracle("b2e").track(lat, c[sl], ids[sl], P, 2)[0]
        want, want_ids, loss = by_id(rows)
        keep = loss < 0
        assert np.array_equal(res.ids[sl], want_ids) and np.array_equal(res.lost_pass[sl] < 0, keep)
        assert np.array_equal(np.ascontiguousarray(res.coords[sl][keep]).view(np.int64),
                              np.ascontiguousarray(want[keep]).view(np.int64))
