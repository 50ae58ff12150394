"""CSRCSBEND at every integration order and with what keeps it from the
straight-line slice (a large angle, rolled and misaligned magnets take it),
against the CPU restatement, bit for bit, over one and several tiles."""
import numpy as np
import pytest

from elegant_b200 import Element, Lattice, Tracker, workloads as w
from reforacle import PortOracle, by_id

pytestmark = pytest.mark.gpu
P0 = 1000 / 0.51099895


@pytest.mark.parametrize("bend", [{"INTEGRATION_ORDER": 2}, {"INTEGRATION_ORDER": 4}, {"INTEGRATION_ORDER": 6},
                                  {"INTEGRATION_ORDER": 6, "ETILT": 1e-3, "DX": 1e-4, "TILT": 0.1},
                                  {"INTEGRATION_ORDER": 4, "N_KICKS": 1, "ANGLE": 1.2},
                                  {"INTEGRATION_ORDER": 2, "EDGE_ORDER": 2, "E1": 0.02, "HGAP": 0.01}])
@pytest.mark.parametrize("n", [127, 129, 5000])
def test_orders(bend, n):
    els = [Element(e.name, e.type, dict(e.params, **dict(bend, ANGLE=np.sign(e.params["ANGLE"]) * bend["ANGLE"])
                                        if "ANGLE" in bend else dict(e.params, **bend)))
           if e.type == "CSRCSBEND" else e for e in w.chicane(bins=80, n_kicks=4).elements]
    lat, beam = Lattice(els), w.chicane_beam(n, seed=n)
    with Tracker(lat, P0, 1) as t:
        res = t.track(beam)
        wakes = t.csr_wakes(1_000_000)
    rows, nl, _, want = PortOracle("b2e").track(lat, beam.coords, beam.ids, P0, 1, capture_wakes=True)
    coords, ids, loss = by_id(rows)
    order = np.argsort(res.ids)
    assert res.n_left == nl and np.array_equal(res.ids[order], ids) and np.array_equal(wakes, want)
    keep = loss < 0
    assert np.array_equal(res.lost_pass[order] < 0, keep)
    assert np.array_equal(res.coords[order][keep], coords[keep])
