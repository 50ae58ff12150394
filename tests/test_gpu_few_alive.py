"""CSR elements with none, one, two or a few particles alive at their
entrance, which decides whether a bunch gets a wake at all: single bunches
that an aperture thins between the dipoles, and a train whose bunches differ,
against the CPU restatement, bit for bit."""
import numpy as np
import pytest

from elegant_b200 import Beam, Element, Lattice, Tracker, workloads as w
from elegant_b200._native import EngineError
from reforacle import PortOracle, by_id

pytestmark = pytest.mark.gpu
P0 = 1000 / 0.51099895


def _lattice(stupakov, drift=None):
    els = list(w.chicane(bins=60, n_kicks=3, stupakov=stupakov, drift=drift or {"N_KICKS": 2}).elements)
    at = next(i for i, e in enumerate(els) if e.name == "B2")
    return Lattice(els[:at] + [Element("A", "MAXAMP", {"X_MAX": 0.5, "Y_MAX": 0.01})] + els[at:])


def _beam(alive, lost, seed=3):
    beam = w.chicane_beam(alive + lost, seed=seed)
    c = beam.coords.copy()
    c[alive:, 2] = 0.02 * np.linspace(1, 2, max(lost, 1))[:lost]
    return Beam(c, beam.ids)


def _same(coords, ids, lost_pass, rows):
    want, want_ids, want_loss = by_id(rows)
    order = np.argsort(ids)
    assert np.array_equal(ids[order], want_ids)
    assert np.array_equal(lost_pass[order] < 0, want_loss < 0)
    keep = want_loss < 0
    assert np.array_equal(coords[order][keep], want[keep])


@pytest.mark.parametrize("stupakov", [False, True])
@pytest.mark.parametrize("alive,lost", [(0, 3), (1, 0), (1, 40), (2, 0), (2, 40), (300, 40)])
def test_thinned_bunch(alive, lost, stupakov):
    lat, beam = _lattice(stupakov), _beam(alive, lost)
    with Tracker(lat, P0, 1) as t:
        res = t.track(beam)
        wakes = t.csr_wakes(1_000_000)
    rows, nl, _, want = PortOracle("b2e").track(lat, beam.coords, beam.ids, P0, 1, capture_wakes=True)
    assert res.n_left == nl and np.array_equal(wakes, want)
    _same(res.coords, res.ids, res.lost_pass, rows)


@pytest.mark.parametrize("stupakov", [False, True])
def test_train_of_unlike_bunches(stupakov):
    lat, parts = _lattice(stupakov), [(1, 30), (400, 20), (0, 2), (2, 0), (1, 0), (257, 1)]
    beams = [_beam(a, l, seed=k) for k, (a, l) in enumerate(parts)]
    offsets = np.concatenate([[0], np.cumsum([a + l for a, l in parts])]).astype(np.int64)
    coords = np.concatenate([b.coords for b in beams])
    ids = np.arange(1, len(coords) + 1, dtype=beams[0].ids.dtype)
    with Tracker(lat, P0, 1) as t:
        t.load_ensemble(offsets, [])
        res = t.track(Beam(coords, ids))
    for k in range(len(parts)):
        sl = slice(offsets[k], offsets[k + 1])
        rows, _, _ = PortOracle("b2e").track(lat, coords[sl], ids[sl], P0, 1)
        _same(res.coords[sl], res.ids[sl], res.lost_pass[sl], rows)


@pytest.mark.parametrize("alive,raises", [(1, False), (2, True)])
def test_invalid_kick_count_is_an_error_only_with_a_wake(alive, raises):
    lat = _lattice(False, {"N_KICKS": 0})
    with Tracker(lat, P0, 1) as t:
        if raises:
            with pytest.raises(EngineError):
                t.track(_beam(alive, 0))
        else:
            t.track(_beam(alive, 0))
