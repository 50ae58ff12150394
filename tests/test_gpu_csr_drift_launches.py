"""A CSRDRIFT launches what its wakes take and no more: the bunches without a
wake drift inside the first kick's kernel, and where an aperture has left no
bunch with two particles the kicks end when the host learns of it."""
import numpy as np
import pytest

from elegant_b200 import Beam, Element, Lattice, Tracker, workloads as w
from reforacle import PortOracle, by_id

pytestmark = pytest.mark.gpu
P0 = 1000 / 0.51099895


def _line(kicks, stupakov, thin):
    els = list(w.chicane(bins=60, n_kicks=3, stupakov=stupakov, drift={"N_KICKS": kicks}).elements)
    at = next(i for i, e in enumerate(els) if e.name == "D1")
    aperture = [Element("A", "MAXAMP", {"X_MAX": 0.5, "Y_MAX": 0.01})] if thin else []
    return Lattice(els[:at] + aperture + els[at:at + 1]), Lattice(els[:at] + aperture)


def _launches(lat, beam, reducer=None):
    with Tracker(lat, P0, 1) as t:
        t.set_csr_reducer(reducer)
        res = t.track(beam)
        first = t.launches
        t.track(beam)
        return t.launches - first, res


def _beam(alive, lost):
    c = w.chicane_beam(alive + lost, seed=3).coords.copy()
    c[alive:, 2] = 0.02
    return Beam(c, np.arange(1, alive + lost + 1))


@pytest.mark.parametrize("stupakov,per_kick,closing", [(False, 2, 2), (True, 5, 1)])
@pytest.mark.parametrize("kicks", [1, 2, 7])
def test_launches_with_a_wake(kicks, stupakov, per_kick, closing):
    """The alive count, the flags, the kicks, the closing half drift and the
    sweep behind the element."""
    whole, before = _line(kicks, stupakov, False)
    beam = _beam(300, 0)
    assert _launches(whole, beam)[0] - _launches(before, beam)[0] <= 3 + per_kick * kicks + closing


@pytest.mark.parametrize("stupakov", [False, True])
@pytest.mark.parametrize("alive", [0, 1])
def test_thinned_bunch_leaves_kicks_out(alive, stupakov):
    """From when the host has the count: it is some kicks ahead of the device by
    then, but not 500 of them."""
    whole, before = _line(1000, stupakov, True)
    beam = _beam(alive, 40)
    n, res = _launches(whole, beam)
    assert n - _launches(before, beam)[0] <= 500 * (5 if stupakov else 2)
    rows, n_left, _ = PortOracle("b2e").track(whole, beam.coords, beam.ids, P0, 1)
    want, want_ids, want_loss = by_id(rows)
    assert res.n_left == n_left == alive
    keep = want_loss < 0
    assert np.array_equal(res.ids, want_ids) and np.array_equal(res.lost_pass < 0, keep)
    assert np.array_equal(res.coords[keep], want[keep])


@pytest.mark.parametrize("alive", [1, 300])
def test_reducer_is_called_only_for_wakes_that_are_formed(alive):
    """Ranges and histograms of a Stupakov drift are reduced over the ranks when
    a bunch has a wake; a thinned one costs the alive count alone."""
    whole, before = _line(3, True, True)
    calls = {}
    for name, lat in (("whole", whole), ("before", before)):
        ops = calls[name] = []
        _launches(lat, _beam(alive, 40), lambda op, ptr, count, stream: ops.append(op))
    extra = (len(calls["whole"]) - len(calls["before"])) / 2  # two runs
    assert extra == 1 if alive == 1 else extra >= 1 + 3 * 2
