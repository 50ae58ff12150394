"""The straight-line element maps and their hand-over to the general ones,
against the CPU restatement, bit for bit: coordinates at zero, at signed
zeros, tiny and non-finite, slopes and angles around every limit that sends a
particle to the general map, and elements at the edges of the rule."""
import numpy as np
import pytest

from elegant_b200 import Element, Lattice, Tracker, workloads as w
from elegant_b200.beam import Beam
from reforacle import PortOracle, by_id

pytestmark = pytest.mark.gpu

P = w.ring_p_central()
ANG = 2 * np.pi / 16


def _compare(lat, c, turns):
    beam = Beam(c, np.arange(1, len(c) + 1))
    with Tracker(lat, P, turns) as t:
        res = t.track(beam)
    rows, n_left, _ = PortOracle("b2e").track(lat, beam.coords, beam.ids, P, turns)
    ref, ids, loss = by_id(rows)
    order = np.argsort(res.ids)
    assert np.array_equal(res.lost_pass[order], loss)
    live = loss < 0
    a, b = res.coords[order][live], ref[live]
    assert np.array_equal(np.ascontiguousarray(a[:, :5]).view(np.int64), np.ascontiguousarray(b[:, :5]).view(np.int64))
    # by value: the restatement turns a delta of -0 into 0, the engine keeps it
    assert np.array_equal(a[:, 5], b[:, 5])
    return n_left


def _line(ap=True, **bend):
    els = [Element("MA", "MAXAMP", {"X_MAX": 0.02, "Y_MAX": 0.015, "ELLIPTICAL": 1})] if ap else []
    sr = {k: v for k, v in bend.items() if k == "SYNCH_RAD"}
    els += [Element("QF", "KQUAD", dict({"L": 0.3, "K1": 1.2, "N_KICKS": 8}, **sr)), Element("D", "DRIF", {"L": 0.5}),
            Element("B", "CSBEND", dict({"L": 1.0, "ANGLE": ANG, "N_KICKS": 8}, **bend)),
            Element("QD", "KQUAD", dict({"L": 0.3, "K1": -1.2, "N_KICKS": 8, "DX": 1e-4, "DZ": 1e-4, "TILT": 0.01}, **sr)),
            Element("S", "KSEXT", dict({"L": 0.2, "K2": 5.0}, **sr))]
    return Lattice(els)


def test_odd_coordinates():
    values = [0.0, -0.0, 1e-300, -5e-324, 1e-160, 2.0 ** -250, 1e-76, 1.5e-8, -1.05e-8, 1e-3, -4e-3, 0.13, 0.99, 1.5,
              9.99, 10.01, np.nan, np.inf]
    rng = np.random.default_rng(2)
    c = rng.choice(values, size=(3000, 6))
    c[:2000][np.abs(c[:2000]) > 0.01] = 1e-4
    c[:2500] = np.where(np.isfinite(c[:2500]), c[:2500], 0.0)
    c[:, 5] = np.where(rng.random(3000) < 0.8, rng.choice([0.0, -2.0 ** -53, 2.0 ** -52, 1e-3, -0.9, 0.5, -1.0], 3000), c[:, 5])
    assert 0 < _compare(_line(), c, 2) < 3000
    _compare(_line(ap=False), c, 2)


@pytest.mark.parametrize("bend", [{}, {"N_KICKS": 1}, {"N_KICKS": 2, "INTEGRATION_ORDER": 6},
                                  {"INTEGRATION_ORDER": 2}, {"ANGLE": -ANG, "E1": 0.05}, {"ANGLE": 1e-5},
                                  {"E1": ANG / 2, "E2": ANG / 2, "HGAP": 0.01}, {"DZ": 1e-3, "TILT": 0.2},
                                  {"ANGLE": 2.5, "N_KICKS": 2}, {"SYNCH_RAD": 1}, {"SYNCH_RAD": 1, "E1": 0.05},
                                  {"SYNCH_RAD": 1, "INTEGRATION_ORDER": 6, "ANGLE": -ANG}])
def test_bend_forms_and_amplitudes(bend):
    rng = np.random.default_rng(3)
    c = rng.normal(size=(1500, 6)) * [3e-3, 2e-3, 3e-3, 2e-3, 3e-3, 5e-3]
    c[500:1000] *= rng.choice([1e-9, 1e-5, 3.0, 10.0], size=(500, 1))
    c[1000:, :4] = np.round(c[1000:, :4], 4)
    _compare(_line(**bend), c, 3)


@pytest.mark.parametrize("ap", [{"X_MAX": 0.02, "Y_MAX": 0.015}, {"X_MAX": 0.02}, {"Y_MAX": 0.015, "ELLIPTICAL": 1},
                                {"X_MAX": 0.02, "Y_MAX": 0.015, "ELLIPTICAL": 1, "EXPONENT": 8, "YEXPONENT": 2},
                                {"X_MAX": 1e-40, "Y_MAX": 0.015, "ELLIPTICAL": 1}])
def test_aperture_quick_test(ap):
    """Points on rays to just inside and outside the edge, where the quick test stops."""
    f = np.concatenate([np.linspace(0.9, 1.01, 40), [np.sqrt(0.998), np.sqrt(0.999)]])
    a = np.linspace(0, 2 * np.pi, 33)
    x, y = 0.02 * np.outer(f, np.cos(a)).ravel(), 0.015 * np.outer(f, np.sin(a)).ravel()
    c = np.zeros((x.size, 6))
    c[:, 0], c[:, 2] = x, y
    els = [Element("MA", "MAXAMP", ap)] + _line(ap=False).elements
    _compare(Lattice(els), c, 1)
