"""Lattices of which no magnet takes the straight-line maps run in kernels with
the general maps in line, against the CPU restatement, bit for bit: quantum
excitation, field terms and steering, second-order edges; with history, with an
ensemble of which one instance alone has straight-line magnets, and with more
element records than shared memory holds."""
import numpy as np
import pytest

from elegant_b200 import Beam, Element, Lattice, Tracker, workloads as w
from reforacle import PortOracle, by_id

pytestmark = pytest.mark.gpu
P = w.ring_p_central()


def _general(kind, cells=2):
    base = w.radiating_ring(isr=True) if kind == "isr" else w.fodo_ring()
    els = []
    for k, e in enumerate(base.elements[:8 * cells]):
        extra = {}
        if kind != "isr" and e.type in ("KQUAD", "KSEXT"):
            extra = {"HKICK": 1e-5 * (1 if k % 2 else -1), "VKICK": 1e-5}
        elif e.type == "CSBEND" and kind != "isr":
            extra = {"K1": 2e-3, "K2": 0.05} if kind == "field" else {"EDGE_ORDER": 2, "E1": 0.1, "HGAP": 0.02, "FINT": 0.5}
        els.append(Element(e.name + str(k), e.type, dict(e.params, **extra)))
    return Lattice(els)


def _beam(n=500):
    c = w.ring_beam(n, seed=8).coords.copy()
    c[n // 2:, :4] *= 40  # losses at the apertures
    return Beam(c, np.arange(1, n + 1))


def _same(res, rows, sl=slice(None)):
    want, ids, loss = by_id(rows)
    assert np.array_equal(res.ids[sl], ids) and np.array_equal(res.lost_pass[sl], loss)
    keep = loss < 0
    assert 0 < keep.sum() < len(keep)
    assert np.array_equal(np.ascontiguousarray(res.coords[sl][keep]).view(np.int64),
                          np.ascontiguousarray(want[keep]).view(np.int64))


def _port(lat, coords, ids, turns):
    port = PortOracle("b2e")
    port.set_isr(7, 3.0)
    rows = port.track(lat, coords, ids, P, turns)[0]
    port.set_isr(0)
    return rows


@pytest.mark.parametrize("cells", [2, 8, 40])
@pytest.mark.parametrize("history", [False, True])
@pytest.mark.parametrize("kind", ["isr", "field", "edges"])
def test_general_maps_alone(kind, history, cells):
    lat = Lattice(_general(kind, min(cells, 8)).elements * max(1, cells // 8))
    beam, turns = _beam(), 3 if cells < 40 else 1
    with Tracker(lat, P, turns, record_history=history, isr_seed=7) as t:
        res = t.track(beam)
    _same(res, _port(lat, beam.coords, beam.ids, turns))


def test_one_instance_with_straight_line_magnets():
    lat = _general("field")
    quads = [i for i, e in enumerate(lat.elements) if e.type in ("KQUAD", "KSEXT")]
    kicks = {i: [(lat.elements[i].params["HKICK"], 1e-5), (0.0, 0.0), (2e-5, 0.0)] for i in quads}
    ov = [(i, k, np.array([v[j] for v in kicks[i]])) for i in quads for j, k in enumerate(("HKICK", "VKICK"))]
    beam = _beam(600)
    offsets = np.array([0, 200, 400, 600], dtype=np.int64)
    order = np.argsort(np.arange(600) % 3, kind="stable")  # survivors and losses in every instance
    coords = beam.coords[order]
    with Tracker(lat, P, 3) as t:
        t.load_ensemble(offsets, ov)
        res = t.track(Beam(coords, beam.ids))
    for k in range(3):
        els = [Element(e.name, e.type, dict(e.params, HKICK=kicks[i][k][0], VKICK=kicks[i][k][1]) if i in kicks
                       else e.params) for i, e in enumerate(lat.elements)]
        sl = slice(200 * k, 200 * (k + 1))
        _same(res, _port(Lattice(els), coords[sl], beam.ids[sl], 3), sl)
