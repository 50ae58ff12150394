"""The work that users of the engine have it do, as measurable cases.

Tracking a beam is one call of a Tracker whose lattice is loaded beforehand:
small beams go through host arrays (Tracker.track), large ones through pinned
host buffers or device tensors, as a program with many particles keeps them.
The ring is the 8-cell FODO ring of elegant_b200.workloads, the chicane its
four-dipole bunch compressor with CSR, the wake network the one of
elegant_b200.wakenet on 1,024-bin profiles.

listed() has the fixed cases, draw() takes more from the same ranges; run()
is one pass through the public entry points and exact() what plain torch
gives for it in 64 bits, where that takes seconds.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from elegant_b200 import Beam, Tracker, workloads
from elegant_b200.flops import flops_per_particle_turn
from elegant_b200.wake_surrogate import wake_batch
from elegant_b200.wakenet import CH, DILATIONS, IN_CH, LAYERS, TAPS, WSIZE, WakeNet, init_params

C = 2.99792458e8
E_CHARGE = 1.602176634e-19
E_MASS = 9.1093837015e-31
DEV = "cuda"


def listed():
    return [
        # a lattice check: a few hundred particles for a few turns, latency only
        {"name": "ring_probe", "kind": "ring", "n": 200, "turns": 10, "radiation": False},
        # one matched bunch for many turns: one warp per SM sub-partition
        {"name": "ring_bunch", "kind": "ring", "n": 10000, "turns": 50, "radiation": False},
        # synchrotron radiation on in every magnet (odd particle count)
        {"name": "ring_radiating", "kind": "ring", "n": 40001, "turns": 8, "radiation": True},
        # error seeds: instances of 500-4,000 particles with the per-pass history, pinned host buffers
        {"name": "ring_ensemble", "kind": "ensemble", "instances": 512, "turns": 30},
        # many-particle dynamic aperture: a grid out to the loss boundary, lost particles compacted away
        {"name": "aperture_scan", "kind": "aperture", "nx": 141, "ny": 71, "turns": 60},
        # frequency map: turn-by-turn records of a grid and its NAFF tunes
        {"name": "frequency_map", "kind": "tunes", "nx": 21, "ny": 20, "turns": 200},
        # a compressor study's coarse bunch, with Stupakov's wake in the drifts
        {"name": "chicane_small", "kind": "chicane", "n": 20011, "bins": 300, "kicks": 10, "half": 1, "stupakov": True},
        # the million-particle compressor run on device tensors
        {"name": "chicane", "kind": "chicane", "n": 1000000, "bins": 600, "kicks": 20, "half": 2, "stupakov": False},
        # a bunch train through the compressor, ragged bunch sizes
        {"name": "bunch_train", "kind": "train", "bunches": 5, "n_min": 200000, "n_max": 1200000, "bins": 600, "kicks": 20},
        # loss and gradients of the wake network for a training batch
        {"name": "wakenet_gradients", "kind": "gradients", "profiles": 256},
        # wake network inference on a batch of profiles
        {"name": "wakenet_forward", "kind": "forward", "profiles": 1500},
        # the plain wake integral of many profiles (training labels)
        {"name": "wake_integrals", "kind": "integrals", "profiles": 3000, "bins": 1024},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ring", "ring", "ensemble", "aperture", "tunes", "chicane", "chicane", "train", "gradients",
                       "forward", "integrals"])
    if kind == "ring":
        n = _log(rng, 64, 400000)
        return {"kind": kind, "n": n, "turns": max(2, min(60, _log(rng, 2, 60), 3000000 // n)),
                "radiation": rng.random() < 0.3}
    if kind == "ensemble":
        return {"kind": kind, "instances": _log(rng, 3, 512), "turns": rng.randint(2, 30)}
    if kind == "aperture":
        return {"kind": kind, "nx": rng.randint(21, 160), "ny": rng.randint(11, 80), "turns": rng.randint(10, 60)}
    if kind == "tunes":
        return {"kind": kind, "nx": rng.randint(3, 30), "ny": rng.randint(3, 30), "turns": rng.randint(60, 200)}
    if kind == "chicane":
        return {"kind": kind, "n": _log(rng, 3000, 1500000), "bins": rng.randint(100, 1000),
                "kicks": rng.randint(5, 25), "half": rng.randint(1, 4), "stupakov": rng.random() < 0.3}
    if kind == "train":
        lo = _log(rng, 20000, 300000)
        return {"kind": kind, "bunches": rng.randint(2, 8), "n_min": lo, "n_max": 3 * lo,
                "bins": rng.randint(200, 800), "kicks": rng.randint(5, 20)}
    if kind == "gradients":
        return {"kind": kind, "profiles": _log(rng, 8, 320)}
    if kind == "forward":
        return {"kind": kind, "profiles": _log(rng, 1, 2500)}
    return {"kind": kind, "profiles": _log(rng, 1, 4000), "bins": rng.randint(300, 1024)}


# ------------------------------------------------------------------ inputs --

def _ring(radiation=False):
    return workloads.radiating_ring() if radiation else workloads.fodo_ring()


def _ring_beam(n, seed):
    return workloads.ring_beam(n, seed=seed, lattice=workloads.fodo_ring(rf=False))


def _chicane(case):
    return workloads.chicane(bins=case["bins"], n_kicks=case["kicks"], sg_halfwidth=case.get("half", 2),
                             stupakov=bool(case.get("stupakov")))


def _chicane_p():
    return workloads.CHICANE_P_MEV / 0.51099895


def _bunch_columns(sizes, seed):
    """SoA columns on the device: chirped 1 mm bunches, one after the other."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    eps, beta = 1e-6 / _chicane_p(), 10.0
    cols = [[] for _ in range(6)]
    for k, n in enumerate(sizes):
        z = torch.randn((6, n), generator=g, dtype=torch.float64, device=DEV)
        z -= z.mean(dim=1, keepdim=True)
        s = 1e-3 * z[4]
        chirp = -15.0 + 10.0 * ((k * 7 + seed) % 11) / 10.0
        for c, v in zip(cols, (math.sqrt(eps * beta) * z[0], math.sqrt(eps / beta) * z[1], math.sqrt(eps * beta) * z[2],
                               math.sqrt(eps / beta) * z[3], s, 1e-4 * z[5] + chirp * s)):
            c.append(v)
    return [torch.cat(c) for c in cols]


def _train_sizes(case):
    rng = np.random.default_rng(case["n_min"])
    return [int(v) for v in rng.integers(case["n_min"], case["n_max"] + 1, size=case["bunches"])]


def _ensemble_offsets(case):
    counts = np.random.default_rng(case["instances"]).integers(500, 4001, size=case["instances"])
    return np.concatenate([[0], np.cumsum(counts)])


def _ensemble_errors(lattice, n, seed):
    """Quadrupole offsets and strength errors of every instance, cut at three sigma."""
    rng, out = np.random.default_rng(seed), []
    for i, e in enumerate(lattice.elements):
        rms = {"KQUAD": {"DX": 50e-6, "DY": 50e-6, "FSE": 1e-3}, "KSEXT": {"FSE": 1e-2}}.get(e.type, {})
        out += [(i, k, np.clip(rng.standard_normal(n), -3, 3) * v) for k, v in rms.items()]
    return out


def _grid_beam(case, seed):
    """Grid of the aperture and frequency-map searches, its limits moved a little by the seed."""
    u = 1.0 + 0.02 * (seed % 17) / 17.0
    full = case["kind"] == "aperture"
    xm, ym = (0.018 * u, 0.016 * u) if full else (0.0030 * u, 0.0020 * u)
    x, y = np.meshgrid(np.linspace(-xm, xm, case["nx"]), np.linspace(1e-6, ym, case["ny"]), indexing="ij")
    n = x.size + 1  # row 0: the reference particle
    c = np.zeros((n, 6))
    c[1:, 0], c[1:, 2] = x.ravel(), y.ravel()
    return Beam(c, np.arange(1, n + 1))


def _profiles(case, seed):
    """Histograms of Gaussian mixtures with shot noise, and slippages in bins."""
    n, nb = case["profiles"], case["bins"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    u = torch.rand((3, n, 1), generator=g, dtype=torch.float64, device=DEV)
    i = torch.arange(nb, dtype=torch.float64, device=DEV)[None, :]
    a = torch.exp(-0.5 * ((i - nb * (0.35 + 0.1 * u[0])) / (nb * (0.04 + 0.06 * u[1]))) ** 2)
    b = torch.exp(-0.5 * ((i - nb * (0.55 + 0.1 * u[2])) / (nb * (0.04 + 0.06 * u[0]))) ** 2)
    counts = (a + u[1] * b) * (2e6 / nb)
    noise = torch.randn((n, nb), generator=g, dtype=torch.float64, device=DEV)
    counts = torch.clamp(counts + noise * torch.sqrt(counts), min=0).contiguous()
    slip = torch.exp(torch.rand(n, generator=g, dtype=torch.float64, device=DEV) * math.log(2.0 * nb)).contiguous()
    return counts, slip


def _net_batch(case, seed):
    """Network inputs [n][4][1024] as the features come out, and smooth targets."""
    n, nb = case["profiles"], 1024
    counts, slip = _profiles({"profiles": n, "bins": nb}, seed)
    d = counts / counts.sum(dim=1, keepdim=True)
    dd = torch.zeros_like(d)
    dd[:, 1:-1] = (d[:, 2:] - d[:, :-2]) / 2
    code = (torch.log2(torch.clamp(slip, 1, nb)) / 10.0)[:, None].expand(n, nb)
    shifted = torch.zeros_like(d)
    shifted[:, 40:] = d[:, :-40]
    x = torch.stack([d * 300, dd * 4000, code, shifted * 300], dim=1).float().contiguous()
    y = torch.cumsum(dd * 40, dim=1).float().contiguous()
    return x, y


# ------------------------------------------------------- prepare, run, work --

def prepare(case, seed):
    kind = case["kind"]
    if kind == "ring":
        t = Tracker(_ring(case["radiation"]), workloads.ring_p_central(), case["turns"])
        return {"case": case, "tracker": t, "beam": _ring_beam(case["n"], seed)}
    if kind == "ensemble":
        lat, offsets = _ring(), _ensemble_offsets(case)
        beam = _ring_beam(int(offsets[-1]), seed)
        t = Tracker(lat, workloads.ring_p_central(), case["turns"], record_history=True)
        t.load_ensemble(offsets, _ensemble_errors(lat, case["instances"], seed))
        start = torch.from_numpy(np.ascontiguousarray(beam.coords.T)).pin_memory()
        ids = torch.from_numpy(beam.ids.copy()).pin_memory()
        lost = [torch.empty(beam.n, dtype=torch.int32).pin_memory() for _ in range(2)]
        return {"case": case, "tracker": t, "start": start, "work": torch.empty_like(start).pin_memory(),
                "ids": ids, "lost": lost}
    if kind == "aperture":
        t = Tracker(_ring(), workloads.ring_p_central(), case["turns"], compact_every=4)
        return {"case": case, "tracker": t, "beam": _grid_beam(case, seed)}
    if kind == "tunes":
        t = Tracker(_ring(), workloads.ring_p_central(), case["turns"] - 1, record_tbt=True, fiducial_particles=1)
        return {"case": case, "tracker": t, "beam": _grid_beam(case, seed)}
    if kind in ("chicane", "train"):
        sizes = [case["n"]] if kind == "chicane" else _train_sizes(case)
        t = Tracker(_chicane(case), _chicane_p(), 1)
        if kind == "train":
            t.load_ensemble(np.concatenate([[0], np.cumsum(sizes)]), [])
        cols = _bunch_columns(sizes, seed)
        return {"case": case, "tracker": t, "start": cols, "cols": [torch.empty_like(c) for c in cols],
                "lost": [torch.empty(sum(sizes), dtype=torch.int32, device=DEV) for _ in range(2)]}
    if kind == "integrals":
        counts, slip = _profiles(case, seed)
        return {"case": case, "counts": counts, "slip": slip}
    net = WakeNet(bins=1024, max_batch=min(case["profiles"], 512))
    net.set_params(init_params(seed % 1000))
    x, y = _net_batch(case, seed)
    return {"case": case, "net": net, "x": x, "y": y}


def run(state):
    kind = state["case"]["kind"]
    t = state.get("tracker")
    if kind in ("ring", "aperture", "tunes"):
        res = t.track(state["beam"])
        out = {"coords": res.coords, "ids": res.ids, "lost_pass": res.lost_pass, "lost_element": res.lost_element}
        if kind == "tunes":
            out.update(t.tbt_tunes(0, state["case"]["turns"]))
        return out
    if kind == "ensemble":
        w = state["work"]
        w.copy_(state["start"])
        ids, lost = state["ids"], state["lost"]
        n = ids.numel()
        t.track_host_pointers([w.data_ptr() + 8 * n * k for k in range(6)], ids.data_ptr(), n, lost[0].data_ptr(),
                              lost[1].data_ptr())
        return {"columns": w, "lost_pass": lost[0], "lost_element": lost[1], **t.history()}
    if kind in ("chicane", "train"):
        for c, s in zip(state["cols"], state["start"]):
            c.copy_(s)
        for v in state["lost"]:
            v.fill_(-1)
        torch.cuda.current_stream().synchronize()  # the engine works on its own stream
        t.track_device(state["cols"], *state["lost"])
        return {"columns": state["cols"], "lost_pass": state["lost"][0], "lost_element": state["lost"][1]}
    if kind == "integrals":
        t1, dens, deriv = wake_batch(state["counts"], state["slip"])
        return {"t1": t1, "density": dens, "derivative": deriv}
    if kind == "forward":
        return {"y": state["net"].forward(state["x"])}
    loss = state["net"].gradients(state["x"], state["y"])
    return {"loss": loss, "gradients": state["net"].grads()}


def work(case):
    kind = case["kind"]
    if kind in ("ring", "ensemble", "aperture", "tunes"):
        per_turn = flops_per_particle_turn(workloads.fodo_ring())
        n = {"ring": lambda: case["n"], "ensemble": lambda: int(_ensemble_offsets(case)[-1]),
             "aperture": lambda: case["nx"] * case["ny"] + 1, "tunes": lambda: case["nx"] * case["ny"] + 1}[kind]()
        # about half of an aperture grid is lost within the first turns
        alive = 0.5 if kind == "aperture" else 1.0
        b, f = n * (48 + 48 + 16), n * alive * per_turn * case["turns"]
        if kind == "tunes":
            f += 4 * n * (2 * case["turns"] ** 2 + 60 * case["turns"] * 45)
        return {"bytes": b, "flops": f}
    if kind in ("chicane", "train"):
        n = case["n"] if kind == "chicane" else sum(_train_sizes(case))
        # a slice is 4 drift substeps and 3 kicks; plus the canonical conversions, the bin and the wake kick
        slice_flops = 4 * (27 + 4 * 20) + 3 * 10 + 18 + 20
        return {"bytes": n * (48 + 48 + 8), "flops": n * 4 * case["kicks"] * slice_flops}
    if kind == "integrals":
        n, nb = case["profiles"], case["bins"]
        # slippage log-uniform in [1, 2 nb]: about 0.4 nb terms of a division and an addition per bin
        return {"bytes": 4 * 8 * n * nb, "flops": n * nb * (2 * 0.4 * nb + 30)}
    rows = case["profiles"] * 1024
    conv = 2 * rows * CH * CH * TAPS
    # the first layer has IN_CH live inputs, the last one live output
    fwd = conv * (LAYERS - 2) + conv * IN_CH // CH + conv // CH
    if kind == "forward":
        return {"bytes": rows * 4 * (IN_CH + 1) + LAYERS * WSIZE * 2, "flops": fwd}
    return {"bytes": rows * 4 * (IN_CH + 1) + LAYERS * WSIZE * 6, "flops": 3 * fwd - conv * IN_CH // CH}


# ----------------------------------------------------------- exact values --
# The element maps, CSR step and network in plain torch, 64 bits.

_BETA = 1.25992104989487316477
_FRAC_D = [0.5 / (2 - _BETA), (1 - _BETA) / (2 - _BETA) / 2, (1 - _BETA) / (2 - _BETA) / 2, 0.5 / (2 - _BETA)]
_FRAC_K = [1 / (2 - _BETA), -_BETA / (2 - _BETA), 1 / (2 - _BETA)]


def _beta(dp, p0):
    p = p0 * (1 + dp)
    return p / torch.sqrt(p * p + 1)


def _exact_kick_magnet(q, e, p0):
    x, xp, y, yp, s, dp0 = q
    order4 = 1 if not e.get("N_KICKS") else max(1, math.ceil(e.get("N_KICKS") / 4))
    L, quad = e.get("L"), e.type == "KQUAD"
    knl = e.get("K1" if quad else "K2") * L / order4
    rad = E_CHARGE ** 2 * p0 ** 3 / (6 * math.pi * _eps0() * C * C * E_MASS) if e.get("SYNCH_RAD") else 0.0
    f = (1 + dp0) / torch.sqrt(1 + xp * xp + yp * yp)
    qx, qy, dp, dist = xp * f, yp * f, dp0, 0.0
    for _ in range(order4):
        for j in range(4):
            h = L / order4 * _FRAC_D[j]
            r = torch.sqrt((1 + dp) ** 2 - qx * qx - qy * qy)
            xp, yp = qx / r, qy / r
            x, y = x + xp * h, y + yp * h
            dist = dist + h * torch.sqrt(1 + xp * xp + yp * yp)
            if j == 3:
                break
            k = knl * _FRAC_K[j]
            dqx, dqy = (-k * x, k * y) if quad else (-k * (x * x - y * y) / 2, k * x * y)
            qx, qy = qx + dqx, qy + dqy
            if rad:
                r = torch.sqrt((1 + dp) ** 2 - qx * qx - qy * qy)
                sx, sy, d = qx / r, qy / r, L / order4
                f2 = (dqx / _FRAC_K[j] / d) ** 2 + (dqy / _FRAC_K[j] / d) ** 2
                new = dp - rad * (1 + dp) ** 2 * f2 * torch.sqrt(1 + sx * sx + sy * sy) * d * _FRAC_K[j]
                qx, qy, dp = qx / (1 + dp) * (1 + new), qy / (1 + dp) * (1 + new), new
    r = torch.sqrt((1 + dp) ** 2 - qx * qx - qy * qy)
    if rad:
        b0, b1 = _beta(dp0, p0), _beta(dp, p0)
        s = b1 * (s / b0 + 2 * dist / (b0 + b1))
    else:
        s = s + dist
    return [x, qx / r, y, qy / r, s, dp]


def _exact_bend_slice(x, qx, y, qy, dp, dist, rho, h, rad):
    for j in range(4):
        f = torch.sqrt((1 + dp) ** 2 - qy * qy)
        sin_phi = qx / f
        phi = torch.asin(sin_phi)
        arg = h * _FRAC_D[j] / rho + phi
        sine, cosi, cos_phi = torch.sin(arg), torch.cos(arg), torch.cos(phi)
        factor = (rho + x) * cos_phi / f * (sine / cosi - sin_phi / cos_phi)
        qx = f * sine
        y = y + qy * factor
        dist = dist + factor * (1 + dp)
        x = rho * (cos_phi / cosi - 1) + cos_phi / cosi * x
        if j == 3:
            break
        k = h * _FRAC_K[j]
        qx = qx - k * (1 + x / rho) / rho
        if rad:
            a = 1 + x / rho
            r = a / torch.sqrt((1 + dp) ** 2 - qx * qx - qy * qy)
            new = dp - rad * (1 + dp) ** 2 * k * torch.sqrt(a * a + (qx * r) ** 2 + (qy * r) ** 2)
            qx, qy, dp = qx / (1 + dp) * (1 + new), qy / (1 + dp) * (1 + new), new
    return x, qx, y, qy, dp, dist


def _eps0():
    return 1 / (4 * math.pi * 1e-7 * C * C)


def _exact_bend(q, e, p0):
    x, xp, y, yp, s, dp0 = q
    rho, h = e.get("L") / e.get("ANGLE"), e.get("L") / e.get("N_SLICES")
    rad = E_CHARGE ** 2 * p0 ** 3 / (6 * math.pi * _eps0() * C * C * E_MASS * rho ** 2) if e.get("SYNCH_RAD") else 0.0
    f = (1 + dp0) / torch.sqrt(1 + xp * xp + yp * yp)
    v = (x, xp * f, y, yp * f, dp0, torch.zeros_like(x))
    for _ in range(int(e.get("N_SLICES"))):
        v = _exact_bend_slice(*v, rho, h, rad)
    x, qx, y, qy, dp, dist = v
    r = torch.sqrt((1 + dp) ** 2 - qx * qx - qy * qy)
    return [x, qx / r, y, qy / r, _beta(dp, p0) * s / _beta(dp0, p0) + dist, dp]


def _exact_cavity(q, e, p0, t0):
    x, xp, y, yp, s, dp = q
    p = p0 * (1 + dp)
    gamma = torch.sqrt(p * p + 1)
    t = s / (C * p / gamma)
    phase = 2 * math.pi * e.get("FREQ") * (t - t0) + math.radians(e.get("PHASE"))
    gamma1 = gamma + e.get("VOLT") / (1e6 * E_MASS * C * C / E_CHARGE / 1e6) * torch.sin(phase)
    p1 = torch.sqrt(gamma1 * gamma1 - 1)
    pz = p / torch.sqrt(1 + xp * xp + yp * yp)
    ratio = pz / torch.sqrt(pz * pz + gamma1 * gamma1 - gamma * gamma)
    return [x, xp * ratio, y, yp * ratio, t * C * p1 / gamma1, (p1 - p0) / p0]


def _exact_ring(coords, lattice, p0, turns):
    q = list(torch.tensor(coords, dtype=torch.float64, device=DEV).unbind(1))
    t0 = None
    for _ in range(turns):
        for e in lattice.elements:
            if e.type == "DRIF":
                L = e.get("L")
                q = [q[0] + L * q[1], q[1], q[2] + L * q[3], q[3], q[4] + L + L / 2 * (q[1] ** 2 + q[3] ** 2), q[5]]
            elif e.type in ("KQUAD", "KSEXT"):
                q = _exact_kick_magnet(q, e, p0)
            elif e.type == "CSBEND":
                q = _exact_bend(q, e, p0)
            elif e.type == "RFCA":
                if t0 is None:
                    t0 = (q[4] / (C * _beta(q[5], p0))).mean()
                q = _exact_cavity(q, e, p0, t0)
    return torch.stack(q, dim=1).cpu().numpy()


def _filter_matrix(nb, half, derivative):
    """Straight-line fit over 2 half + 1 bins, windows shifted inwards at the ends: value or slope at the bin."""
    m = np.zeros((nb, nb))
    width = min(2 * half + 1, nb)
    for b in range(nb):
        lo = min(max(b - half, 0), nb - width)
        t = np.arange(lo, lo + width) - b
        a = np.linalg.pinv(np.stack([np.ones(width), t], axis=1))
        m[b, lo:lo + width] = a[1] if derivative else a[0]
    return torch.tensor(m, device=DEV)


def _exact_wake(counts, dct, slip_bins, smooth, slope):
    """Density, derivative, T1 and the slippage in bins of histograms [n][nb] (transient wake, trapezoid rule)."""
    n, nb = counts.shape
    sm = torch.clamp(counts @ smooth.T, min=0)
    hist = sm * (counts.sum(1, keepdim=True) / sm.sum(1, keepdim=True)) / dct
    deriv = hist @ slope.T
    d = torch.clamp(torch.floor(slip_bins), 0, nb).long()[:, None]
    i = torch.arange(nb, device=DEV)[None, :]
    last = torch.minimum(i + d, torch.full_like(i, nb - 1))  # last bin of the integral
    t1 = torch.zeros_like(hist)
    for k in range(1, min(nb - 1, int(d.max())) + 1):
        t1[:, :nb - k] += torch.where(k <= d, deriv[:, k:] / (dct * k) ** (1 / 3), torch.zeros_like(deriv[:, k:]))
    inside = (d > 0) & (i + 1 < nb)
    nxt = torch.cat([deriv[:, 1:], torch.zeros_like(deriv[:, :1])], dim=1)
    first = nxt / dct ** (1 / 3) / 2
    final = torch.gather(deriv, 1, last) / torch.clamp(dct * (last - i).double(), min=1e-300) ** (1 / 3)
    t1 += torch.where(inside, 0.3 * dct ** (2 / 3) * (2 * nxt + 3 * deriv) / dct, torch.zeros_like(t1))
    t1 -= torch.where(last - i > 1, (first + final) / 2, torch.zeros_like(t1))
    return hist, deriv, t1, d


def _exact_bunch(cols, lattice, p0):
    x, xp, y, yp, s, dp = [c.clone() for c in cols]
    n, charge = x.numel(), lattice.elements[0].get("TOTAL")
    wake = None

    def kick(pos, lower, dct, table, scale):
        f = (pos - lower) / dct
        b = f.long()
        ok = (b >= 0) & (b < table.numel() - 1)
        b = torch.clamp(b, 0, table.numel() - 2)
        f = f - b
        return torch.where(ok, ((1 - f) * table[b] + f * table[b + 1]) / p0 * scale, torch.zeros_like(f))

    def span(ct):
        lo, hi = ct.min(), ct.max()
        mid, r = (lo + hi) / 2, (hi - lo) * 1.2
        return mid - r / 2, (mid + r / 2) - (mid - r / 2)

    for e in lattice.elements:
        if e.type == "CSRDRIFT":
            L = e.get("L")
            table, dct, s0, ds0 = wake
            x, y = x + xp * L / 2, y + yp * L / 2
            ct = (s + L / 2 * torch.sqrt(1 + xp * xp + yp * yp)) / _beta(dp, p0)
            s0 = s0 + L / 2
            dp = dp + kick(ct, s0, dct, table, L / ds0)
            s = ct * _beta(dp, p0)
            x, y, s = x + xp * L / 2, y + yp * L / 2, s + L / 2 * torch.sqrt(1 + xp * xp + yp * yp)
            wake = (table, dct, s0 + L / 2, ds0)
        elif e.type == "CSRCSBEND":
            kicks, nb, L = int(e.get("N_SLICES")), int(e.get("BINS")), e.get("L")
            # an element bent the other way is the same bend with x turned over
            sg, rho = math.copysign(1.0, e.get("ANGLE")), L / abs(e.get("ANGLE"))
            x, xp, y, yp = sg * x, sg * xp, sg * y, sg * yp
            half = int(e.get("SG_HALFWIDTH"))
            smooth, slope = _filter_matrix(nb, half, False), _filter_matrix(nb, half, True)
            const = 2 * charge / n * E_CHARGE / (3 * rho * rho) ** (1 / 3) / (4 * math.pi * _eps0() * E_MASS * C * C)
            b0 = _beta(dp, p0)
            ct, table = s / b0, None
            lower = dct = 0.0
            for k in range(kicks):
                if table is not None:
                    dp = dp + kick(ct, lower, dct, table, 1 + x / rho)
                f = (1 + dp) / torch.sqrt(1 + xp * xp + yp * yp)
                x, qx, y, qy, _, dist = _exact_bend_slice(x, xp * f, y, yp * f, dp, torch.zeros_like(x), rho,
                                                          L / kicks, 0.0)
                r = torch.sqrt((1 + dp) ** 2 - qx * qx - qy * qy)
                xp, yp, ct = qx / r, qy / r, ct + dist / b0
                lower, r = span(ct)
                dct = r / nb
                counts = torch.bincount(torch.clamp(((ct - lower) / dct).long(), 0, nb - 1), minlength=nb).double()
                slip = rho * (abs(e.get("ANGLE")) * (k + 1) / kicks) ** 3 / 24
                hist, _, t1, d = _exact_wake(counts[None], dct, (slip / dct)[None], smooth, slope)
                d, d4 = int(d), int(min(4 * slip / dct, nb))
                h = torch.cat([hist[0], torch.zeros(nb, dtype=torch.float64, device=DEV)])
                table = const * L / kicks * (t1[0] - (h[d:d + nb] - h[d4:d4 + nb]) / slip ** (1 / 3))
            dp = dp + kick(ct, lower, dct, table, 1 + x / rho)
            wake = (table, dct, span(ct)[0], L / kicks)
            s = ct * _beta(dp, p0)
            x, xp, y, yp = sg * x, sg * xp, sg * y, sg * yp
    return [x, xp, y, yp, s, dp]


def _exact_net(params, x):
    h = torch.nn.functional.pad(x.double(), (0, 0, 0, CH - IN_CH))
    w = params[:LAYERS * WSIZE].reshape(LAYERS, TAPS, CH, CH)
    b = params[LAYERS * WSIZE:].reshape(LAYERS, CH)
    for k, d in enumerate(DILATIONS):
        out = 1 if k == LAYERS - 1 else CH
        z = b[k, :out, None]
        pad = torch.nn.functional.pad(h, (2 * d, 2 * d))
        for t in range(TAPS):
            z = z + torch.matmul(w[k, t, :out], pad[:, :, t * d:t * d + h.shape[2]])
        h = z if k == LAYERS - 1 else torch.nn.functional.gelu(z)
    return h[:, 0]


def exact(case, seed):
    """What run() returns for these inputs in 64 bits; None where plain torch takes too long (many turns) or where
    the value hangs on the path taken (Stupakov's root search)."""
    kind = case["kind"]
    if kind == "ring" and case["turns"] <= 10:
        beam, lattice = _ring_beam(case["n"], seed), _ring(case["radiation"])
        kept = np.full(beam.n, -1, dtype=np.int32)
        return {"coords": _exact_ring(beam.coords, lattice, workloads.ring_p_central(), case["turns"]),
                "ids": beam.ids, "lost_pass": kept, "lost_element": kept}
    if kind == "chicane" and not case["stupakov"] or kind == "train":
        sizes = [case["n"]] if kind == "chicane" else _train_sizes(case)
        lattice, parts = _chicane(case), []
        for cols in zip(*[c.split(sizes) for c in _bunch_columns(sizes, seed)]):
            parts.append(_exact_bunch(cols, lattice, _chicane_p()))
        kept = torch.full((sum(sizes),), -1, dtype=torch.int32)
        return {"columns": [torch.cat([p[k] for p in parts]) for k in range(6)], "lost_pass": kept,
                "lost_element": kept}
    if kind == "integrals":
        counts, slip = _profiles(case, seed)
        hist, deriv, t1, _ = _exact_wake(counts, 1.0, slip, _filter_matrix(case["bins"], 2, False),
                                         _filter_matrix(case["bins"], 2, True))
        return {"t1": t1, "density": hist, "derivative": deriv}
    if kind in ("forward", "gradients"):
        params = torch.tensor(init_params(seed % 1000), dtype=torch.float64, device=DEV,
                              requires_grad=kind == "gradients")
        x, y = _net_batch(case, seed)
        if kind == "forward":
            return {"y": torch.cat([_exact_net(params, x[k:k + 64]) for k in range(0, len(x), 64)])}
        loss = 0.0
        for k in range(0, len(x), 32):
            part = ((_exact_net(params, x[k:k + 32]) - y[k:k + 32].double()) ** 2).sum() / y.numel()
            part.backward()
            loss += part.item()
        return {"loss": loss, "gradients": params.grad.cpu().numpy()}
    return None
