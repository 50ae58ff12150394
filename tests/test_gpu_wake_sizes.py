"""The batched wake integral against the CPU restatement, bit for bit, where
its paths meet: filter windows up to 17 bins (weights as an argument) and
beyond (a table), fewer bins than a window, bin counts around the block's
four bins per thread, empty and full integrals, and counts too small for the
quotients by stored reciprocals."""
import numpy as np
import pytest

from elegant_b200.wake_surrogate import wake_batch
from reforacle import PortOracle

pytestmark = pytest.mark.gpu


def _check(counts, slip, **kw):
    import torch
    t1, dens, deriv = wake_batch(torch.tensor(counts, device="cuda"), torch.tensor(slip, device="cuda"), **kw)
    port = PortOracle("b2e")
    for k in range(len(counts)):
        a, h, d = port.wake_t1(counts[k], slip[k], **kw)
        for got, want in ((dens, h), (deriv, d), (t1, a)):
            assert np.array_equal(got[k].cpu().numpy(), want, equal_nan=True)


def _profiles(nb, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(0, 1000, (4, nb)) * (rng.uniform(size=(4, nb)) < 0.9)
    c[1] = np.round(c[1])
    c[2, nb // 2:] = 0
    return c, np.array([0.5, 1.0, 2.7 + nb / 3, 5.0 * nb])


@pytest.mark.parametrize("nb", [2, 3, 5, 17, 255, 256, 257, 1023, 1024, 1025, 2100])
@pytest.mark.parametrize("half", [0, 1, 8, 9])
def test_sizes(nb, half):
    _check(*_profiles(nb, nb + half), sg_half=half, sg_order=min(half, 2) or 1)


@pytest.mark.parametrize("trapz", [True, False])
@pytest.mark.parametrize("steady", [True, False])
def test_forms(trapz, steady):
    _check(*_profiles(700, 9), sg_half=2, trapz=trapz, steady=steady)


def test_extreme_counts():
    c, slip = _profiles(300, 4)
    c[0] *= 1e-90
    c[1] *= 1e250
    c[2, 7] = np.inf
    c[3] = 0
    _check(c, slip, sg_half=2)
