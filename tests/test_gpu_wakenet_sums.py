"""Bias gradients of the wake network against 64-bit sums of the same BF16
gradients of the pre-activations.

The last layer's are the residuals, y - target rounded to BF16.  With GELU' = 1
in the layer before (its z is 30 everywhere) and one centre tap of a power of
two per channel, that layer's are the same values, scaled.  Sizes: one tile, one
more tile than blocks, a remainder, and a large batch.

Tolerances.  "one binade": residuals in [1, 2), multiples of 2^-7, so that sums
of 32 bins are exact in FP32 and what is left is the rounding of the result,
2^-24.  "many binades": 31 roundings of 2^-24 in a sum of 32 bins, relative to
the sum of magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,bins", [(1, 128), (149, 128), (37, 1024), (300, 1024), (512, 1024)])
@pytest.mark.parametrize("spread", ["one binade", "many binades"])
def test_bias_gradients_are_the_sums(n, bins, spread):
    import torch
    from elegant_b200.wakenet import CH, LAYERS, TAPS, WSIZE, WakeNet, init_params
    weights = LAYERS * WSIZE
    p = init_params(3)
    p[4 * WSIZE:5 * WSIZE] = 0
    p[weights + 4 * CH:weights + 5 * CH] = 30
    last = p[5 * WSIZE:6 * WSIZE].reshape(TAPS, CH, CH)
    last[:] = 0
    scale = 2.0 ** -(np.arange(CH) % 5)
    last[2, 0, :] = scale
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((n, 4, bins), generator=g, device="cuda")
    u = torch.rand((n, bins), generator=g, device="cuda")
    resid = 1 + torch.floor(u * 128) / 128 if spread == "one binade" else torch.exp2(12 * u - 6)
    with WakeNet(bins=bins, max_batch=n) as net:
        net.set_params(p)
        y = net.forward(x)
        target = y - resid
        net.gradients(x, target)
        got = net.grads().astype(np.float64)[weights:]
    d = (y - target).bfloat16().double()
    total, magnitude = d.sum().item(), d.abs().sum().item()
    to_mean = float(np.float32(2.0 / (n * bins)))
    tol = (2.0 ** -24 if spread == "one binade" else 32 * 2.0 ** -24) * 1.01
    assert abs(got[5 * CH] - total * to_mean) <= tol * magnitude * to_mean
    assert np.all(got[5 * CH + 1:] == 0)
    assert np.all(np.abs(got[4 * CH:5 * CH] - total * to_mean * scale) <= tol * magnitude * to_mean * scale)
