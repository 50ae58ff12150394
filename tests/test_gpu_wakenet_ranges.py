"""Gradients of the wake network where its pre-activations leave the range in
which GELU' comes from a table (|z| < 8, with one value below 2^-25): vanishing,
ordinary and large activations, and inputs whose first layers are exactly
zero, against the numpy oracle.  Tolerance: z, a and the gradients are stored
in BF16 (2^-9 each), three roundings a layer over six layers, 3.5e-2."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1e-6, 1e-3, 1.0, 30.0])
@pytest.mark.parametrize("zeros", [False, True])
def test_gradients_over_the_range_of_z(scale, zeros):
    import torch
    import wakenet_oracle as wo
    from elegant_b200.wakenet import WakeNet, init_params
    rng = np.random.default_rng(5)
    params = init_params(5, out_scale=1.0)
    weights = wo.LAYERS * wo.WSIZE
    params[weights:] = 0 if zeros else scale * rng.normal(0, 0.05, wo.LAYERS * wo.CH).astype(np.float32)
    params[weights + 5 * 64 + 1:] = 0  # output channels 1..63 are not live
    inputs = (scale * rng.normal(0, 1, (3, 4, 256))).astype(np.float32)
    if zeros:
        inputs[1] = 0
        inputs[2, :, 100:] = 0
    targets = rng.normal(0, 1, (3, 256)).astype(np.float32)
    with WakeNet(bins=256, max_batch=4) as net:
        net.set_params(params)
        loss = net.gradients(torch.tensor(inputs, device="cuda"), torch.tensor(targets, device="cuda"))
        got = net.grads().astype(np.float64)
    ref_loss, ref = wo.loss_and_gradients(params, inputs, targets, net.dilations)
    assert abs(loss - ref_loss) < 3.5e-2 * ref_loss
    for layer in range(wo.LAYERS):
        for sl in (slice(layer * wo.WSIZE, (layer + 1) * wo.WSIZE),
                   slice(weights + layer * wo.CH, weights + (layer + 1) * wo.CH)):
            a, b = got[sl], ref[sl]
            assert np.linalg.norm(a - b) <= 3.5e-2 * np.linalg.norm(b), (layer, sl)
