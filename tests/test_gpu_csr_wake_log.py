"""The wake log of a train holds zeros for the bunches that have no wake on a
kick, whatever the memory held before."""
import numpy as np
import pytest

from elegant_b200 import Beam, Tracker, workloads as w

pytestmark = pytest.mark.gpu
P0 = 1000 / 0.51099895


@pytest.mark.parametrize("stupakov", [False, True])
@pytest.mark.parametrize("sizes", [[300, 1, 200], [1, 0, 400], [2, 1, 1, 1]])
def test_bunches_without_a_wake_log_zeros(sizes, stupakov):
    bins, kicks = 60, 3
    lat = w.chicane(bins=bins, n_kicks=kicks, stupakov=stupakov, drift={"N_KICKS": 2})
    offsets = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(offsets[-1])
    c = w.chicane_beam(n, seed=5).coords
    ids = np.arange(1, n + 1)
    # memory that the log will get, full of other numbers
    import torch
    dirty = [torch.full((4 * kicks * len(sizes) * bins,), 3.25, dtype=torch.float64, device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    del dirty
    torch.cuda.empty_cache()
    with Tracker(lat, P0, 1) as t:
        t.load_ensemble(offsets, [])
        t.track(Beam(c, ids))
        wakes = t.csr_wakes(1_000_000).reshape(4 * kicks, len(sizes), bins)
    for k, size in enumerate(sizes):
        assert wakes[:, k].any() == (size > 1) and np.isfinite(wakes[:, k]).all()
