"""The event sort of times on a coarse grid, at both sides of the line between ranking by comparison and the radix sort (48 comparisons
per item), with spike counts: slots past a count hold finite leftovers, some below it no spike. And a coarse grid may not cost
more than a few times what as many distinct times do."""
import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counted", [False, True])
@pytest.mark.parametrize("n_pre,k", [(301, 7), (33, 40), (900, 1), (517, 30), (5000, 14)])  # the last: 32-bit slots, global scratch
@pytest.mark.parametrize("steps", [400, 100, 60, 40, 3])
def test_coarse_times(cuda, n_pre, k, steps, counted):
    rng = np.random.default_rng(steps + k)
    B = 3
    t = (rng.integers(0, steps, (B, n_pre, k)) * np.float32(0.001)).astype(np.float32)
    n = rng.integers(0, k + 1, (B, n_pre))
    n[1, : n_pre // 2] = 0
    spike = np.arange(k) < n[..., None]
    hole = spike & (rng.random(t.shape) < 0.1)
    if counted:
        t[hole] = np.inf
        spike &= ~hole
    else:
        t[~spike] = np.inf
    tt = torch.as_tensor(t).cuda()
    ev = K.sort_events(tt, 0.13, 0.26, pre_counts=torch.as_tensor(n.astype(np.int32)).cuda() if counted else None)
    for s in range(B):
        slots = np.flatnonzero(spike[s].reshape(-1))
        want = slots[np.argsort(t[s].reshape(-1)[slots], kind="stable")]
        assert int(ev.counts[s]) == want.size > 150
        assert np.array_equal(ev.slots[s, :want.size].cpu().numpy(), want)
        assert np.array_equal(ev.events[s, :want.size, 0].cpu().numpy(), t[s].reshape(-1)[want])


def test_coarse_times_are_no_trap(cuda):
    rng = np.random.default_rng(0)
    t = np.sort(np.where(rng.random((54, 492, 16)) < 0.7, rng.uniform(0, 0.1, (54, 492, 16)), np.inf), -1).astype(np.float32)

    def run(x):
        x = torch.as_tensor(x).cuda()
        ev, best = K.sort_events(x, 0.13, 0.26), np.inf
        for _ in range(5):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(500_000)
            start.record()
            K.sort_events(x, 0.13, 0.26, out=ev)
            end.record()
            end.synchronize()
            best = min(best, start.elapsed_time(end))
        return best

    fine, coarse = run(t), run(np.where(np.isfinite(t), np.floor(t * 200) / 200, t).astype(np.float32))
    assert coarse < 4 * fine, (coarse, fine)
