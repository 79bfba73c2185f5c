"""The event sort on time distributions that its bucket path likes and dislikes: the order is by time, ties by slot,
whatever the path (ranks of small samples, time buckets, the radix sort of crowded times, the global scratch)."""
import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K

pytestmark = pytest.mark.gpu


def _times(kind, rng, n):
    t = rng.uniform(0.0, 0.2, n)
    if kind == "ties":
        t = np.round(t, 3)
    elif kind == "equal":
        t = np.full(n, 0.125)
    elif kind == "crowded":  # one outlier stretches the range: nearly every item falls into one bucket
        t = 0.1 + 1e-6 * t
        t[: max(1, n // 1000)] = 50.0
    elif kind == "signs":
        t = np.concatenate([-t[: n // 2], t[n // 2:]])
        t[:4] = (0.0, -0.0, -3e38, 3e38)[: min(4, n)]
    return t.astype(np.float32)


@pytest.mark.parametrize("kind", ["uniform", "ties", "equal", "crowded", "signs"])
@pytest.mark.parametrize("n_pre,k,counts", [
    (50, 1, [1, 2, 3, 50]), (37, 5, [4, 7, 185, 0]), (90, 9, [255, 256, 257, 810]),
    (301, 7, [300, 513, 2100, 2107]), (400, 40, [383, 385, 6000, 16000]), (2500, 30, [9000, 40000, 100, 75000])])
def test_order_is_by_time_then_slot(cuda, kind, n_pre, k, counts):
    rng = np.random.default_rng(n_pre + k)
    t = np.full((len(counts), n_pre * k), np.inf, np.float32)
    for s, m in enumerate(counts):
        t[s, rng.permutation(n_pre * k)[:m]] = _times(kind, rng, m)
    tt = torch.tensor(t.reshape(len(counts), n_pre, k), device="cuda")
    full = torch.full((len(counts), n_pre), k, dtype=torch.int32, device="cuda")
    order = torch.tensor(rng.permutation(len(counts)).astype(np.int32), device="cuda")
    for kw in ({}, {"pre_counts": full}, {"pre_counts": full, "sample_order": order}):
        ev = K.sort_events(tt, 0.13, 0.26, **kw)
        got, slots = ev.events.cpu().numpy(), ev.slots.cpu().numpy()
        assert np.array_equal(ev.counts.cpu().numpy(), counts)
        for s, m in enumerate(counts):
            valid = np.flatnonzero(np.isfinite(t[s]))
            key = t[s, valid]
            # -0 sorts before +0, as their bits do
            want = valid[np.lexsort((valid, ~np.signbit(key), key))]
            assert np.array_equal(slots[s, :m], want)
            assert np.array_equal(got[s, :m, 0].view(np.uint32), t[s, want].view(np.uint32))
            assert np.array_equal(got[s, :m, 1].copy().view(np.int32), want // k)
            if ev.bucketed is not None:
                b = (want // k) // ev.bucket_width
                by = np.argsort(b, kind="stable")
                bt = ev.bucketed[s, :m].cpu().numpy()
                assert np.array_equal(bt[:, 1].copy().view(np.int32), (want // k)[by])
                assert np.array_equal(bt[:, 0].view(np.uint32), t[s, want][by].view(np.uint32))
                off = ev.bucket_offsets[s].cpu().numpy()
                assert np.array_equal(off, np.concatenate([[0], np.cumsum(np.bincount(b, minlength=off.size - 1))]))
