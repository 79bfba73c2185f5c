"""The conv forward's per-position event lists: sizes at the edges of its tiles, rounds of 64 events and groups of 8,
against the float64 oracle (counts up to the conditioning of grazing neurons, times as in test_gpu_conv_pool)."""
import numpy as np
import pytest
import torch

from tests._helpers import conditioned_reference, count_mismatches, leading_mask
from tests.test_gpu_conv_pool import run_conv

pytestmark = pytest.mark.gpu


def _input(counts, X, Y, C, k, seed):
    rng = np.random.default_rng(seed)
    t = np.full((len(counts), X * Y * C, k), np.inf, np.float32)
    for s, m in enumerate(counts):
        slots = rng.permutation(X * Y * C * k)[:m]
        tm = rng.uniform(0, 0.1, m).astype(np.float32)
        for j in np.unique(slots // k):
            own = np.sort(tm[slots // k == j])
            t[s, j, :own.size] = own
    return t


@pytest.mark.parametrize("X,Y,C,fx,fy,C_out,k,K_post,counts", [
    (5, 5, 1, 5, 5, 1, 3, 1, [0, 1, 2, 75]),           # one position, one channel, K 1
    (9, 6, 2, 3, 2, 7, 3, 4, [8, 9, 63, 64, 65, 300]),  # partial tiles, rounds of 64
    (12, 7, 3, 5, 3, 40, 4, 10, [16, 17, 512, 513, 900]),
    (7, 7, 4, 2, 2, 33, 5, 40, [128, 129, 980]),        # even filter rows, K over a warp
    (6, 6, 2, 3, 3, 600, 2, 3, [144, 7]),               # more channels than a tile's threads
    (8, 8, 40, 5, 5, 64, 1, 3, [700, 64]),              # filters larger than shared memory
])
def test_conv_forward_lists_against_the_oracle(cuda, X, Y, C, fx, fy, C_out, k, K_post, counts):
    t = _input(counts, X, Y, C, k, seed=X * 100 + C_out)
    rng = np.random.default_rng(C_out)
    filt = rng.uniform(-1, 1, (C_out, fx, fy, C)).astype(np.float32)
    args = (np.float32(0.13), 0.3, 0.3, K_post, np.float32(0.2))
    ours, _ = run_conv(t, filt, (X, Y, C), K_post, 0.13, 0.3, 0.2)
    o64, bounds, sens = conditioned_reference(t, filt, *args, conv=(X, Y, C))
    assert ours[0].sum() > 0 or C_out == 1  # (the one neuron of the first case stays below its threshold)
    _, unexplained = count_mismatches(ours[0], o64[0], bounds)
    assert unexplained == 0
    valid = leading_mask(ours[0], K_post)
    assert np.isinf(ours[3][~valid]).all() and np.isinf(ours[4][~valid]).all()
    same = (ours[0] == o64[0])[:, :, None] & leading_mask(o64[0], K_post)
    e = np.abs(ours[3][same] - o64[3][same])
    assert np.all(e <= 1e-5 * np.abs(o64[3][same]) + 1e-5 * 0.26 + 20 * sens[same])
