"""The pooling forward (places of the slots counted in shared memory) against a merge written out: equal in every slot. One
slot per child, more slots than lanes, the largest buffer that fits and one more, an odd input, children with equal times,
-inf, NaN after the spikes, finite values past an empty slot and trains out of order."""
import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K

pytestmark = pytest.mark.gpu


def _merge(n, t, X, Y, C, k):
    B, Xo, Yo = len(n), X // 2, Y // 2
    on = np.zeros((B, Xo * Yo * C), np.int32)
    ot = np.zeros((B, Xo * Yo * C, 4 * k), np.float32)
    oi = np.zeros((B, Xo * Yo * C, 4 * k), np.int32)
    for s in range(B):
        for o in range(Xo * Yo * C):
            c, yo, xo = o % C, o // C % Yo, o // C // Yo
            kids = [((2 * xo + (h >> 1)) * Y + 2 * yo + (h & 1)) * C + c for h in range(4)]
            on[s, o] = n[s, kids].sum()
            cnt = [next((q for q in range(k) if not t[s, j, q] < np.inf), k) for j in kids]
            pos, seq = [0] * 4, []
            while any(pos[h] < cnt[h] for h in range(4)):
                h = min((h for h in range(4) if pos[h] < cnt[h]), key=lambda h: (t[s, kids[h], pos[h]], h))
                seq.append((kids[h], pos[h]))
                pos[h] += 1
            seq += [(kids[h], q) for h in range(4) for q in range(cnt[h], k)]
            ot[s, o] = [t[s, j, q] for j, q in seq]
            oi[s, o] = [(s * X * Y * C + j) * k + q for j, q in seq]
    return on, ot, oi


@pytest.mark.parametrize("B,X,Y,C,k", [(3, 2, 2, 1, 1), (2, 5, 7, 3, 8), (2, 4, 4, 2, 33), (5, 6, 4, 40, 10), (1, 2, 2, 1, 1023),
                                       (1, 2, 2, 1, 1024)])
@pytest.mark.parametrize("kind", ["ordered", "odd"])
def test_places_equal_the_merge(cuda, B, X, Y, C, k, kind):
    rng = np.random.default_rng(k + X)
    t = rng.integers(0, 20 + k, (B, X * Y * C, k)).astype(np.float32) / 64  # many equal times
    n = rng.integers(0, k + 1, (B, X * Y * C)).astype(np.int32)
    t[np.arange(k) >= n[..., None]] = np.inf
    t.sort(axis=-1)
    if kind == "odd":
        t[0, 0] = rng.permutation(t[0, 0])              # out of order, finite values past an empty slot
        t[-1, -1, 0] = -np.inf
        t[-1, 0, k // 2] = np.nan
    got = K.aggregate_spikes_conv(torch.as_tensor(n).cuda(), torch.as_tensor(t).cuda(), np.array([X, Y, C]))
    for g, w in zip(got, _merge(n, t, X, Y, C, k)):
        np.testing.assert_array_equal(g.cpu().numpy().reshape(w.shape), w)
