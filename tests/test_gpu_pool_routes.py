"""The 2x2 spike pooling at both sides of the line between its two kernels (one slot per child; up to 40 slots; more, with few neurons
and with many), against a stable sort of the four children's slots."""
import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,X,Y,C,k", [
    (1, 2, 2, 1, 1), (40, 13, 8, 21, 1), (3, 6, 6, 5, 2), (2, 9, 4, 7, 40), (60, 20, 18, 6, 40), (2, 4, 4, 5, 41), (52, 20, 24, 5, 41),
    (3, 4, 5, 3, 200), (34, 12, 10, 6, 200), (1, 2, 3, 2, 1024)])
def test_pool_is_a_stable_sort(cuda, B, X, Y, C, k):
    rng = np.random.default_rng(k + B)
    n = rng.integers(0, k + 1, (B, X * Y * C))
    n[:, rng.random(X * Y * C) < 0.2] = k
    t = np.where(np.arange(k) < n[..., None], np.sort(rng.integers(0, 4 * k, (B, X * Y * C, k)) * np.float32(0.01), -1), np.inf)
    t = torch.as_tensor(t.astype(np.float32)).cuda()
    counts = torch.as_tensor(n.astype(np.int32)).cuda()
    on, ot, oi = K.aggregate_spikes_conv(counts, t, (X, Y, C))
    Xo, Yo = X // 2, Y // 2
    slot = torch.arange(B * X * Y * C * k, device="cuda").reshape(B, X, Y, C, k)[:, :2 * Xo, :2 * Yo]

    def children(v):  # (B, Xo * Yo * C, 4 k), children (0, 0), (0, 1), (1, 0), (1, 1)
        v = v.reshape(B, Xo, 2, Yo, 2, C, -1).permute(0, 1, 3, 5, 2, 4, 6)
        return v.reshape(B, Xo * Yo * C, -1)

    want, order = torch.sort(children(t.reshape(B, X, Y, C, k)[:, :2 * Xo, :2 * Yo]), dim=-1, stable=True)
    assert torch.equal(ot, want)
    assert torch.equal(oi.long(), torch.gather(children(slot), -1, order))
    assert torch.equal(on, children(counts.reshape(B, X, Y, C, 1)[:, :2 * Xo, :2 * Yo]).sum(-1).int())
