"""Event lists into spike trains: every slot of every row, for rows of one slot to more than a CTA's threads, one neuron to more than the
shared-memory counts hold, one sample and more than 608 (fewer warps per sample), against a plain loop."""
import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,N,k,S", [(1, 1, 1, 3), (3, 700, 1, 500), (2, 5, 2, 40), (609, 33, 1, 20), (700, 7, 31, 60), (2, 40, 33, 900),
                                     (4, 3, 600, 1500), (2, 9000, 3, 1100), (610, 2, 129, 10)])
def test_every_slot(cuda, B, N, k, S):
    rng = np.random.default_rng(N + k)
    idx = rng.integers(0, N, (B, S)).astype(np.int32)
    idx[B // 2, S // 2:] = -1  # a sample that ends early
    tm = np.sort(rng.uniform(0, 0.2, (B, S)).astype(np.float32), axis=1)
    want_t, want_n = np.full((B, N, k), np.inf, np.float32), np.zeros((B, N), np.int32)
    for s in range(B):
        for j, t in zip(idx[s], tm[s]):
            if j < 0:
                break
            if want_n[s, j] < k:
                want_t[s, j, want_n[s, j]] = t
                want_n[s, j] += 1
    out_t, out_n = K.convert_to_spike_per_neuron(torch.as_tensor(idx).cuda(), torch.as_tensor(tm).cuda(), N, k)
    assert np.array_equal(out_n.cpu().numpy(), want_n)
    assert np.array_equal(out_t.cpu().numpy(), want_t)
