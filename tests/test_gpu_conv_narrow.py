"""The conv forward on grids past a wave with few neurons per tile, which take shorter lists and fewer warps, against the same samples in
small batches, which take the full ones: bit for bit, at the edges of a round of 32 and 64 kept events, with 1 to 10 filters, partial
tiles, full spike buffers; and filters that several threads stage in many copies (9 x 9 x 40)."""
import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K
from tests.test_gpu_conv_lists import _input
from tests.test_gpu_conv_pool import cu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("X,Y,C,fx,fy,C_out,k,K_post,B", [
    (12, 12, 2, 3, 3, 1, 2, 4, 140), (12, 12, 2, 3, 3, 3, 2, 10, 140), (13, 11, 1, 2, 3, 10, 3, 33, 160), (28, 28, 1, 5, 5, 2, 1, 5, 40),
    (10, 10, 40, 9, 9, 4, 1, 3, 3)])
def test_batch_against_slices(cuda, X, Y, C, fx, fy, C_out, k, K_post, B):
    cap = X * Y * C * k
    counts = ([0, 1, 31, 32, 33, 63, 64, 65, 66, 97, 128, 129, cap] * B)[:B]
    t = cu(_input([min(c, cap) for c in counts], X, Y, C, k, seed=C_out))
    rng = np.random.default_rng(C_out)
    filt = cu(rng.uniform(-0.2, 1.0, (C_out, fx, fy, C)).astype(np.float32))
    tau32, _, _ = K.lif_constants(0.13, 0.05, 0.05)

    def run(x):
        ev = K.sort_events(x, np.float32(0.13), tau32, bucketed=False)
        out = (torch.zeros((x.shape[0], (X - fx + 1) * (Y - fy + 1) * C_out), dtype=torch.int32, device="cuda"),
               *(torch.zeros((x.shape[0], (X - fx + 1) * (Y - fy + 1) * C_out, K_post), device="cuda") for _ in range(4)))
        return K.conv_forward(ev, filt, (X, Y, C), K_post, 0.13, 0.05, 0.05, 0.2, outs=out)

    whole = run(t)
    assert (int(whole[0].max()) == K_post or K_post > 32) and int(whole[0].min()) == 0 < int(whole[0].max())
    step = 10 if B > 10 else 1
    for lo in range(0, B, step):
        for w, p in zip(whole, run(t[lo:lo + step].contiguous())):
            assert torch.equal(w[lo:lo + step], p)
