"""The weight gradient of narrow layers (a bucket's pre neurons split among the warps of a CTA) against the kernel over the
unbucketed events, whose order of terms it reproduces: equal bit for bit. Layers at the edges of a warp, the last bucket partly
filled, bucket sizes around a batch of 32 events, one sample per group and all samples in one."""
import dataclasses

import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("group", [1, 2, 40])
@pytest.mark.parametrize("n_pre,n_post,k_pre,k_post,batch", [
    (1, 1, 1, 1, 3),
    (31, 32, 5, 30, 40),
    (33, 10, 40, 7, 35),      # 1280 events in a full bucket
    (800, 31, 2, 12, 67),
    (129, 3, 64, 33, 5),      # spike buffers past a warp's lanes
])
def test_narrow_gradient_is_bit_identical(cuda, n_pre, n_post, k_pre, k_post, batch, group):
    rng = np.random.default_rng(n_pre + n_post)
    t = np.sort(np.where(rng.random((batch, n_pre, k_pre)) < 0.6, rng.uniform(0, 0.05, (batch, n_pre, k_pre)), np.inf), axis=-1)
    t[batch // 2] = np.inf  # a sample without events
    theta, tau_s = 0.05, 0.1
    tau, c, dtt = K.lif_constants(tau_s, theta, theta)
    w = torch.as_tensor(rng.uniform(-0.3, 1.0, (n_post, n_pre)).astype(np.float32)).cuda()
    ev = K.sort_events(torch.as_tensor(t.astype(np.float32)).cuda(), tau_s, tau, bucket_width=K.BUCKET_WIDTH)
    n, a, x, ts, z = K.lif_forward_fc(ev, K.transpose_weights(w), n_post, k_post, tau_s, theta, theta, 0.2)
    err = torch.as_tensor(rng.normal(size=ts.shape).astype(np.float32)).cuda()
    tabs = K.backward_prep(ts, a, x, z, err, c, tau, dtt)
    plain = dataclasses.replace(ev, bucketed=None, bucket_offsets=None)
    kw = dict(per_sample=True) if group == 1 else dict(per_sample=False, reduce="sum", group=group)
    got = K.weights_gradient(ev, ts, tabs, n_pre, **kw)
    want = K.weights_gradient(plain, ts, tabs, n_pre, **kw)
    assert n_pre == 1 or (int(n.sum()) > 0 and float(want.abs().max()) > 0)  # one event makes no spike
    assert torch.equal(got, want)
