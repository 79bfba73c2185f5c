"""The position-grouped conv backward (events of a position on the lanes) against the event-ordered cluster kernel, up to
the order of the sums (1e-5 of the largest entry, as in test_gpu_conv_pool): spike buffers of every search depth, layers
of one tap and of more taps than a warp, positions of more events than a batch, filters outside shared memory."""
import dataclasses

import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K
from tests.test_gpu_conv_lists import _input
from tests.test_gpu_conv_pool import cu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("want_pre", [True, False])
@pytest.mark.parametrize("X,Y,C,fx,fy,C_out,k,K_post,theta,counts", [
    (4, 4, 2, 1, 1, 1, 3, 1, 0.05, [0, 5, 90]),            # one tap
    (7, 6, 3, 3, 2, 7, 4, 5, 0.1, [33, 400, 1]),            # search of three steps
    (9, 9, 4, 5, 5, 24, 6, 10, 0.1, [700, 31, 32]),         # more taps than a warp, partial last warp
    (6, 5, 3, 3, 3, 9, 8, 16, 0.03, [600, 64]),
    (6, 5, 3, 3, 3, 9, 10, 32, 0.01, [800, 10]),            # full rows of 32 spikes
    (5, 5, 2, 2, 2, 4, 20, 40, 0.005, [900]),               # K past the lanes
    (3, 3, 16, 2, 2, 6, 45, 12, 0.05, [6000, 2000]),        # positions of more than 512 events
    (6, 6, 50, 5, 5, 30, 1, 8, 0.1, [900, 300]),            # filters outside shared memory
])
def test_grouped_matches_cluster(cuda, X, Y, C, fx, fy, C_out, k, K_post, theta, counts, want_pre):
    t = cu(_input(counts, X, Y, C, k, seed=C_out + K_post))
    rng = np.random.default_rng(K_post)
    filt = cu(rng.uniform(-0.5, 1, (C_out, fx, fy, C)).astype(np.float32))
    tau_s = np.float32(0.13)
    tau32, c, dtt = K.lif_constants(0.13, theta, theta)
    ev = K.sort_events(t, tau_s, tau32, bucket_width=C)
    n, a, x, ts, z = K.conv_forward(ev, filt, (X, Y, C), K_post, 0.13, theta, theta, 0.2)
    assert int(n.max()) == K_post or K_post > 32
    err = cu(rng.normal(size=ts.shape).astype(np.float32))
    tabs = K.backward_prep(ts, a, x, z, err, c, tau32, dtt)
    g1, p1 = K.conv_backward(ev, filt, (X, Y, C), ts, tabs, tau_s, tau32, want_pre_errors=want_pre)
    plain = dataclasses.replace(ev, bucketed=None, bucket_offsets=None)
    g2, p2 = K.conv_backward(plain, filt, (X, Y, C), ts, tabs, tau_s, tau32, want_pre_errors=want_pre)
    g1, g2 = g1.cpu().numpy().astype(np.float64), g2.cpu().numpy().astype(np.float64)
    assert np.abs(g2).max() > 0
    assert np.max(np.abs(g1 - g2)) <= 1e-5 * np.abs(g2).max()
    if want_pre:
        p1, p2 = p1.cpu().numpy().astype(np.float64), p2.cpu().numpy().astype(np.float64)
        assert np.abs(p2).max() > 0
        assert np.max(np.abs(p1 - p2)) <= 1e-5 * np.abs(p2).max()
