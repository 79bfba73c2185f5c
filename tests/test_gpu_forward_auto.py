"""The forward's own choice of kernel (FWD_AUTO: warp per neuron, 64- or 128-neuron tiles) against the 128-neuron tile kernel, bit for bit,
on both sides of each of its lines: layers of 8, 16, 32 neurons and wider ones at their largest batch of warps and one more,
layers that fill 64-neuron tiles better, at the largest batch for them and one more."""
import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K

pytestmark = pytest.mark.gpu
SUB = 152 * 4


@pytest.mark.parametrize("n_post,batch", [
    (8, 1216), (9, 1351), (9, 1352), (16, 760), (16, 761), (17, 572), (17, 573), (32, 304), (32, 305), (33, 147), (33, 148),
    (131, 37), (131, 38), (192, 26), (256, 20), (131, 1013), (131, 1014), (300, 608), (300, 609), (320, 30),
])
def test_the_choice_does_not_change_the_results(cuda, n_post, batch):
    rng = np.random.default_rng(n_post + batch)
    t = np.sort(np.where(rng.random((batch, 60, 2)) < 0.7, rng.uniform(0, 0.05, (batch, 60, 2)), np.inf), axis=-1)
    t[0] = np.inf
    theta, tau_s, k = 0.2, 0.13, 12
    tau, _, _ = K.lif_constants(tau_s, theta, theta)
    wt = K.transpose_weights(torch.as_tensor(rng.uniform(-0.3, 1.0, (n_post, 60)).astype(np.float32)).cuda())
    ev = K.sort_events(torch.as_tensor(t.astype(np.float32)).cuda(), tau_s, tau)
    got, want = (K.lif_forward_fc(ev, wt, n_post, k, tau_s, theta, theta, 0.2, algo=a) for a in (K.FWD_AUTO, K.FWD_TILE))
    n = want[0]
    assert int(n.sum()) > 0 and torch.equal(got[0], n)
    spike = torch.arange(k, device="cuda") < n[..., None]
    for g, w in zip(got[1:3], want[1:3]):  # a, x: undefined past the spikes
        assert torch.equal(g[spike], w[spike])
    for g, w in zip(got[3:], want[3:]):
        assert torch.equal(g, w)
