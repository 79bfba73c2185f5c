"""The events form of the position-grouped conv backward (filters of at least 192 taps in all, few neurons that spike) against the
taps form, bit for bit. The taps form's results come from the same layer in slices of 32 taps, which have too few taps for the
events form: the gradients of the slices, and the pre-errors as their sum in slice order (a slice is one tile of 32 taps).
Spike buffers of every search depth (K 5, 16, 31, 32 with its 32nd spike) and past the lanes (K 40), positions of more events than a
batch, whose staging is split, a layer whose filters do not fit beside the gradient. Which form the batch goes to is asserted, by the
rule itself and with room for what its sample of the neurons may miss; where every neuron spikes, the taps form."""
import dataclasses

import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K
from tests.test_conv_form import load_rule
from tests.test_gpu_conv_lists import _input
from tests.test_gpu_conv_pool import cu

pytestmark = pytest.mark.gpu

FX, FY = 2, 4  # 8 taps a filter: slices of four filters


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    return load_rule(tmp_path_factory.mktemp("form"))


@pytest.mark.parametrize("want_pre", [True, False])
@pytest.mark.parametrize("few", [True, False])
@pytest.mark.parametrize("X,Y,C,C_out,k,K_post,theta,counts", [
    (9, 9, 4, 24, 6, 5, 0.1, [700, 900, 1]),
    (7, 8, 6, 28, 8, 16, 0.03, [1500, 800]),
    (7, 8, 6, 24, 10, 31, 0.01, [1800, 900, 0]),
    (6, 9, 5, 32, 12, 32, 0.01, [2500, 40]),
    (6, 9, 5, 24, 14, 40, 0.005, [2500]),
    (3, 5, 16, 32, 45, 12, 0.05, [10000, 9000]),   # 600 to 667 events a position
    (8, 9, 70, 32, 1, 8, 0.1, [2400, 2000]),       # 140 KB of filters
])
def test_events_form_equals_taps_form(cuda, rule, X, Y, C, C_out, k, K_post, theta, counts, few, want_pre):
    t = cu(_input(counts, X, Y, C, k, seed=C_out + K_post))
    B = len(counts)
    rng = np.random.default_rng(K_post)
    w = rng.uniform(-0.3, 1, (C_out, FX, FY, C)).astype(np.float32)
    if few:  # one filter in twelve spikes
        w[np.arange(C_out) % 12 != 3] -= np.float32(2.0)
    filt = cu(w)
    tau_s = np.float32(0.13)
    tau32, c, dtt = K.lif_constants(0.13, theta, theta)
    ev = K.sort_events(t, tau_s, tau32, bucket_width=C)
    n, a, x, ts, z = K.conv_forward(ev, filt, (X, Y, C), K_post, 0.13, theta, theta, 0.2)
    assert int(n.max()) == K_post
    tabs = K.backward_prep(ts, a, x, z, cu(rng.normal(size=ts.shape).astype(np.float32)), c, tau32, dtt)
    taps, spiking = C_out * FX * FY, int((tabs.nvalid > 0).sum())
    assert taps >= 192 and ev.cap * (taps // 32) >= 10000
    for room in (0.6, 1.6):
        form = rule(int(spiking * room), int(ev.counts.sum()), B, X * Y, taps, FX * FY)
        if few:
            assert form
        elif X > 3 and room < 1:  # (the small layer is nearly all edge: its line lies past all neurons)
            assert not form
    g, p = K.conv_backward(ev, filt, (X, Y, C), ts, tabs, tau_s, tau32, want_pre_errors=want_pre)
    Xo, Yo = X - FX + 1, Y - FY + 1
    acc = torch.zeros((B, ev.n_neurons, ev.k), device="cuda")
    for lo in range(0, C_out, 4):
        def part(v):
            return v.reshape(B, Xo * Yo, C_out, -1)[:, :, lo:lo + 4].contiguous()

        tab = part(tabs.tables).reshape(B, Xo * Yo * 4, K_post + 1, 2)
        sub = K.BackwardTables(None, None, tab, part(tabs.nvalid).reshape(B, Xo * Yo * 4))
        gs, ps = K.conv_backward(ev, filt[lo:lo + 4].contiguous(), (X, Y, C), part(ts).reshape(B, Xo * Yo * 4, K_post), sub, tau_s,
                                 tau32, want_pre_errors=want_pre)
        assert torch.equal(gs, g[:, lo:lo + 4]), f"filters {lo}"
        if want_pre:
            acc += ps
    assert float(g.abs().max()) > 0
    if want_pre:
        assert torch.equal(p, acc) and float(p.abs().max()) > 0
    # Both against the event-ordered kernel, another order of the same sums (1e-5 of the largest entry, as elsewhere).
    g2, _ = K.conv_backward(dataclasses.replace(ev, bucketed=None, bucket_offsets=None), filt, (X, Y, C), ts, tabs, tau_s, tau32,
                            want_pre_errors=False)
    assert float((g.double() - g2.double()).abs().max()) <= 1e-5 * float(g2.abs().max())
