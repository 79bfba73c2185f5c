"""The backward prep that leaves the errors alone and finds the counts itself, and the one that is given the counts, against the
thread-per-neuron prep over the same state: counts and every table entry below them equal bit for bit, the errors untouched or the same,
the cursor heads those of the rows. One slot, full buffers of 32, a last warp partly filled, silent neurons, +inf before the end of a
train, both sides of the line between the kernels (3040 warps); and a gradient that is an expanded scalar."""
import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K
from bats_gb300._lib import call, ptr, stream_ptr
from bats_gb300.autograd import lif_fc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("counted", [False, True])
@pytest.mark.parametrize("B,N,k", [(1, 1, 1), (3, 33, 32), (7, 70, 30), (64, 5, 2), (2947, 33, 3), (2948, 33, 3), (3100, 32, 32)])
def test_readonly_prep(cuda, B, N, k, counted):
    rng = np.random.default_rng(B + k)
    n = rng.integers(0, k + 1, (B, N))
    n[0, 0] = k
    slot = np.arange(k) < n[..., None]
    t = np.where(slot, np.sort(rng.uniform(0, 1, (B, N, k)), axis=-1), np.inf).astype(np.float32)
    if k > 4:
        t[0, 0, 3] = np.inf  # finite times past it do not count
    z, x, a = (torch.as_tensor(rng.uniform(0.5, 2, (B, N, k)).astype(np.float32)).cuda() for _ in range(3))
    err = torch.as_tensor(np.where(slot, rng.normal(size=(B, N, k)), np.nan).astype(np.float32)).cuda()
    t = torch.as_tensor(t).cuda()
    kept = err.clone()
    first = torch.where(torch.isinf(t), torch.arange(k, device="cuda"), k).amin(-1).int()
    if counted:
        got = K.backward_prep(t, a, x, z, kept, 0.4, 0.26, 0.7, n_spikes=first)
    else:
        got = K.backward_prep(t, a, x, z, err, 0.4, 0.26, 0.7, keep_errors=True)
        assert torch.equal(err.view(torch.int32), kept.view(torch.int32))
    assert torch.equal(got.nvalid, first)
    z_inf = torch.where(torch.arange(k, device="cuda") < first[..., None], z, torch.full_like(z, float("inf")))
    f1, f2, tab, nv = torch.empty_like(t), torch.empty_like(t), torch.empty((B, N, k + 1, 2), device="cuda"), torch.empty((B, N), dtype=torch.int32, device="cuda")
    call("bats_backward_prep", ptr(t), ptr(a), ptr(x), ptr(z_inf), ptr(err), B, N, k, 0.4, 0.26, 0.7, 1, 1, ptr(f1), ptr(f2),
         ptr(tab), ptr(nv), stream_ptr())
    valid = torch.arange(k + 1, device="cuda") < first[..., None]
    assert torch.equal(got.tables[valid], tab[valid])
    if counted:  # the reset errors below the counts
        assert torch.equal(kept[valid[..., :k]], err[valid[..., :k]])
    pairs = B * N
    heads = got.heads.cpu().numpy()
    ht = heads[:8 * pairs].view(np.float32).reshape(B, N, 2)
    hab = heads[(8 * pairs + 15) // 16 * 16:][:16 * pairs].view(np.float32).reshape(B, N, 2, 2)
    tt, tb, f = t.cpu().numpy(), tab.cpu().numpy(), first.cpu().numpy()
    for p in range(min(2, k)):
        has = f > p
        np.testing.assert_array_equal(ht[..., p], np.where(has, tt[..., p], np.inf))
        np.testing.assert_array_equal(hab[..., p, :], np.where(has[..., None], tb[:, :, p], 0.0))


def test_expanded_gradient(cuda):
    t = torch.sort(torch.rand((4, 30, 3), device="cuda", generator=torch.Generator("cuda").manual_seed(1)) * 0.05, dim=-1).values
    outs = []
    for scale in (False, True):
        w = torch.linspace(0.0, 1.0, 30 * 20, device="cuda").reshape(20, 30).requires_grad_()
        times, n = lif_fc(t, w, 0.1, 0.2, 0.2, 16, 0.3)
        assert int(n.sum()) > 0
        g = torch.ones((), device="cuda").expand(times.shape)
        times.backward(g if not scale else g.contiguous().double().float())
        outs.append(w.grad)
    assert torch.equal(*outs) and float(outs[0].abs().max()) > 0
