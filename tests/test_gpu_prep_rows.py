"""The backward prep of rows that its kernels treat apart, against the thread-per-neuron prep over the same state, bit for bit: warps
without a spike, with one spiking neuron, with full buffers (equal rows, which take the neurons on the lanes), rows whose first time is
+inf though a count says otherwise; K at and around the edges of its variants; few warps and more than 3040."""
import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K
from bats_gb300._lib import call, ptr, stream_ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["counted", "clear", "readonly", "layer"])
@pytest.mark.parametrize("k", [1, 4, 5, 10, 11, 16, 31, 32])
@pytest.mark.parametrize("N", [70, 24600])
def test_rows(cuda, N, k, how):
    rng = np.random.default_rng(k + N)
    B = 4
    n = rng.integers(0, k + 1, (B, N))
    kind = (np.arange(N) // 32) % 4
    n[:, kind == 0] = 0
    n[:, kind == 1] = k
    n[:, (kind == 2) & (np.arange(N) % 32 != 7)] = 0
    times = np.where(np.arange(k) < n[..., None], np.sort(rng.uniform(0, 1, (B, N, k)), axis=-1), np.inf).astype(np.float32)
    times[:, 35 % N, 0] = np.inf  # (a full row's)
    t = torch.as_tensor(times).cuda()
    z, x, a = (torch.as_tensor(rng.uniform(0.5, 2, (B, N, k)).astype(np.float32)).cuda() for _ in range(3))
    err = torch.as_tensor(rng.normal(size=(B, N, k)).astype(np.float32)).cuda()
    first = torch.where(torch.isinf(t), torch.arange(k, device="cuda"), k).amin(-1).int()
    counts = torch.as_tensor(n.astype(np.int32)).cuda()
    got_e = err.clone()
    tab, nv = torch.full((B, N, k + 1, 2), 3.0, device="cuda"), torch.full((B, N), k, dtype=torch.int32, device="cuda")
    heads = K.alloc_cursor_heads(B, N)
    args = (B, N, k, 0.4, 0.26, 0.7)
    if how == "layer":
        call("bats_backward_prep_layer", ptr(t), ptr(a), ptr(x), ptr(z), ptr(got_e), *args, None, None, ptr(tab), ptr(nv), stream_ptr())
    elif how == "readonly":
        call("bats_backward_prep_readonly", ptr(t), ptr(a), ptr(x), ptr(z), ptr(got_e), *args, ptr(tab), ptr(nv), ptr(heads), stream_ptr())
    else:
        call("bats_backward_prep_counted" + ("_clear" if how == "clear" else ""), ptr(t), ptr(counts), ptr(a), ptr(x), ptr(z),
             ptr(got_e), *args, ptr(tab), ptr(nv), ptr(heads), stream_ptr())
    live = torch.arange(k, device="cuda") < first[..., None]
    z_inf = torch.where(live, z, torch.full_like(z, float("inf")))
    want_e, f1, f2 = err.clone(), torch.empty_like(t), torch.empty_like(t)
    want_tab, want_n = torch.empty_like(tab), torch.empty_like(nv)
    call("bats_backward_prep", ptr(t), ptr(a), ptr(x), ptr(z_inf), ptr(want_e), *args, 1, 1, ptr(f1), ptr(f2), ptr(want_tab),
         ptr(want_n), stream_ptr())
    assert torch.equal(nv, first) and torch.equal(want_n, first)
    assert torch.equal(tab[:, :, :k][live], want_tab[:, :, :k][live])
    if how == "readonly":
        assert torch.equal(got_e, err)
    else:
        assert torch.equal(got_e[live], want_e[live])
        assert torch.equal(got_e[~live], torch.zeros_like(err)[~live] if how == "clear" else err[~live])
    if how != "layer":
        pairs = B * N
        raw = heads.cpu().numpy()
        ht = raw[:pairs * 8].view(np.float32).reshape(B, N, 2)
        at = (pairs * 8 + 15) // 16 * 16
        hab = raw[at:at + pairs * 16].view(np.float32).reshape(B, N, 2, 2)
        m = first.cpu().numpy()
        w_t, w_ab = np.full((B, N, 2), np.inf, np.float32), np.zeros((B, N, 2, 2), np.float32)
        for q in range(min(2, k)):
            w_t[..., q] = np.where(m > q, times[..., q], np.inf)
            w_ab[:, :, q] = np.where((m > q)[..., None], want_tab[:, :, q].cpu().numpy(), 0.0)
        assert np.array_equal(ht, w_t) and np.array_equal(hab, w_ab)
