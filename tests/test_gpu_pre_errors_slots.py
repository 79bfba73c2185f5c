"""The pre-errors written at the events' slots only, against the ones that set the other slots to 0: equal at the events' slots (narrow
layers of one and of 32 neurons, one and several tiles), the other slots as they were; and the narrow kernel on events out of time
order, which have no common place, against the same events in order."""
import dataclasses

import numpy as np
import pytest
import torch

from bats_gb300 import kernels as K
from bats_gb300._lib import call, ptr, stream_ptr

pytestmark = pytest.mark.gpu


def _state(n_post, seed):
    rng = np.random.default_rng(seed)
    t = np.sort(np.where(rng.random((9, 50, 4)) < 0.5, rng.uniform(0, 0.05, (9, 50, 4)), np.inf), axis=-1)
    t[3] = np.inf
    tau, c, dtt = K.lif_constants(0.1, 0.1, 0.1)
    wt = K.transpose_weights(torch.as_tensor(rng.uniform(-0.3, 1.0, (n_post, 50)).astype(np.float32)).cuda())
    ev = K.sort_events(torch.as_tensor(t.astype(np.float32)).cuda(), 0.1, tau)
    n, a, x, ts, z = K.lif_forward_fc(ev, wt, n_post, 9, 0.1, 0.1, 0.1, 0.2)
    assert int(n.sum()) > 0
    tabs = K.backward_prep(ts, a, x, z, torch.as_tensor(rng.normal(size=ts.shape).astype(np.float32)).cuda(), c, tau, dtt)
    return ev, wt, ts, tabs, tau


@pytest.mark.parametrize("n_post", [1, 31, 32, 64, 200])
def test_only_event_slots_are_written(cuda, n_post):
    ev, wt, ts, tabs, tau = _state(n_post, n_post)
    want = K.pre_errors(ev, wt, ts, tabs, 0.1, tau)
    got = torch.full_like(want, 7.0)
    size = K.call_size("bats_pre_errors_workspace_bytes", 9, ev.cap, n_post)
    ws = torch.empty(max(size, 1), dtype=torch.uint8, device="cuda")
    call("bats_pre_errors_slots", ptr(ev.events), ptr(ev.slots), ptr(ev.counts), ev.cap, ptr(wt), wt.shape[1], ptr(ts),
         ptr(tabs.tables), ptr(tabs.nvalid), 9, n_post, 9, 50, 4, 0.1, float(tau), ptr(got), ptr(ws), size, stream_ptr())
    written = torch.zeros(9, 200, dtype=torch.bool, device="cuda")
    for s in range(9):
        written[s, ev.slots[s, :int(ev.counts[s])].long()] = True
    written = written.reshape(want.shape)
    assert torch.equal(got[written], want[written]) and bool((got[~written] == 7.0).all())
    assert bool((want[~written] == 0.0).all()) and float(want.abs().max()) > 0


@pytest.mark.parametrize("n_post", [3, 32])
def test_narrow_events_out_of_order(cuda, n_post):
    ev, wt, ts, tabs, tau = _state(n_post, 5)
    want = K.pre_errors(ev, wt, ts, tabs, 0.1, tau)
    events, slots = ev.events.clone(), ev.slots.clone()
    for s in range(9):
        k = int(ev.counts[s])
        order = torch.randperm(k, device="cuda")
        events[s, :k], slots[s, :k] = ev.events[s, order], ev.slots[s, order]
    assert torch.equal(K.pre_errors(dataclasses.replace(ev, events=events, slots=slots), wt, ts, tabs, 0.1, tau), want)
