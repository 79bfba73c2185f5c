"""Calls from several host threads: launch attributes belong to the process, not to the thread that sets them."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from bats_gb300 import kernels as K  # noqa: E402

pytestmark = pytest.mark.gpu


def _pre_errors(n_post, k_post):
    """Pre-spike errors of a narrow layer, whose kernel takes shared memory in proportion to n_post k_post."""
    rng = np.random.default_rng(n_post)
    t = torch.tensor(np.sort(rng.uniform(0, 0.1, (2, 40, 3)), axis=2).astype(np.float32), device="cuda")
    w = torch.tensor(rng.uniform(0, 1, (n_post, 40)).astype(np.float32), device="cuda")
    tau, c, dtt = K.lif_constants(0.13, 0.2, 0.2)
    ev = K.sort_events(t, 0.13, tau)
    wt = K.transpose_weights(w)
    n, a, x, times, z = K.lif_forward_fc(ev, wt, n_post, k_post, 0.13, 0.2, 0.2)
    tabs = K.backward_prep(times, a, x, z, torch.ones_like(times), c, tau, dtt, n_spikes=n)
    return K.pre_errors(ev, wt, times, tabs, 0.13, tau)


def test_a_smaller_launch_in_another_thread_leaves_the_limit(cuda):
    first = _pre_errors(32, 32)
    failed = []

    def small():
        try:
            _pre_errors(2, 2)
        except Exception as exc:
            failed.append(exc)

    th = threading.Thread(target=small)
    th.start()
    th.join()
    assert not failed, failed
    assert torch.equal(first, _pre_errors(32, 32))
    assert torch.isfinite(_pre_errors(16, 20)).all()
