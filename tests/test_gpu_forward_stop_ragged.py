"""A tile whose last warps own no neuron ends its event stream as early as a full one once its neurons hold their K spikes (the tile and
work-queue forwards of n_post 129 .. 224 neurons): far quicker than with one neuron that stays silent and needs every event.
Without the early end both take the same time."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from bats_gb300 import kernels as K  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("algo", [K.FWD_TILE, K.FWD_QUEUE, K.FWD_TILE64])
@pytest.mark.parametrize("n_post", [136, 161, 200])
def test_ragged_tile_stops(cuda, algo, n_post):
    rng = np.random.default_rng(n_post)
    t = np.sort(rng.uniform(0, 0.2, (1, 2000, 30)), axis=-1).astype(np.float32)
    tau, c, dtt = K.lif_constants(0.13, 0.2, 0.02)
    ev = K.sort_events(torch.as_tensor(t).cuda(), np.float32(0.13), tau, bucketed=False)

    def run(silent):
        w = rng.uniform(0.5, 1.5, (n_post, 2000)).astype(np.float32)
        if silent:
            w[-1] *= np.float32(1e-6)
        wt = K.transpose_weights(torch.as_tensor(w).cuda())
        best = np.inf
        for _ in range(4):
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            start.record()
            out = K.lif_forward_fc(ev, wt, n_post, 1, 0.13, 0.2, 0.02, 0.2, algo=algo)
            end.record()
            end.synchronize()
            best = min(best, start.elapsed_time(end))
        n = out[0][0].cpu().numpy()
        assert (n[:-1] == 1).all() and n[-1] == (0 if silent else 1)
        return best

    every, stopped = run(True), run(False)
    assert stopped < every / 4, (stopped, every)
