"""After a train step the pre-errors of a layer are 0 at every slot without a spike, whatever an earlier step wrote there: eager
steps, graph replays, one stream, and a layer of K > 32 between."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from bats_gb300.train import FCLayerSpec, FCTrainStep  # noqa: E402

pytestmark = pytest.mark.gpu


def _input(p, seed):
    rng = np.random.default_rng(seed)
    return torch.as_tensor(np.where(rng.random((5, 60, 1)) < p, rng.uniform(0, 0.02, (5, 60, 1)), np.inf).astype(np.float32))


@pytest.mark.parametrize("k", [12, 40])
@pytest.mark.parametrize("mode", ["eager", "graph", "one_stream"])
def test_slots_without_a_spike_are_zero(cuda, mode, k):
    rng = np.random.default_rng(2)
    sizes = (60, 70, 40, 6)
    w = [torch.as_tensor(rng.uniform(-0.5, 1.0, (o, i)).astype(np.float32)) for i, o in zip(sizes[:-1], sizes[1:])]
    specs = [FCLayerSpec(n, 0.13, 0.2, 0.2, k) for n in sizes[1:]]
    ts = FCTrainStep(5, 60, 1, specs, w, 9.0, 2.0, learning_rate=1e-4, max_simulation=0.2)
    labels = torch.arange(5, dtype=torch.int32)
    if mode == "one_stream":
        ts.aux = None
    ts.set_inputs(_input(0.9, 0), labels)
    if mode == "graph":
        assert ts.try_capture(), ts.capture_error
    ts.run()
    many = [int(c.counts.sum()) for c in ts.ev[1:]]
    ts.set_inputs(_input(0.1, 1), labels)
    ts.run()
    torch.cuda.synchronize()
    for li in (1, 2):
        ev, pe = ts.ev[li], ts.pre_err[li].reshape(5, -1)
        assert 0 < int(ev.counts.sum()) < many[li - 1]  # fewer spikes: some slots written before have none now
        spike = torch.zeros_like(pe, dtype=torch.bool)
        for s in range(5):
            spike[s, ev.slots[s, :int(ev.counts[s])].long()] = True
        assert bool((pe[~spike] == 0).all()) and float(pe[spike].abs().max()) > 0
