"""A train step of one layer has no launch on the second stream: its capture must not wait for that stream, and the graph must
give what the launch list gives."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from bats_gb300.train import FCLayerSpec, FCTrainStep  # noqa: E402

pytestmark = pytest.mark.gpu


def _step():
    rng = np.random.default_rng(4)
    t = np.where(rng.random((6, 40, 1)) < 0.5, rng.uniform(0, 0.02, (6, 40, 1)), np.inf).astype(np.float32)
    w = torch.as_tensor(rng.uniform(-0.5, 1.0, (5, 40)).astype(np.float32))
    ts = FCTrainStep(6, 40, 1, [FCLayerSpec(5, 0.13, 0.2, 0.2, 12)], [w], 9.0, 2.0, learning_rate=0.01, max_simulation=0.2)
    ts.set_inputs(torch.as_tensor(t), torch.arange(6, dtype=torch.int32) % 5)
    return ts


def test_one_layer_step_is_captured(cuda):
    graph, eager = _step(), _step()
    assert graph.try_capture(), graph.capture_error  # one eager step first
    eager.step()
    for _ in range(2):
        graph.run()
        eager.step()
    torch.cuda.synchronize()
    assert int(eager.out[0][0].sum()) > 0
    assert torch.equal(graph.W[0], eager.W[0]) and torch.equal(graph.loss, eager.loss)
