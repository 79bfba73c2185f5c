"""The tile and work-queue forwards end a sample's event stream once every neuron of the tile holds K spikes: the
results are those of the lanes kernel, which stops neuron by neuron, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from bats_gb300 import kernels as K  # noqa: E402
from bats_gb300._lib import check_device_status  # noqa: E402
from tests.test_gpu_forward import _assert_identical, _both_algos  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_post,k_post,late", [(20, 1, False), (32, 3, True), (33, 2, False), (64, 1, True),
                                                (128, 2, False), (161, 4, True)])
def test_streams_that_end_early(cuda, n_post, k_post, late):
    """Strong weights fill every neuron's buffer after a few events of samples with 0 to 1800 events (event counts
    around multiples of the stage and of the producer's block among them); late: one neuron per tile of 32 fills only
    on its last events, or never, and keeps the stream alive."""
    rng = np.random.default_rng(n_post)
    counts = [0, 1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 600, 1800, 1799, 5]
    t = np.full((len(counts), 100, 32), np.inf, np.float32)
    for s, m in enumerate(counts):
        ch = np.repeat(np.arange(100), 32)[rng.permutation(3200)[:m]]
        tm = np.sort(rng.uniform(0, 0.2, m)).astype(np.float32)
        for j in np.unique(ch):
            own = tm[ch == j]
            t[s, j, :own.size] = own
    W = rng.uniform(0.5, 1.5, (n_post, 100)).astype(np.float32)
    if late:
        W[::32] *= np.float32(1e-3)
    outs = _both_algos(t, W, 0.13, 0.2, 0.02, k_post)
    lanes = outs[1]
    assert (lanes[0][12] == k_post).mean() > 0.9 and (lanes[0] == 0).any()
    for q, o in enumerate(outs):
        _assert_identical(lanes, o, f"variant {q}")
    check_device_status()
