"""Whether a train step's first gradient waits for the second stream: only where it is large and the larger part (measured layers on
both sides of the rule)."""
from types import SimpleNamespace

import pytest

from bats_gb300.train import FCTrainStep


@pytest.mark.parametrize("batch,sizes,k_in,joined", [
    (4096, (1024, 1024, 20), 16, True), (1024, (1024, 1024, 20), 16, True), (4096, (784, 800, 10), 1, True),
    (2048, (1000, 400, 20), 8, True), (1024, (784, 800, 10), 1, False), (8, (784, 800, 10), 1, False),
    (300, (700, 64, 20), 16, False), (4096, (300, 200, 10), 8, False), (256, (784, 800, 800, 10), 1, False),
    (4096, (784, 800, 800, 10), 1, False), (4096, (784, 10), 16, False)])
def test_rule(batch, sizes, k_in, joined):
    ts = FCTrainStep.__new__(FCTrainStep)
    ts.B = batch
    ts.specs = [SimpleNamespace(n_neurons=n, max_n_spike=30) for n in sizes[1:]]
    ts.ev = [SimpleNamespace(n_neurons=n, k=k) for n, k in zip(sizes[:-1], [k_in] + [30] * len(sizes))]
    assert ts._joined_launches() == (("L1.grad_adam",) if joined else ())
