"""A garbage collection that comes due while a train step is captured must not break the capture."""
import gc

import pytest

torch = pytest.importorskip("torch")
from tests.test_gpu_train_step import case, make_step  # noqa: E402

pytestmark = pytest.mark.gpu


def test_capture_with_a_collectable_older_step(cuda):
    """The older, captured step is garbage in a reference cycle; with a threshold of one allocation a collection would
    come due at any point of the capture."""
    t, n, ws, labels = case(seed=5)
    old = make_step(t, ws, labels)
    assert old.try_capture(), old.capture_error
    old.replay()
    torch.cuda.synchronize()
    new = make_step(t, ws, labels)
    was = gc.get_threshold()
    del old
    try:
        gc.set_threshold(1)
        assert new.try_capture(), new.capture_error
    finally:
        gc.set_threshold(*was)
    assert gc.isenabled()
    new.replay()
    torch.cuda.synchronize()
