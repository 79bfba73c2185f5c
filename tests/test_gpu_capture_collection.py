"""A garbage collection that comes due while a train step is captured must not break the capture."""
import gc

import pytest

torch = pytest.importorskip("torch")
from tests.test_gpu_train_step import case, make_step  # noqa: E402

pytestmark = pytest.mark.gpu


def test_capture_with_a_collectable_older_step(cuda):
    """The older, captured step becomes garbage (in a reference cycle) in the middle of the capture, and the automatic
    collection, where it is on, comes due there."""
    t, n, ws, labels = case(seed=5)
    old = make_step(t, ws, labels)
    assert old.try_capture(), old.capture_error
    old.replay()
    torch.cuda.synchronize()
    new = make_step(t, ws, labels)
    box, calls = [old], []
    del old

    def due(stream):
        calls.append(stream)
        if len(calls) == 2:  # the first call is the eager step before the capture
            box.clear()
            if gc.isenabled():
                gc.collect()

    new.launches.insert(len(new.launches) // 2, ("due", due))
    assert new.try_capture(), new.capture_error
    assert len(calls) == 2 and gc.isenabled()
    new.replay()
    torch.cuda.synchronize()
