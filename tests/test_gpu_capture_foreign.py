"""A graph capture of the caller's own (torch.cuda.graph around a step), in which a garbage collection comes due and frees an older
captured train step: the capture stays valid, and the older step's graph is freed afterwards."""
import gc
import weakref

import numpy as np
import pytest

torch = pytest.importorskip("torch")
from tests import test_gpu_conv_train_step as conv_case  # noqa: E402
from tests._helpers import mnist_like_input  # noqa: E402
from tests.test_gpu_train_step import case, make_step  # noqa: E402

pytestmark = pytest.mark.gpu


def _fc():
    t, _, ws, labels = case(seed=3)
    return make_step(t, ws, labels)


def _conv():
    t, _ = mnist_like_input(conv_case.B, seed=9)
    return conv_case.make_step(conv_case.weights(seed=4), t, np.zeros(conv_case.B, np.int32))


@pytest.mark.parametrize("make", [_fc, _conv])
def test_collection_in_a_capture_of_the_callers(cuda, make):
    old, new = make(), _fc()
    assert old.try_capture(), old.capture_error
    old.replay()
    new.step()
    torch.cuda.synchronize()
    step, graph = weakref.ref(old), weakref.ref(old.graph)
    del old
    g, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    gc.disable()  # it comes due where this test says
    try:
        with torch.cuda.stream(side):
            with torch.cuda.graph(g, stream=side):
                new.native_step()
                gc.collect()
                new.native_step()
    finally:
        gc.enable()
    torch.cuda.current_stream().wait_stream(side)
    g.replay()
    torch.cuda.synchronize()
    assert step() is None
    assert new.try_capture(), new.capture_error
    assert graph() is None
