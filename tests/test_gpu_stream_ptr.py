"""The raw stream handle of the calls: that of torch's current stream, on the default stream, inside a stream context, in
another thread, and for a stream given."""
import threading

import pytest
import torch

from bats_gb300._lib import stream_ptr

pytestmark = pytest.mark.gpu


def test_stream_ptr_is_the_current_stream(cuda):
    assert stream_ptr() == torch.cuda.current_stream().cuda_stream
    side = torch.cuda.Stream()
    seen = []
    with torch.cuda.stream(side):
        assert stream_ptr() == side.cuda_stream
        thread = threading.Thread(target=lambda: seen.append((stream_ptr(), torch.cuda.current_stream().cuda_stream)))
        thread.start()
        thread.join()
    assert seen[0][0] == seen[0][1]
    assert stream_ptr(side) == side.cuda_stream
    assert stream_ptr() == torch.cuda.current_stream().cuda_stream
