"""Choices that the autotuner saved with another build of the library are timed anew, those of the same build are taken."""
import json

import pytest

torch = pytest.importorskip("torch")
from bats_gb300 import _lib  # noqa: E402
from bats_gb300.autotune import Autotuner  # noqa: E402


def test_choices_belong_to_a_build(tmp_path, monkeypatch):
    monkeypatch.setattr(Autotuner, "device_tag", staticmethod(lambda device=None: "gpu"))
    lib, path = tmp_path / "libbats_gb300.so", tmp_path / "tune.json"
    monkeypatch.setattr(_lib, "LIB_PATH", str(lib))

    def saved_under(content):
        lib.write_bytes(content)
        return Autotuner(path=str(path)).key("fc_forward", 4, 5)

    first, second = saved_under(b"one build"), saved_under(b"another build")
    assert first != second and saved_under(b"one build") == first
    path.write_text(json.dumps({first: "lanes"}))
    tuner = Autotuner(path=str(path))
    assert tuner.pick("fc_forward", (4, 5), {"tile": None, "lanes": None}) == "lanes"  # nothing is run
    lib.write_bytes(b"another build")
    with pytest.raises(Exception):  # not taken: the candidates would be run (they cannot be)
        tuner.pick("fc_forward", (4, 5), {"tile": None, "lanes": None})


@pytest.mark.gpu
def test_the_default_is_a_candidate(cuda):
    """131 neurons, 128 samples: the library's own choice, 64-neuron tiles of 8-event stages, has no name of its own."""
    import numpy as np

    from bats_gb300.serving import InferenceServer, LayerSpec, make_requests
    from bats_gb300.train import FCLayerSpec, FCTrainStep
    rng = np.random.default_rng(0)
    t = np.where(rng.random((128, 200, 1)) < 0.6, rng.uniform(0, 0.02, (128, 200, 1)), np.inf).astype(np.float32)
    sizes = (200, 131, 9)
    ws = [rng.uniform(-0.5, 1.0, (o, i)).astype(np.float32) for i, o in zip(sizes[:-1], sizes[1:])]
    ts = FCTrainStep(128, 200, 1, [FCLayerSpec(n, 0.13, 0.2, 0.2, 10) for n in sizes[1:]], [torch.as_tensor(w) for w in ws],
                     9.0, 2.0, max_simulation=0.2)
    ts.set_inputs(torch.as_tensor(t), torch.zeros(128, dtype=torch.int32))
    tuner = Autotuner(path=None)
    ts.autotune(tuner, force=True)
    server = InferenceServer(ws, [LayerSpec(n, 0.13, 0.2, 0.2, 10) for n in sizes[1:]], 200, 300, k_in=32, max_batch=2,
                             max_lanes=1)
    server.autotune(make_requests(4, n_channels=200, hi=300), tuner)
    timed = [set(v) for k, v in tuner.timings.items() if k.startswith("fc_forward")]
    assert len(timed) >= 4 and all("auto" in names for names in timed), timed
