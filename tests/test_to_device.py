"""Lists on their way to a device, whatever the program's default device is."""
import pytest
import torch

from pisceslx_b200.models.generation import to_device


def test_default_device_on_cpu():
    with torch.device("meta"):
        t = to_device([3, 1], torch.int32, torch.device("cpu"))
    assert t.tolist() == [3, 1] and t.dtype == torch.int32 and t.device.type == "cpu"


@pytest.mark.gpu
@pytest.mark.parametrize("default", ["cuda", "cpu"])
def test_default_device_on_the_gpu(default):
    """A prompt through the engine, whose numbers are lists on the host."""
    from pisceslx_b200 import YvConfig
    from pisceslx_b200.models import build_model
    from pisceslx_b200.serve.engine import YvEngineConfig, YvInferenceEngine
    cfg = YvConfig.tiny_text_moe()
    cfg.vocab_size, cfg.n_layer = 512, 1
    engine = YvInferenceEngine(build_model(cfg, "cuda", torch.bfloat16).eval(), cfg=YvEngineConfig(num_blocks=8))
    out = []
    for d in ("cpu", default):
        with torch.device(d):
            engine.cache.add_sequence(0)
            out.append(engine.run_tokens(0, list(range(100)), [99, 3]))
            engine.cache.free_sequence(0)
    assert torch.equal(*out)
