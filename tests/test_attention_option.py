"""``moe_deterministic`` reaches every attention layer of the modules that are made from a configuration."""
import pytest

from pisceslx_b200 import YvConfig
from pisceslx_b200.models.attention import YvAttention
from pisceslx_b200.models.multimodal import YvVideoEncoder, YvVisionEncoder
from pisceslx_b200.models.multimodal.fusion import YvAudioEncoder, YvDynamicModalFusion
from pisceslx_b200.models.reasoning_engine import YvLatentCoTReasoner, YvMultiPathReasoningEngine
from pisceslx_b200.models.reasoning_multipath import YvMultiModalReasoningEnhancer


@pytest.mark.parametrize("on", [True, False])
@pytest.mark.parametrize("make", [lambda c: YvAttention(c, 0), YvVisionEncoder, YvVideoEncoder, YvAudioEncoder, YvDynamicModalFusion,
                                  YvMultiPathReasoningEngine, YvLatentCoTReasoner, YvMultiModalReasoningEnhancer])
def test_option(make, on):
    cfg = YvConfig.tiny_text_moe()
    cfg.vocab_size = 64
    if on:
        cfg.extra["moe_deterministic"] = True
    layers = [m for m in make(cfg).modules() if hasattr(m, "deterministic")]
    assert layers and all(m.deterministic is on for m in layers)
