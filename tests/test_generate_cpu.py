"""What ``generate_qwen`` reports, with a stand-in for the model (no GPU)."""
import time
from types import SimpleNamespace

import numpy as np
import pytest

from webllm_b200 import SamplerOptions, generate_qwen

DRAW = 0.05


class SlowDraw:
    """A model whose passes take no time and whose draws take ``DRAW`` seconds, on the device (``sample``) or on the host (``rng``)."""
    max_t = 64

    def __init__(self):
        self.gpu = SimpleNamespace(synchronize=lambda: None)

    def reset_cache(self):
        pass

    def prefill(self, tokens, last_only=False):
        return "row"

    decode_step = prefill

    def read_tensor_slice(self, logits, offset, count):
        return np.zeros(count, np.float32)

    def sample(self, logits, temperature, top_k, top_p, u):
        time.sleep(DRAW)
        return 3

    def rng(self):
        time.sleep(DRAW)
        return 0.5


@pytest.mark.parametrize("top_k", [8, 0])
def test_the_first_draw_counts_as_decoding(top_k):
    model = SlowDraw()
    options = SamplerOptions(temperature=1.0, top_k=top_k, rng=model.rng if top_k == 0 else lambda: 0.5)
    r = generate_qwen(model, SimpleNamespace(vocab_size=16), [1, 2], 1, options)
    assert r.generated == 1 and r.prefill_ms < DRAW * 1e3 and r.tokens_per_second < 1 / DRAW
