"""The device sampler (sampler.cu) against sample_token on the same row: the same token for the same random number, at vocabularies
below, at and above its block and vector sizes, with ties at the cut, and what it hands back to the host."""
import numpy as np
import pytest

from webllm_b200 import Gpu, QwenGpt, SamplerOptions, sample_token, synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(built_lib):
    with Gpu(0, weight_bytes=1 << 20, act_bytes=8 << 20) as g:
        yield g


@pytest.mark.parametrize("V", [5, 1023, 4096, 151936])
@pytest.mark.parametrize("top_k,top_p,spread", [(1, 1.0, 3.0), (40, 0.9, 3.0), (1000, 0.5, 1.0), (40, 1.0, 0.0)])
def test_device_sampler_equals_host(gpu, V, top_k, top_p, spread):
    rng = np.random.default_rng(V + top_k)
    model = QwenGpt(gpu, synthetic.QwenShape(V, 1, 1, 1, 64, 64))
    gpu.arena.reset()
    t = gpu.arena.alloc(V)
    for T in (0.7, 1.3):
        row = np.round(rng.standard_normal(V) * spread, 2).astype(np.float32)  # rounded: equal weights happen
        gpu.write(t, row)
        for u in (0.0, 0.31, 0.77, 0.999):
            want = sample_token(row, 0, V, SamplerOptions(T, top_k, top_p, lambda: u))
            got = model.sample(t, T, top_k, top_p, u)
            assert got == want or (spread == 0.0 and V > 2048 and got is None)
    row[V // 2] = np.nan
    gpu.write(t, row)
    assert model.sample(t, 1.0, top_k, top_p, 0.5) is None


def test_host_sampler_prefixes_equal_the_whole_order():
    """The vectorised host sampler against the plain loops, where it looks at a prefix of the order only."""
    from webllm_b200.generate import _walk
    rng = np.random.default_rng(3)
    for spread, top_k, top_p in ((0.0, 0, 1.0), (0.3, 0, 0.9), (2.0, 0, 1.0), (2.0, 7000, 0.99), (0.1, 7000, 1.0)):
        row = np.round(rng.standard_normal(20000) * spread, 2).astype(np.float32)
        w = np.exp((row - row.max()).astype(np.float64)).astype(np.float32)
        order = sorted(range(row.size), key=lambda i: -float(w[i]))[:top_k or row.size]
        for u in (0.0, 0.2, 0.9, 0.9999):
            opt = SamplerOptions(1.0, top_k, top_p, lambda: u)
            assert sample_token(row, 0, row.size, opt) == _walk(list(order), w, opt)
