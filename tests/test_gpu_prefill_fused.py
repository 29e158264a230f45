"""GPU parity of the many-row kernels of the model at the edges of their tiles: f32 attention (tiles of 32 rows and keys),
silu(gate) * up in the gate | up projection (tiles of 128 to 256 rows), prefill attention on the tensor cores."""
import numpy as np
import pytest

from test_gpu_qwen import SMALL, _dense_from_gptq, _ocfg
from webllm_b200 import Gpu, QwenGpt, synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small(oracle):
    G = synthetic.random_qwen_gptq(SMALL, seed=11, std=0.05)
    return G, _dense_from_gptq(oracle, G)


@pytest.mark.parametrize("B,T", [(1, 2), (3, 31), (2, 32), (2, 33), (1, 97)])
def test_f32_attention_tiles(built_lib, oracle, small, B, T):
    """Uncached forward and, for one sequence, the cached prefill, both in the fp32-activation mode."""
    G, Wd = small
    tokens = np.random.default_rng(B * 1000 + T).integers(0, SMALL.vocab_size, B * T).astype(np.uint32)
    ref = oracle.qwen_forward_ref(_ocfg(oracle, SMALL), Wd, tokens, B, T, threads=oracle.max_threads())
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    with Gpu(0, weight_bytes=64 << 20, act_bytes=128 << 20) as gpu:
        model = QwenGpt(gpu, SMALL, max_t=T, kv_dtype="f32")
        model.upload_gptq_model(G, fuse=True)
        model.set_exact(True)
        got = model.read_tensor(model.forward(tokens, B, T)).reshape(B * T, -1)
        assert oracle.check_tolerance(got, ref, 2e-4 * rms, 2e-4).ok
        if B == 1:
            got = model.read_tensor(model.prefill(tokens)).reshape(T, -1)
            assert oracle.check_tolerance(got, ref, 2e-4 * rms, 2e-4).ok
        model.close()


@pytest.mark.parametrize("n", [128, 200, 257, 390])
def test_gate_up_silu_in_one_kernel(built_lib, oracle, small, n):
    """Row counts that fill, leave ragged and just pass a token tile."""
    G, Wd = small
    tokens = np.random.default_rng(n).integers(0, SMALL.vocab_size, n).astype(np.uint32)
    ref = oracle.qwen_forward_ref(_ocfg(oracle, SMALL), Wd, tokens, 1, n, threads=oracle.max_threads())
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    with Gpu(0, weight_bytes=128 << 20, act_bytes=128 << 20) as gpu:
        got = {}
        for fuse in (True, False):
            model = QwenGpt(gpu, SMALL, max_t=n, kv_dtype="f32")
            model.upload_gptq_model(G, fuse=fuse)
            got[fuse] = model.read_tensor(model.forward(tokens, 1, n)).reshape(n, -1)
            model.close()
        assert oracle.check_tolerance(got[True], ref, 1e-2 * rms, 2e-2).ok
        err = {f: float(np.sqrt(np.mean((g - ref).astype(np.float64) ** 2))) / rms for f, g in got.items()}
        assert err[True] < 1.05 * err[False] + 1e-6, err  # no precision given up by the fusion
