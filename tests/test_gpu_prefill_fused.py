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


@pytest.mark.parametrize("B,T", [(11, 128), (11, 127), (80, 33)])
def test_f32_attention_ctas(built_lib, oracle, small, B, T):
    """More tiles of 32 rows than SMs: from 128 tokens on up to two an SM go to the kernel's form of one CTA an SM, fewer tokens (127) and
    more tiles (640) to the one of two."""
    test_f32_attention_tiles(built_lib, oracle, small, B, T)


WIDE = synthetic.QwenShape(256, 1, 14, 2, 896, 4992)  # K = 896: long enough for the CTA-pair kernel at some hundred rows


@pytest.mark.parametrize("n", [385, 512, 1025])
def test_gate_up_silu_in_one_kernel(built_lib, oracle, n):
    """Row counts that leave a token tile ragged, fill it and just pass it; against the same model with gate and up on their own."""
    G = synthetic.random_qwen_gptq(WIDE, seed=12, std=0.05)
    tokens = np.random.default_rng(n).integers(0, WIDE.vocab_size, n).astype(np.uint32)
    ref = oracle.qwen_forward_ref(_ocfg(oracle, WIDE), _dense_from_gptq(oracle, G), tokens, 1, n, threads=oracle.max_threads())
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    err = {}
    for fuse in (True, False):
        with Gpu(0, weight_bytes=64 << 20, act_bytes=256 << 20) as gpu:
            model = QwenGpt(gpu, WIDE, max_t=n, kv_dtype="f32")
            model.upload_gptq_model(G, fuse=fuse)
            got = model.read_tensor(model.forward(tokens, 1, n)).reshape(n, -1)
            if fuse:
                p = gpu.plan(gpu.weight("L0.gateUpW"), n, "f16")
                assert p["kernel_name"] == "gemm_tc_pair" and p["split_k"] == 1, p
            model.close()
        assert oracle.check_tolerance(got, ref, 1e-2 * rms, 2e-2).ok
        err[fuse] = float(np.sqrt(np.mean((got - ref).astype(np.float64) ** 2))) / rms
    assert err[True] < 1.05 * err[False], err  # no precision given up by the fusion


@pytest.mark.parametrize("n", [129, 256, 257, 384])
def test_gate_up_silu_where_the_plain_product_takes_another_kernel(built_lib, oracle, n):
    """The edges of the row counts at which only the fused form runs on CTA pairs, with the same bounds as above."""
    G = synthetic.random_qwen_gptq(WIDE, seed=13, std=0.05)
    tokens = np.random.default_rng(n).integers(0, WIDE.vocab_size, n).astype(np.uint32)
    ref = oracle.qwen_forward_ref(_ocfg(oracle, WIDE), _dense_from_gptq(oracle, G), tokens, 1, n, threads=oracle.max_threads())
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    err = {}
    for fuse in (True, False):
        with Gpu(0, weight_bytes=64 << 20, act_bytes=256 << 20) as gpu:
            model = QwenGpt(gpu, WIDE, max_t=n, kv_dtype="f32")
            model.upload_gptq_model(G, fuse=fuse)
            got = model.read_tensor(model.forward(tokens, 1, n)).reshape(n, -1)
            model.close()
        assert oracle.check_tolerance(got, ref, 1e-2 * rms, 2e-2).ok
        err[fuse] = float(np.sqrt(np.mean((got - ref).astype(np.float64) ** 2))) / rms
    assert err[True] < 1.05 * err[False], err


@pytest.mark.parametrize("n", [64, 65, 127, 128, 129, 193, 320, 511, 512, 513, 575, 577, 640, 705, 897])
def test_tcgen05_prefill_attention(built_lib, oracle, small, n):
    """fp16 cache; the warp-level kernel below 512 rows, tcgen05 from there on: every row against the reference at row counts beside the
    tiles of 128 rows and 64 keys (key groups of different numbers of blocks, a first row tile of which two groups have none,
    ragged last tiles and blocks)."""
    G, Wd = small
    tokens = np.random.default_rng(n).integers(0, SMALL.vocab_size, n).astype(np.uint32)
    ref = oracle.qwen_forward_ref(_ocfg(oracle, SMALL), Wd, tokens, 1, n, threads=oracle.max_threads())
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    with Gpu(0, weight_bytes=64 << 20, act_bytes=128 << 20) as gpu:
        model = QwenGpt(gpu, SMALL, max_t=n, kv_dtype="f16")
        model.upload_gptq_model(G, fuse=True)
        got = model.read_tensor(model.prefill(tokens)).reshape(n, -1)
        gpu.synchronize()  # surfaces a device-side wait that gave up
        model.close()
    row_err = np.sqrt(np.mean((got - ref).astype(np.float64) ** 2, axis=1)) / rms
    assert oracle.check_tolerance(got, ref, 1e-2 * rms, 2e-2).ok and row_err.max() < 1e-2, (float(row_err.max()), int(row_err.argmax()))


@pytest.mark.parametrize("B,T", [(1, 8), (2, 8), (1, 9), (2, 9)])
def test_f32_attention_where_the_tiles_begin(built_lib, oracle, small, B, T):
    test_f32_attention_tiles(built_lib, oracle, small, B, T)


@pytest.mark.parametrize("T", [2, 9])  # the scalar kernel and the tiles
def test_more_sequences_than_a_grid_dimension_holds(built_lib, oracle, T):
    cfg = synthetic.QwenShape(16, 1, 1, 1, 64, 64)
    G = synthetic.random_qwen_gptq(cfg, seed=13, std=0.05)
    some = np.random.default_rng(T).integers(0, 16, (64, T)).astype(np.uint32)
    ref = oracle.qwen_forward_ref(_ocfg(oracle, cfg), _dense_from_gptq(oracle, G), some.ravel(), 64, T).reshape(64, -1)
    pick = np.random.default_rng(14).integers(0, 64, 65535 + 40)
    with Gpu(0, weight_bytes=64 << 20, act_bytes=4 << 30) as gpu:
        model = QwenGpt(gpu, cfg, max_t=T, kv_dtype="f32")
        model.upload_gptq_model(G, fuse=True)
        got = model.read_tensor(model.forward(some[pick].ravel(), pick.size, T)).reshape(pick.size, -1)
        model.close()
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    assert np.abs(got - ref[pick]).max() < 2e-2 * rms  # fp16 operands, as in the tests above


# o and down cut along K with their slices left to the next norm: 16 slices, and the largest numbers that o and down of 896 columns
# take; slices of the CTA-pair kernel; more than eight row tiles of the tensor-memory kernel on a K above 4096.
@pytest.mark.parametrize("C,heads,I,n", [(256, 4, 4992, 340), (896, 14, 4992, 256), (896, 14, 4992, 600), (1024, 16, 8192, 1300), (896, 14, 4992, 1100)])
def test_slices_that_the_norm_adds(built_lib, oracle, C, heads, I, n):
    cfg = synthetic.QwenShape(256, 1, heads, 2, C, I)
    G = synthetic.random_qwen_gptq(cfg, seed=15, std=0.05)
    tokens = np.random.default_rng(n).integers(0, cfg.vocab_size, n).astype(np.uint32)
    ref = oracle.qwen_forward_ref(_ocfg(oracle, cfg), _dense_from_gptq(oracle, G), tokens, 1, n, threads=oracle.max_threads())
    rms = float(np.sqrt(np.mean(ref.astype(np.float64) ** 2)))
    with Gpu(0, weight_bytes=96 << 20, act_bytes=512 << 20) as gpu:
        model = QwenGpt(gpu, cfg, max_t=n, kv_dtype="f16")
        model.upload_gptq_model(G, fuse=True)
        for got in (model.read_tensor(model.forward(tokens, 1, n)), model.read_tensor(model.prefill(tokens))):
            assert oracle.check_tolerance(got.reshape(n, -1), ref, 1e-2 * rms, 2e-2).ok
        model.close()


def test_rounded_activations_and_kept_slices_share_the_workspace(built_lib):
    """A long prompt through separate projections, whose f32 activations are rounded into the workspace: 57 MB for down, beside which 46 MB of
    K slices would not fit. Against the same model with fused projections."""
    cfg, n = synthetic.QwenShape(256, 1, 14, 2, 896, 8960), 3200
    G = synthetic.random_qwen_gptq(cfg, seed=16, std=0.05)
    tokens = np.random.default_rng(n).integers(0, cfg.vocab_size, n).astype(np.uint32)
    got = []
    for fuse in (True, False):
        with Gpu(0, weight_bytes=64 << 20, act_bytes=1 << 30) as gpu:
            model = QwenGpt(gpu, cfg, max_t=n, kv_dtype="f16")
            model.upload_gptq_model(G, fuse=fuse)
            got.append(model.read_tensor(model.prefill(tokens)).astype(np.float64))
            model.close()
    rms = float(np.sqrt(np.mean(got[0] ** 2)))
    assert np.abs(got[1] - got[0]).max() < 3e-2 * rms
