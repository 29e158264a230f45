"""The tiled double-precision kernel (fp32-activation mode at many rows, ragged K) against gemmNTRef, bit for bit, at the edges of its
tiles: rows and columns on and beside 32 and 64, K remainders inside a packed row, a group and a stage, both tile widths."""
import numpy as np
import pytest

from webllm_b200 import Gpu, _lib, synthetic

from helpers import oracle_weight, register, run_linear

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu(built_lib):
    with Gpu(0, weight_bytes=64 << 20, act_bytes=64 << 20) as g:
        yield g


@pytest.mark.parametrize("M,N,K,group,zeros", [(64, 32, 32, 32, "any"), (33, 65, 72, 8, "none"), (145, 1236, 1000, 128, "7or8"),
                                               (70, 4864, 896, 128, "any"), (7, 31, 999, 64, "sym")])
def test_generic_equals_reference_bits(gpu, oracle, M, N, K, group, zeros):
    t = synthetic.random_gptq(K, N, group, seed=M + N, zeros=zeros)
    h = register(gpu, f"gen_{M}_{N}_{K}", t)
    x = np.random.default_rng(K).standard_normal((M, K)).astype(np.float32)
    hb = gpu.f32_upload(f"genb_{M}_{N}_{K}", np.random.default_rng(N).standard_normal(N).astype(np.float32))
    gpu.plan_override(_lib.WB_KERNEL_GENERIC, 0)
    try:
        got = run_linear(gpu, h, x, M, N, hb, exact=True)
    finally:
        gpu.plan_override(0, 0)
    bias = np.random.default_rng(N).standard_normal(N).astype(np.float32)
    ref = oracle.gemm_nt_ref(x, oracle_weight(oracle, t), M, N, K, bias, threads=oracle.max_threads())
    assert np.array_equal(got.view(np.uint32), np.asarray(ref, np.float32).reshape(got.shape).view(np.uint32))


@pytest.mark.parametrize("M", [65535 * 32, 65535 * 32 + 33])
def test_more_rows_than_a_second_grid_dimension_holds(gpu, oracle, M):
    K, N = 4, 3
    rng = np.random.default_rng(M)
    W, x = rng.standard_normal((N, K)).astype(np.float16), rng.standard_normal((M, K)).astype(np.float32)
    h = gpu.f16_alloc(f"rows_{M}", N, K)
    gpu.f16_write_bits(h, 0, W)
    got = run_linear(gpu, h, x, M, N, exact=True)
    assert np.array_equal(got, oracle.gemm_nt_ref(x, W.astype(np.float32), M, N, K))
