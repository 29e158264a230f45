"""The tiled double-precision kernel (fp32-activation mode at many rows, ragged K) against gemmNTRef, bit for bit, at the edges of its
tiles: each of the four row counts of a tile, columns on and beside 32, K remainders inside a packed row, a group and a stage; and with
operands whose sums depend on the order of every addition."""
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


@pytest.mark.parametrize("M,rows", [(7, 8), (100, 16), (145, 24), (1000, 32)])
def test_every_tile_height(gpu, oracle, M, rows):
    K, N = 200, 1236
    t = synthetic.random_gptq(K, N, 40, seed=M, zeros="any")
    h = register(gpu, f"genr_{M}", t)
    x = np.random.default_rng(M).standard_normal((M, K)).astype(np.float32)
    gpu.plan_override(_lib.WB_KERNEL_GENERIC, 0)
    try:
        assert gpu.plan(h, M, "f32", exact=True)["tile_m"] == rows
        got = run_linear(gpu, h, x, M, N, exact=True)
    finally:
        gpu.plan_override(0, 0)
    ref = oracle.gemm_nt_ref(x, oracle_weight(oracle, t), M, N, K, threads=oracle.max_threads())
    assert np.array_equal(got.view(np.uint32), np.asarray(ref, np.float32).reshape(got.shape).view(np.uint32))


def test_the_order_of_the_chain(gpu, oracle):
    """gemmNTRef adds its products in ascending k, each sum rounded to double. Here that order shows: products over some sixty binades, half
    of them the exact opposites of the others, so that the result is nothing but what the additions rounded off."""
    M, N, K = 65, 136, 1024
    rng = np.random.default_rng(9)
    W = (rng.choice([-1.0, 1.0], (N, K)) * rng.uniform(1, 2, (N, K)) * 2.0 ** rng.integers(-10, 11, (N, K))).astype(np.float16)
    x = (rng.choice([-1.0, 1.0], (M, K)) * rng.uniform(1, 2, (M, K)) * 2.0 ** rng.integers(-20, 21, (M, K))).astype(np.float32)
    order = rng.permutation(K)
    W[:, order[K // 2:]], x[:, order[K // 2:]] = W[:, order[: K // 2]], -x[:, order[: K // 2]]
    h = gpu.f16_alloc("gen_chain", N, K)
    gpu.f16_write_bits(h, 0, W)
    gpu.plan_override(_lib.WB_KERNEL_GENERIC, 0)
    try:
        got = run_linear(gpu, h, x, M, N, exact=True)
    finally:
        gpu.plan_override(0, 0)
    W32 = W.astype(np.float32)
    ref = np.asarray(oracle.gemm_nt_ref(x, W32, M, N, K, threads=oracle.max_threads()), np.float32).reshape(M, N)
    for step in (4, 2):  # the inputs do what they are for: groups of four, and pairs, the other way round give other bits
        by = np.arange(K).reshape(-1, step)[:, ::-1].ravel()
        other = np.asarray(oracle.gemm_nt_ref(x[:, by].copy(), W32[:, by].copy(), M, N, K, threads=oracle.max_threads()), np.float32).reshape(M, N)
        assert np.mean(ref.view(np.uint32) != other.view(np.uint32)) > 0.5
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))


@pytest.mark.parametrize("M", [65535 * 32, 65535 * 32 + 33])
def test_more_rows_than_a_second_grid_dimension_holds(gpu, oracle, M):
    K, N = 4, 3
    rng = np.random.default_rng(M)
    W, x = rng.standard_normal((N, K)).astype(np.float16), rng.standard_normal((M, K)).astype(np.float32)
    h = gpu.f16_alloc(f"rows_{M}", N, K)
    gpu.f16_write_bits(h, 0, W)
    got = run_linear(gpu, h, x, M, N, exact=True)
    assert np.array_equal(got, oracle.gemm_nt_ref(x, W.astype(np.float32), M, N, K))
