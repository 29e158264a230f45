"""GPU parity of the small-batch int4 GEMM on large matrices (9 to 16 rows): ragged row counts, a last column group that is not full,
slices that do not divide K, groups of one and several chunks, both column widths and output types."""
import numpy as np
import pytest

from helpers import assert_close, oracle_weight, register, run_linear
from webllm_b200 import synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,N,group,zeros", [(1152, 8224, 128, "any"), (8576, 1056, 128, "7or8"), (2560, 3360, 256, "none")])
@pytest.mark.parametrize("M", [9, 13, 16])
def test_small_batch_on_a_large_matrix(gpu, oracle, K, N, group, zeros, M):
    t = synthetic.random_gptq(K, N, group, seed=K + N, zeros=zeros)
    h = register(gpu, f"gs_{K}_{N}_{M}", t)
    hb = gpu.f32_upload(f"gsb_{K}_{N}_{M}", np.random.default_rng(N).standard_normal(N).astype(np.float32))
    bias = np.random.default_rng(N).standard_normal(N).astype(np.float32)
    x = np.random.default_rng(M).standard_normal((M, K)).astype(np.float32)
    x16 = x.astype(np.float16)
    ref = oracle.gemm_nt_ref(x16.astype(np.float32), oracle_weight(oracle, t), M, N, K) + bias
    p = gpu.plan(h, M, "f32")
    if p["kernel_name"] == "gemm_tc":
        assert p["block"] == 256 and p["launches"] == 1
    for act, xin in (("f16", x16), ("f32", x)):
        first = run_linear(gpu, h, xin, M, N, hb, act=act, out=act)
        assert_close(oracle, first, ref, 1e-3, f"{K}x{N} M={M} {act}")
        assert np.array_equal(first, run_linear(gpu, h, xin, M, N, hb, act=act, out=act))  # slices are added in order


@pytest.mark.parametrize("K,N", [(8576, 1056), (2560, 3360)])
@pytest.mark.parametrize("split", [0, 1, 2, 20, 64])
def test_every_number_of_slices(gpu, oracle, K, N, split):
    """The kernel for certain (its plan has blocks of 256), at the planner's number of slices and at given ones: one, halves, a last
    slice shorter than the others or of a single chunk."""
    t = synthetic.random_gptq(K, N, 128, seed=K + N, zeros="any")
    h = register(gpu, f"gss_{K}_{N}_{split}", t)
    x = np.random.default_rng(split).standard_normal((11, K)).astype(np.float32)
    ref = oracle.gemm_nt_ref(x.astype(np.float16).astype(np.float32), oracle_weight(oracle, t), 11, N, K)
    gpu.plan_override(0, split)
    try:
        for act in ("f16", "f32"):
            p = gpu.plan(h, 11, act)
            taken = p["block"] == 256 and p["launches"] == 1
            if split:  # slices that are too long for the shared memory, or would be empty, stay with the tcgen05 kernel
                per = -(-(K // 128) // min(split, K // 128))
                assert taken == (-(-(K // 128) // per) == min(split, K // 128) and per <= 25), p
            assert p["kernel_name"] == "gemm_tc" and (taken or split), p
            assert_close(oracle, run_linear(gpu, h, x.astype(np.float16) if act == "f16" else x, 11, N, act=act, out=act), ref, 1e-3, f"{K}x{N} {split} {act}")
    finally:
        gpu.plan_override(0, 0)


@pytest.mark.parametrize("K,N,small", [(896, 9728, True), (1152, 8224, True), (896, 4864, False), (1152, 8228, False)])
def test_which_calls_it_takes_on_wide_matrices(gpu, K, N, small):
    """Short K, wide N, 9 to 16 rows: fp16 activations where the matrix has 8 M weights and whole tiles; f32 activations stay with the
    GEMV, which keeps their bits."""
    h = register(gpu, f"gsp_{K}_{N}", synthetic.random_gptq(K, N, 128, seed=N))
    for M in (8, 9, 12, 13, 16):
        f16, f32 = gpu.plan(h, M, "f16"), gpu.plan(h, M, "f32")
        assert (f16["kernel_name"] == "gemm_tc" and f16["block"] == 256) == (small and M > 8), (M, f16)
        assert (f16["kernel_name"] == "gemv_mma") == (M <= 8 or (M <= 12 and not small)), (M, f16)
        assert f32["kernel_name"] == "gemv_mma", (M, f32)


@pytest.mark.parametrize("K,N", [(896, 9728), (2560, 3360)])
def test_column_sharded_calls_on_its_matrices(gpu, oracle, K, N):
    """A call with a placement has no use of the kernel by itself, but may write the dense piece with it that a scatter launch spreads
    (short K) or go to the tcgen05 kernel's own placement: the tensor equals the product, the columns beside it are left alone."""
    t = synthetic.random_gptq(K, N, 128, seed=N, zeros="any")
    h = register(gpu, f"gsg_{K}_{N}", t)
    x = np.random.default_rng(K).standard_normal((9, K)).astype(np.float16)
    ref = oracle.gemm_nt_ref(x.astype(np.float32), oracle_weight(oracle, t), 9, N, K)
    gpu.arena.reset()
    A, full, tmp = gpu.arena.alloc(9 * K, [9, K], "f16"), gpu.arena.alloc(9 * (N + 64), [9, N + 64], "f32"), gpu.arena.alloc(9 * N, [9, N], "f32")
    gpu.write(A, x)
    gpu.write(full, np.full(9 * (N + 64), -7.0, np.float32))
    gpu.linear_gather(h, A, full, tmp, None, 9, N + 64, 32, [])
    got = gpu.read(full).reshape(9, N + 64)
    assert np.all(got[:, :32] == -7.0) and np.all(got[:, 32 + N:] == -7.0)
    assert_close(oracle, got[:, 32:32 + N], ref, 1e-3, f"{K}x{N}")
