"""GPU parity of the int4 GEMM with its weights in tensor memory (up to 128 rows): row counts around its tiles, columns and K that do not
fill theirs, groups smaller and larger than its chunks, every number of slices, both activation and result types."""
import json
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from helpers import assert_close, oracle_weight, register, run_linear
from webllm_b200 import synthetic

pytestmark = pytest.mark.gpu

BLOCK = 896  # of its plans


def _reference(oracle, t, x16, M, N, K, bias=0.0):
    W16 = oracle.round_f16(oracle_weight(oracle, t)).reshape(N, K)
    return oracle.gemm_nt_ref(x16.astype(np.float32), W16, M, N, K) + bias


# K 832 and 1472: the last chunk of 128 is half there; N 1236 and 2052: the last tile, zero word and 16-byte store are not full
@pytest.mark.parametrize("K,N,group,zeros", [(896, 4864, 128, "any"), (832, 1236, 64, "any"), (1472, 2052, 192, "7or8"), (1152, 264, 384, "none"),
                                             (256, 128, 128, "any"), (64, 260, 64, "any")])
@pytest.mark.parametrize("M", [17, 32, 63, 65, 128])
def test_rows_columns_and_groups(gpu, oracle, K, N, group, zeros, M):
    t = synthetic.random_gptq(K, N, group, seed=K + N, zeros=zeros)
    h = register(gpu, f"th_{K}_{N}_{M}", t)
    bias = np.random.default_rng(N).standard_normal(N).astype(np.float32)
    hb = gpu.f32_upload(f"thb_{K}_{N}_{M}", bias)
    x = np.random.default_rng(M).standard_normal((M, K)).astype(np.float32)
    x16 = x.astype(np.float16)
    ref = _reference(oracle, t, x16, M, N, K, bias)
    assert gpu.plan(h, M, "f16")["block"] == BLOCK
    for act, xin in (("f16", x16), ("f32", x)):
        first = run_linear(gpu, h, xin, M, N, hb, act=act, out=act)
        assert_close(oracle, first, ref, 1e-3, f"{K}x{N} M={M} {act}")
        assert np.array_equal(first, run_linear(gpu, h, xin, M, N, hb, act=act, out=act))


@pytest.mark.parametrize("split", range(1, 9))
@pytest.mark.parametrize("M", [20, 100])
def test_every_number_of_slices(gpu, oracle, split, M):
    """Clusters of one to eight CTAs: rows that do not divide by them, a last slice shorter than the others, CTAs with fewer chunks than
    accumulators."""
    K, N = 3456, 392  # 27 chunks
    t = synthetic.random_gptq(K, N, 128, seed=split, zeros="any")
    h = register(gpu, f"ths_{split}_{M}", t)
    x16 = np.random.default_rng(split).standard_normal((M, K)).astype(np.float16)
    ref = _reference(oracle, t, x16, M, N, K)
    gpu.plan_override(0, split)
    try:
        p = gpu.plan(h, M, "f16")
        taken = -(-27 // -(-27 // split)) == split  # (no slice would be empty)
        assert (p["block"] == BLOCK and p["split_k"] == split) == taken, p
        assert_close(oracle, run_linear(gpu, h, x16, M, N, act="f16", out="f32"), ref, 1e-3, f"{split} slices")
    finally:
        gpu.plan_override(0, 0)


def test_more_tiles_than_sms(gpu, oracle):
    K, N, M = 256, 19460, 24
    t = synthetic.random_gptq(K, N, 128, seed=1, zeros="any")
    h = register(gpu, "th_wide", t)
    x16 = np.random.default_rng(1).standard_normal((M, K)).astype(np.float16)
    assert gpu.plan(h, M, "f16")["block"] == BLOCK
    assert_close(oracle, run_linear(gpu, h, x16, M, N, act="f16", out="f16"), _reference(oracle, t, x16, M, N, K), 1e-3, "wide")


def test_infinities_and_nan_stay_in_their_rows(gpu, oracle):
    """K ends inside a chunk and the row count inside a tile: what lies beyond both must not meet a row that holds no number."""
    K, N, M = 832, 132, 19
    t = synthetic.random_gptq(K, N, 64, seed=3, zeros="any")
    h = register(gpu, "th_inf", t)
    x = np.random.default_rng(3).standard_normal((M, K)).astype(np.float16)
    x[4, 831], x[7, 0] = np.inf, np.nan
    got = run_linear(gpu, h, x, M, N, act="f16", out="f32").reshape(M, N)
    clean = [m for m in range(M) if m not in (4, 7)]
    ref = _reference(oracle, t, x[clean], len(clean), N, K).reshape(len(clean), N)
    assert np.isnan(got[7]).all() and not np.isfinite(got[4]).any()
    assert_close(oracle, got[clean].ravel(), ref.ravel(), 1e-3, "rows beside them")


@pytest.mark.parametrize("K,N,M", [(896, 1152, 404), (1472, 260, 129), (896, 132, 1000), (3456, 392, 300), (896, 4868, 177), (512, 9604, 256)])
def test_several_row_tiles(gpu, oracle, K, N, M):
    """Row tiles of equal size (up to 128 or up to 256 rows), the last one not full, alone and with slices."""
    t = synthetic.random_gptq(K, N, 64, seed=M, zeros="any")
    h = register(gpu, f"thm_{K}_{M}", t)
    bias = np.random.default_rng(N).standard_normal(N).astype(np.float32)
    hb = gpu.f32_upload(f"thmb_{K}_{M}", bias)
    x = np.random.default_rng(M).standard_normal((M, K)).astype(np.float32)
    x16 = x.astype(np.float16)
    ref = _reference(oracle, t, x16, M, N, K, bias)
    p = gpu.plan(h, M, "f16")
    assert p["block"] == BLOCK and p["grid_x"] in (-(-M // 128), -(-M // 256)) and p["grid_x"] * p["tile_m"] >= M, p
    for split in (0, 1, 3):
        gpu.plan_override(0, split)
        try:
            for act, xin, out in (("f16", x16, "f32"), ("f32", x, "f16")):
                assert_close(oracle, run_linear(gpu, h, xin, M, N, hb, act=act, out=out), ref, 1e-3, f"{K}x{N} M={M} {act} split {split}")
        finally:
            gpu.plan_override(0, 0)


@pytest.mark.parametrize("M,split", [(1100, 2), (1280, 2), (2300, 1), (2368, 1)])
def test_long_k_and_many_rows_by_themselves(gpu, oracle, M, split):
    """Slices of 128-row tiles while two fit, one slice where the tiles fill four fifths of the SMs."""
    K, N = 4864, 896
    t = synthetic.random_gptq(K, N, 128, seed=4, zeros="any")
    h = register(gpu, f"thl_{M}", t)
    x16 = np.random.default_rng(M).standard_normal((M, K)).astype(np.float16)
    p = gpu.plan(h, M, "f16")
    assert p["block"] == BLOCK and p["tile_m"] <= 128 and p["split_k"] == split, p
    rows = [0, 127, 128, 700, M - 1]
    got = run_linear(gpu, h, x16, M, N, act="f16", out="f32").reshape(M, N)
    assert_close(oracle, got[rows].ravel(), _reference(oracle, t, x16[rows], len(rows), N, K), 1e-3, f"{M}")


@pytest.mark.parametrize("var,value,key,want", [("MT", 192, "tile_m", 192), ("NH", 2, "tile_n", 256), ("SPLIT", 3, "split_k", 3), ("THIN", 0, None, None)])
def test_pins_hold_where_this_kernel_would_be_taken(gpu, var, value, key, want):
    """The switches are read once per process, so a child asks for the plan."""
    h = register(gpu, f"thp_{var}", synthetic.random_gptq(896, 1152, 128, seed=2))
    assert gpu.plan(h, 404, "f16")["block"] == BLOCK
    code = ("import json; from webllm_b200 import Gpu, synthetic\n"
            "with Gpu(0, weight_bytes=16 << 20, act_bytes=16 << 20) as g:\n"
            "    t = synthetic.random_gptq(896, 1152, 128, seed=2)\n"
            "    h = g.gptq_register('w', t.qweight, t.qzeros, t.scales, 896, 1152, 128)\n"
            "    print(json.dumps(g.plan(h, 404, 'f16')))\n")
    r = subprocess.run([sys.executable, "-c", code], env={**os.environ, f"WEBLLM_B200_GEMM_{var}": str(value)}, capture_output=True, text=True,
                       cwd=Path(__file__).resolve().parent.parent, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    p = json.loads(r.stdout.splitlines()[-1])
    assert p["block"] != BLOCK and (key is None or p[key] == want), p
