"""The tensor-core GEMMs whose unpack sets do not divide the stages of their ring (gemm_tc.cuh: mbar_wait_set): every tile shape that has
such a ring, over weights that come from memory, many launches behind one another. What goes wrong without the wait is one launch in a
great many, so all of a shape's results are compared, bit for bit."""
import numpy as np
import pytest

from helpers import assert_close, oracle_weight
from webllm_b200 import Gpu, _lib, synthetic

pytestmark = pytest.mark.gpu

COPIES = 64  # of 2.2 MB: more than the L2 holds
TC, PAIR = _lib.WB_KERNEL_GEMM_TC, _lib.WB_KERNEL_GEMM_TC_PAIR


@pytest.fixture(scope="module", params=[(4864, 896), (896, 4864)], ids=["long_k", "wide"])
def weights(built_lib, oracle, request):
    K, N = request.param
    t = synthetic.random_gptq(K, N, 128, seed=5, zeros="any")
    W16 = oracle.round_f16(oracle_weight(oracle, t)).reshape(N, K)
    with Gpu(0, weight_bytes=256 << 20, act_bytes=96 << 20) as g:
        yield g, [g.gptq_register(f"ring_{i}", t.qweight, t.qzeros, t.scales, K, N, 128) for i in range(COPIES)], W16


# long K: stages and sets 6 and 4, 5 and 4, 3 and 2, 3 and 2; pairs 6 and 4 (tiles of 128 and 192 rows) and, with staging tiles, 5 and 4.
# Wide: the persistent loop of the one-CTA kernel, 6 and 4, 5 and 4.
CASES = {4864: [(1800, TC, 1, (128, 128)), (1800, TC, 6, (192, 128)), (1800, TC, 3, (192, 256)), (1800, TC, 8, (256, 256)),
                (1800, PAIR, 1, (128, 256)), (1800, PAIR, 3, (192, 256)), (1800, PAIR, 4, (256, 256))],
         896: [(800, TC, 1, (128, 128)), (2000, TC, 1, (192, 128))]}


def test_every_launch_gives_the_same_bits(weights, oracle):
    g, hs, W16 = weights
    N, K = W16.shape
    for M, kind, split, tile in CASES[K]:
        x = np.random.default_rng(M).standard_normal((M, K)).astype(np.float16)
        rows = [0, 1, 127, 128, 700, M - 1]
        ref = oracle.gemm_nt_ref(x[rows].astype(np.float32), W16, len(rows), N, K, threads=oracle.max_threads())
        g.arena.reset()
        A, C = g.arena.alloc(M * K, [M, K], "f16"), g.arena.alloc(M * N, [M, N])
        g.write(A, x)
        g.plan_override(kind, split)
        try:
            p = g.plan(hs[0], M, "f16")
            assert (p["kernel"], p["split_k"], p["tile_m"], p["tile_n"]) == (kind, split, *tile), p
            g.linear(hs[0], A, C, None, M)
            first = g.read(C).reshape(M, N)
            assert_close(oracle, first[rows], ref, 1e-3, f"{p}")
            for n in [COPIES] * 3 + [5] * 12:  # read after many and after few
                for h in hs[-n:]:
                    g.linear(h, A, C, None, M)
                assert np.array_equal(g.read(C).reshape(M, N), first), p
        finally:
            g.plan_override(0, 0)
