"""A recorded command batch runs calls that share no tensors side by side: reads after writes, overwritten inputs, overwritten
results, partly overlapping tensors, calls that use scratch and calls that keep stream order in between."""
import numpy as np
import pytest

from helpers import register
from webllm_b200 import Gpu, Tensor, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 4, 8, 24, 40])
def test_recorded_calls_see_their_inputs(built_lib, M):
    K = 512
    with Gpu(0, weight_bytes=64 << 20, act_bytes=64 << 20) as gpu:
        w = [register(gpu, f"w{i}", synthetic.random_gptq(K, K, 128, seed=i)) for i in range(3)]
        wide = register(gpu, "wide", synthetic.random_gptq(K, 4 * K, 128, seed=9))
        deq = gpu.arena.alloc(K * K, [K, K])
        t = [gpu.arena.alloc(M * K, [M, K]) for _ in range(6)]
        long = gpu.arena.alloc(M * 4 * K, [M, 4 * K])
        tail = Tensor(long.offset + 3 * M * K * 4, M * K, [M, K])  # the last quarter of `long`
        many = [gpu.arena.alloc(M * K, [M, K]) for _ in range(11)]
        x = np.random.default_rng(M).standard_normal(M * K).astype(np.float32)

        def calls():
            gpu.linear(w[0], t[0], t[1], None, M)
            gpu.linear(w[1], t[0], t[2], None, M)    # beside the first
            gpu.linear(w[2], t[1], t[3], None, M)    # after the first
            gpu.linear(w[0], t[2], t[0], None, M)    # overwrites what the first two read
            gpu.linear(w[1], t[3], t[2], None, M)    # overwrites what the fourth read
            gpu.linear(wide, t[0], long, None, M)
            gpu.linear(w[2], tail, t[4], None, M)    # part of the result before
            gpu.gptq_dequant(w[0], deq)              # stream order
            gpu.linear(w[0], t[4], t[5], None, M)
            gpu.linear(w[1], t[5], t[4], None, M)
            for i, y in enumerate(many):             # more than run side by side
                gpu.linear(w[i % 3], t[5], y, None, M)
            gpu.linear(w[0], many[0], t[1], None, M)

        def result(run):
            gpu.write(t[0], x)
            run()
            return [gpu.read(v) for v in (*t, *many, long, deq)]

        ref = result(calls)
        with gpu.batch() as b:
            calls()
        for _ in range(3):
            for got, want in zip(result(b.submit), ref):
                assert np.array_equal(got, want)
        b.destroy()
