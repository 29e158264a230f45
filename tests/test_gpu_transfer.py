"""Host <-> device copies at the sizes where transfer.cu changes its ways: below and at 2 MB, a whole and a broken last piece, more
pieces than slots, an odd host address; from several threads at once; from pinned memory."""
import threading

import numpy as np
import pytest

from webllm_b200 import Gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbytes", [1, (2 << 20) - 4, 2 << 20, (2 << 20) + 12, (8 << 20) + (512 << 10), (33 << 20) + 3])
def test_round_trip(built_lib, nbytes):
    src = np.random.default_rng(nbytes).integers(0, 256, nbytes + 1, dtype=np.uint8)[1:]  # an odd address
    with Gpu(0, weight_bytes=1 << 20, act_bytes=nbytes + 8192) as gpu:
        t = gpu.arena.alloc((nbytes + 3) // 4)
        gpu.write_bytes(t.offset, src)
        assert np.array_equal(gpu.read(t).view(np.uint8)[:nbytes], src)


def test_threads_and_pinned_memory(built_lib):
    import torch
    n, bad = 5 << 20, []

    def work(seed):
        src = torch.from_numpy(np.random.default_rng(seed).integers(0, 256, n, dtype=np.uint8))
        src = (src.pin_memory() if seed % 2 else src).numpy()
        with Gpu(0, weight_bytes=1 << 20, act_bytes=n + 8192) as gpu:
            t = gpu.arena.alloc(n // 4)
            for _ in range(5):
                gpu.write_bytes(t.offset, src)
                if not np.array_equal(gpu.read(t).view(np.uint8), src):
                    bad.append(seed)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not bad
