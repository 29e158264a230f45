"""GPU parity of the decode step in five kernels a layer (qwen_model.cu: norm and silu prologues of the int4 GEMV, rotary embedding and
cache append inside the cluster attention), which serves fused models that the persistent decode kernel does not take: head sizes
other than 64 and a hidden size above 1024. Greedy over the replayed graph and single steps, contexts around the key splits."""
import numpy as np
import pytest

from webllm_b200 import Gpu, QwenGpt, synthetic

from test_gpu_qwen import _dense_from_gptq, _ocfg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,H,KVH,I,prompt,kv", [
    (256, 2, 1, 1280, 7, "f32"),     # head size 128
    (512, 4, 2, 1408, 250, "f16"),
    (3584, 28, 4, 2560, 65, "f16"),  # the attention of a 7B-class model
    (128, 4, 2, 384, 33, "f16"),     # head size 32
    (1152, 18, 2, 1280, 100, "f32"),  # head size 64, too wide for the persistent kernel
])
def test_five_kernel_step_matches_oracle(built_lib, oracle, C, H, KVH, I, prompt, kv):
    cfg = synthetic.QwenShape(500, 2, H, KVH, C, I)
    G = synthetic.random_qwen_gptq(cfg, seed=C + prompt, std=0.05)
    ids = np.random.default_rng(prompt).integers(0, cfg.vocab_size, prompt).astype(np.uint32)
    steps = 12
    ref = oracle.CachedForward(_ocfg(oracle, cfg), _dense_from_gptq(oracle, G), max_t=prompt + 16, kv_f16=kv == "f16",
                               threads=oracle.max_threads())
    tok = first = oracle.sample_greedy(ref.prefill(ids))
    want = []
    for _ in range(steps):
        row = ref.decode_step(tok)
        tok = oracle.sample_greedy(row)
        want.append(tok)
    rms = float(np.sqrt(np.mean(row.astype(np.float64) ** 2)))
    with Gpu(0, weight_bytes=256 << 20, act_bytes=256 << 20) as gpu:
        model = QwenGpt(gpu, cfg, max_t=prompt + 16, kv_dtype=kv)
        model.upload_gptq_model(G, fuse=True)
        model.set_exact(True)
        model.prefill(ids, last_only=True)
        assert model.decode_greedy(first, steps).tolist() == want
        assert oracle.check_tolerance(model.last_logits(), row, 5e-4 * rms, 5e-4).ok  # as the persistent kernel is held to
        model.reset_cache()
        model.prefill(ids, last_only=True)
        for t in [first] + want[:3]:
            launches = gpu.launch_count
            logits = model.read_tensor(model.decode_step(t))
            assert gpu.launch_count - launches == 5 * cfg.n_layer + 3  # and the embedding, the final norm, lm_head
        assert int(logits.argmax()) == want[3]
        model.close()
