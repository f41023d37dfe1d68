"""Kernels of a batch start while the one before still runs (programmatic dependence) and ask for weights before they wait for it.  Oracle: the same
calls with each kernel after the other (option pdl 0); tolerance zero.  Depths of the products in steps of the batch GEMM: fewer than its stages
(512: 1), as many (3072: 6) and more (4096: 8)."""
import numpy as np
import pytest

from powerserve_b200 import capi, gguf, synth
from tests import _libs as L

pytestmark = pytest.mark.gpu
SHAPES = {
    "q4_k": synth.ModelShape("dl-k", "llama", 512, 4096, 3, 8, 2, 64, 1000, False, 0, 1e4, 1e-5, gguf.GGML_Q4_K, n_ctx=256),
    "q4_k_long": synth.ModelShape("dl-l", "llama", 3072, 512, 2, 24, 8, 128, 520, False, 0, 1e4, 1e-5, gguf.GGML_Q4_K, n_ctx=256),
    "q8_0": synth.ModelShape("dl-8", "qwen2", 160, 224, 3, 5, 1, 32, 520, True, 2, 1e6, 1e-6, gguf.GGML_Q8_0, n_ctx=256, qkv_bias=True),
}


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_same_bits_as_one_kernel_after_the_other(name, tmp_path):
    sh = SHAPES[name]
    cm = capi.CudaModel(synth.write_model_dir(str(tmp_path), sh, seed=9), max_batch=64)
    toks = synth.random_prompt(500, 200, seed=3)
    got = []
    for pdl in (0, 1, 1):
        cm.be.set_option("pdl", pdl)
        cm.reset()
        out = [cm.forward(toks[:64]), cm.forward(toks[64:77]), cm.forward(toks[77:79])]
        n = 9
        mask = np.tril(np.ones((n, n), np.uint8))
        mask[5, 3] = 0
        out.append(cm.forward_tree(toks[79:79 + n], [cm.position + min(i, 6) for i in range(n)], mask))
        cm.reset()
        ids = [0] + [cm.session_create() for _ in range(17)]
        for step in range(2):
            out.append(cm.forward_sessions(ids, toks[100 + 18 * step:118 + 18 * step])[0])
        for i in ids[1:]:
            cm.session_destroy(i)
        got.append(out)
    cm.close()
    for run in got[1:]:
        for a, b in zip(run, got[0]):
            L.assert_bit_equal(a, b, name)
