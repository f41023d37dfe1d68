"""GPU parity of the products of token batches that run on the CUDA cores (ps_k_matmul_qb on GGUF rows, ps_k_matmul_ob on octet copies)
where their shapes change, and their way out.  Oracle: the plain-C restatement of the reference; tolerance zero."""
import numpy as np
import pytest

from powerserve_b200 import capi, gguf, synth
from tests import _libs as L
from tests import _model as M

pytestmark = pytest.mark.gpu


def _shape(quant, dim, ffn, heads, vocab):
    return synth.ModelShape("products", "llama", dim, ffn, 1, heads, heads, dim // heads, vocab, False, 0, 1e4, 1e-5, quant, n_ctx=64)


@pytest.mark.parametrize("quant", [gguf.GGML_Q8_0, gguf.GGML_Q4_0])
def test_a_warp_that_gives_up_ends_the_call(quant, tmp_path):
    """octet copies: one warp of every CTA takes its first piece as not arrived; the call says so and the next one has all bits"""
    d = synth.write_model_dir(str(tmp_path / "m"), _shape(quant, 256, 512, 4, 512), seed=3)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=8)
    assert cm.be.counter("mv32_ok") == 1
    tokens = synth.random_prompt(512, 5, seed=1)
    want = om.forward(tokens)
    for warp in (0, 3):
        cm.be.set_option("give_up_warp", warp)
        with pytest.raises(capi.PsCudaError, match="copy of a batch product"):
            cm.forward(tokens)
        cm.be.set_option("give_up_warp", -1)
        cm.reset()
        L.assert_bit_equal(cm.forward(tokens), want, f"after warp {warp} gave up")
        cm.reset()
    om.close()
    cm.close()
