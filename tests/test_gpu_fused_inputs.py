"""GPU parity of the launches that join a product's input to what makes it (norm or SiLU with the quantiser, rotations with the cache stores) at
their edges: rows that do not fill a warp's four blocks, token groups that do not fill 32, one kv head, a mixed file.  Oracle: the plain-C
restatement of the reference; tolerance zero."""
import pytest

from powerserve_b200 import capi, gguf, synth
from tests import _libs as L
from tests import _model as M

pytestmark = pytest.mark.gpu
SHAPES = {
    "q8_0": synth.ModelShape("fi-q8", "qwen2", 160, 224, 2, 5, 1, 32, 520, True, 2, 1e6, 1e-6, gguf.GGML_Q8_0, n_ctx=256, qkv_bias=True),
    "q4_0": synth.ModelShape("fi-q4", "llama", 96, 416, 2, 3, 3, 32, 520, False, 0, 1e4, 1e-5, gguf.GGML_Q4_0, n_ctx=256),
    "mixed": synth.ModelShape("fi-mix", "llama", 256, 768, 2, 4, 2, 64, 520, False, 0, 1e4, 1e-5, gguf.GGML_Q4_K, n_ctx=256, output_type=gguf.GGML_Q6_K),
}


@pytest.fixture(scope="module", params=sorted(SHAPES))
def pair(request, tmp_path_factory):
    d = synth.write_model_dir(str(tmp_path_factory.mktemp("fused_inputs")), SHAPES[request.param], seed=6)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=70)
    yield om, cm
    om.close()
    cm.close()


@pytest.mark.parametrize("cuts", [[2, 1], [31], [32, 33], [64, 5, 1]])
def test_portions(pair, cuts):
    om, cm = pair
    om.reset()
    cm.reset()
    tokens = synth.random_prompt(520, sum(cuts), seed=len(cuts))
    for n in cuts:
        L.assert_bit_equal(cm.forward(tokens[:n]), om.forward(tokens[:n]), f"{n} tokens of {cuts}")
        tokens = tokens[n:]
