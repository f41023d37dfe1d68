"""GPU parity of the batch products of 32-element blocks on the tensor cores (ps_k_matmul_mt) at their edges: rows and row blocks that do not fill a tile
or a group, one to four column tiles a unit, more units than CTAs, and the kernel that takes over where its weight records found no room.  Oracle: the
plain-C restatement of the reference; tolerance zero."""
import pytest

from powerserve_b200 import capi, gguf, synth
from tests import _libs as L
from tests import _model as M

pytestmark = pytest.mark.gpu
# width, feed-forward rows, heads, kv heads, vocabulary.  18 952 rows are 1 185 tiles: units of four column tiles from 25 columns on, of two from 9;
# 160 and 416 elements are 5 and 13 blocks; 264 rows are 16.5 tiles
SHAPES = {"wide_head": (160, 416, 5, 1, 18952), "long_rows": (256, 9760, 4, 2, 264)}


@pytest.fixture(scope="module", params=[(n, q) for n in sorted(SHAPES) for q in (gguf.GGML_Q4_0, gguf.GGML_Q8_0)], ids=lambda p: f"{p[0]}-{p[1]}")
def pair(request, tmp_path_factory):
    name, quant = request.param
    dim, ffn, nh, nkv, vocab = SHAPES[name]
    shape = synth.ModelShape("mt-" + name, "qwen2", dim, ffn, 1, nh, nkv, dim // nh, vocab, True, 2, 1e6, 1e-6, quant, n_ctx=128, qkv_bias=True)
    d = synth.write_model_dir(str(tmp_path_factory.mktemp("mt")), shape, seed=8)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=70)
    assert cm.be.counter("mv32_ok") == 1 and cm.be.counter("mt_ok") == 1
    yield om, cm, vocab
    om.close()
    cm.close()


@pytest.mark.parametrize("n", [2, 7, 8, 9, 17, 25, 32, 33, 70])
def test_columns(pair, n):
    om, cm, vocab = pair
    tokens = synth.random_prompt(vocab, n, seed=n)
    om.reset()
    want = om.forward(tokens)
    for mt_min in (2, 1000):
        cm.be.set_option("mt_min", mt_min)
        cm.reset()
        launches = cm.be.counter("mt_launches")
        L.assert_bit_equal(cm.forward(tokens), want, f"{n} tokens, mt_min {mt_min}")
        assert cm.be.counter("mt_launches") - launches == (5 if mt_min == 2 else 0)
    cm.be.set_option("mt_min", 2)


def test_more_than_a_million_rows(tmp_path):
    """a head of 65 535 x 16 rows and more: a launch's y and z end at 65 535"""
    vocab = 65535 * 16 + 1000
    shape = synth.ModelShape("mt-rows", "llama", 64, 64, 1, 2, 2, 32, vocab, True, 0, 1e4, 1e-5, gguf.GGML_Q4_0, n_ctx=32)
    d = synth.write_model_dir(str(tmp_path), shape, seed=8)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=4)
    assert cm.be.counter("mv32_ok") == 1
    tokens = synth.random_prompt(vocab, 3, seed=1)
    L.assert_bit_equal(cm.forward(tokens), om.forward(tokens), "3 tokens")
    om.close()
    cm.close()
