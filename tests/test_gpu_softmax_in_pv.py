"""The P.V kernel of batches takes the soft-max of its rows with it where its blocks fill the GPU and on short rows, else a launch before it does: rows of fewer than eight and
32 positions and with leftovers of both, the last length of one side and the first of the other, blocks that are not full, masks of a tree.  Oracle: the first-generation kernels
(option attn_tile 0), whose soft-max is a launch of its own; tolerance zero."""
import numpy as np
import pytest

from powerserve_b200 import capi, gguf, synth
from tests import _libs as L

pytestmark = pytest.mark.gpu
SHAPES = {
    "hs64": synth.ModelShape("sp-64", "llama", 256, 512, 1, 7, 1, 64, 520, False, 0, 1e4, 1e-5, gguf.GGML_Q8_0, n_ctx=1500),
    "hs128": synth.ModelShape("sp-128", "llama", 512, 512, 1, 32, 4, 128, 520, False, 0, 1e4, 1e-5, gguf.GGML_Q4_K, n_ctx=1500),
}
#: cached positions before, rows: 256 and 257 positions lie on either side of the line for few blocks; 32 heads x 40 rows and more fill the GPU at any length
PORTIONS = [(0, 5), (0, 7), (0, 31), (0, 32), (0, 33), (240, 16), (241, 16), (900, 12), (1001, 40), (1400, 64)]


@pytest.mark.parametrize("name", sorted(SHAPES))
def test_same_bits_as_a_launch_of_its_own(name, tmp_path):
    cm = capi.CudaModel(synth.write_model_dir(str(tmp_path), SHAPES[name], seed=5), max_batch=64)
    toks = synth.random_prompt(500, 1500, seed=2)
    tree = np.tril(np.ones((11, 11), np.uint8))
    tree[7, 2:6] = 0
    got = {}
    for tiled in (0, 1):
        cm.be.set_option("attn_tile", tiled)
        out = []
        for ctx, n in PORTIONS:
            cm.reset()
            if ctx:
                cm.prefill(np.r_[toks[:ctx], toks[:1]], 64)
            out.append(cm.forward(toks[ctx:ctx + n]))
        for ctx in (5, 1100):
            cm.reset()
            cm.prefill(np.r_[toks[:ctx], toks[:1]], 64)
            out.append(cm.forward_tree(toks[ctx:ctx + 11], [ctx + min(i, 6) for i in range(11)], tree))
        got[tiled] = out
    cm.close()
    for a, b, what in zip(got[1], got[0], PORTIONS + [5, 1100]):
        L.assert_bit_equal(a, b, f"{name} {what}")


@pytest.mark.parametrize("rest", range(1, 8))
def test_leftovers_that_other_lanes_stored(rest, tmp_path):
    """rows whose last one to seven positions begin at lane 8, 16 or 24 of a chunk: the lane that takes the exponential of such a position is not the one that stored its score"""
    cm = capi.CudaModel(synth.write_model_dir(str(tmp_path), SHAPES["hs64"], seed=6), max_batch=64)
    toks = synth.random_prompt(500, 300, seed=rest)
    got = {}
    for tiled in (0, 1):
        cm.be.set_option("attn_tile", tiled)
        got[tiled] = []
        for n8 in (8, 16, 24, 40, 208):
            cm.reset()
            if n8 > 32:
                cm.prefill(np.r_[toks[:n8 - 8], toks[:1]], 64)
            lo = cm.position
            got[tiled].append(cm.forward(toks[lo:n8 + rest]))
    cm.close()
    for a, b in zip(got[1], got[0]):
        L.assert_bit_equal(a, b, f"rest {rest}")
