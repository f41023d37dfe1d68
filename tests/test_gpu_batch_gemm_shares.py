"""GPU parity of the batch GEMM (powerserve_b200/csrc/ps_tc.cuh) where its passes are cut into one share per CTA: shares of one pass, shares that
begin or end inside a tile, inside a pair of passes, that hold whole tiles; every column-tile width at its edges.  Oracle: the plain-C restatement
of the reference; tolerance zero."""
import pytest

from powerserve_b200 import capi, gguf, synth
from tests import _libs as L
from tests import _model as M

pytestmark = pytest.mark.gpu

# row tiles: q | k | v 4, o 2, gate | up 52, down 2, head 101 (the last one has 8 rows); super-blocks of 256: one, and the down product's 13, an odd
# count whose last step is half padding when the rings of five or six stages have gone round
SHAPE = synth.ModelShape("tc-shares", "llama", 256, 256 * 13, 1, 4, 2, 64, 128 * 100 + 8, False, 0, 5e5, 1e-5, gguf.GGML_Q4_K, n_ctx=512)


@pytest.fixture(scope="module")
def pair(tmp_path_factory):
    d = synth.write_model_dir(str(tmp_path_factory.mktemp("tc_shares")), SHAPE, seed=8)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=144)
    yield om, cm
    om.close()
    cm.close()


@pytest.mark.parametrize("bs", [6, 15, 31, 47, 48, 49, 63, 64, 65, 95, 127, 128, 129, 144])
def test_shares(pair, bs):
    om, cm = pair
    tokens = synth.random_prompt(SHAPE.vocab_size, bs, seed=bs)
    om.reset()
    cm.reset()
    L.assert_bit_equal(cm.forward(tokens), om.forward(tokens), f"{bs} tokens")


@pytest.mark.parametrize("bs", [16, 128])
def test_every_role_that_gives_up_ends_the_call(pair, bs):
    """28 warps at 16 columns, 20 at 64: epilogue, de-quantising (first and last of both groups), copies, issuer"""
    om, cm = pair
    tokens = synth.random_prompt(SHAPE.vocab_size, bs, seed=bs)
    om.reset()
    want = om.forward(tokens)
    last = 23 if bs == 16 else 15
    for warp in (0, 3, 7, 8, last, last + 1, last + 2):
        cm.reset()
        cm.be.set_option("give_up_warp", warp)
        with pytest.raises(capi.PsCudaError, match="tcgen05 pipeline time-out"):
            cm.forward(tokens)
        cm.be.set_option("give_up_warp", -1)
        cm.reset()
        L.assert_bit_equal(cm.forward(tokens), want, f"after warp {warp} gave up")
