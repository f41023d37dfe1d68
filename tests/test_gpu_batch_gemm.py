"""GPU parity of the tensor-core GEMM behind token batches (powerserve_b200/csrc/ps_tc.cuh) at the edges of its tiling: batches on both
sides of every column-tile width and over more than one column tile, matrices whose rows do not fill a 128-row tile (q | k | v segments
that start on tile borders, biases), an odd number of super-blocks, and shapes for which a CTA's share is one pass, two or more.
Oracle: the plain-C restatement of the reference; tolerance zero (the contract of this path)."""
import numpy as np
import pytest

from powerserve_b200 import capi, gguf, synth
from tests import _libs as L
from tests import _model as M

pytestmark = pytest.mark.gpu

# 3 and 5 super-blocks; q 6, k and v 1.5 row tiles, gate / up 10, output 50 and a bit
ODD = synth.ModelShape("tc-odd", "llama", 768, 1280, 2, 8, 2, 96, 6400 + 24, False, 0, 5e5, 1e-5, gguf.GGML_Q4_K, n_ctx=512, qkv_bias=True)


@pytest.fixture(scope="module")
def odd(tmp_path_factory):
    d = synth.write_model_dir(str(tmp_path_factory.mktemp("tc_odd")), ODD, seed=5)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=200)
    yield om, cm
    om.close()
    cm.close()


@pytest.mark.parametrize("bs", [6, 16, 17, 32, 33, 64, 65, 96, 97, 128, 129, 200])
def test_batch_widths(odd, bs):
    om, cm = odd
    tokens = synth.random_prompt(ODD.vocab_size, bs, seed=bs)
    om.reset()
    cm.reset()
    n = cm.be.counter("tc_gemm_launches")
    got = cm.forward(tokens)
    assert cm.be.counter("tc_gemm_launches") > n
    L.assert_bit_equal(got, om.forward(tokens), f"{bs} tokens")


def test_shares_of_two_passes():
    """layer shapes of an 8B model: 48 row tiles of q | k | v, 288 passes for 148 SMs"""
    d = M.model_dir("slice-8b")
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=32)
    tokens = synth.random_prompt(2048, 20, seed=3)
    L.assert_bit_equal(cm.forward(tokens), om.forward(tokens), "8B slice, 20 tokens")
    assert cm.be.counter("tc_gemm_pass2") > 0
    again = cm.forward(tokens[:9])          # the counters of the shared tiles are left as they were found
    assert np.isfinite(again).all() and cm.be.counter("tc_error") == 0
    L.assert_bit_equal(again, om.forward(tokens[:9]), "8B slice, 9 more tokens")
    om.close()
    cm.close()


@pytest.mark.parametrize("width", [16, 32, 48, 64])
def test_a_warp_that_gives_up_ends_the_call(width):
    """one warp of every CTA takes its first wait as run out - the first and the last epilogue warp while the others of the tile go on to hand numbers
    over, the first and the last de-quantising one, the copies' warp, the issuing one: every other wait ends by its own limit, the call reports the
    time-out, and the next call on the same context has all bits.  All products of an 8B layer on `width` tokens take tiles of that many columns;
    a number behind the last warp of theirs is nobody's, and the call goes through."""
    d = M.model_dir("slice-8b")
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=64)
    tokens = synth.random_prompt(2048, width, seed=width)
    want = om.forward(tokens)
    om.close()
    copies = 8 + (16 if width <= 32 else 8)                  # epilogue, then de-quantising warps
    for warp in (0, 7, 8, copies - 1, copies, copies + 1):
        cm.reset()
        cm.be.set_option("give_up_warp", warp)
        with pytest.raises(capi.PsCudaError, match="tcgen05 pipeline time-out"):
            cm.forward(tokens)
        cm.be.set_option("give_up_warp", -1)
        cm.reset()
        L.assert_bit_equal(cm.forward(tokens), want, f"after warp {warp} gave up")
    for warp in (copies + 4, 40):
        cm.reset()
        cm.be.set_option("give_up_warp", warp)
        L.assert_bit_equal(cm.forward(tokens), want, f"no warp {warp}")
    cm.close()


def test_shares_of_one_pass_and_of_more_than_two(odd):
    """what the widths above are spread over: 4 to 10 row tiles, and the head's 51"""
    cm = odd[1]
    cm.reset()
    n = [cm.be.counter(f"tc_gemm_pass{p}") for p in (1, 6)]
    cm.forward(synth.random_prompt(ODD.vocab_size, 40, seed=40))
    assert cm.be.counter("tc_gemm_pass1") > n[0] and cm.be.counter("tc_gemm_pass6") > n[1]


@pytest.mark.parametrize("bs", [97, 128])
def test_two_column_tiles_of_64(bs):
    """an 8B layer's products on more tokens than the widest tile has columns"""
    d = M.model_dir("slice-8b")
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=128)
    tokens = synth.random_prompt(2048, bs, seed=bs)
    L.assert_bit_equal(cm.forward(tokens), om.forward(tokens), f"8B slice, {bs} tokens")
    om.close()
    cm.close()


def test_workspace_follows_the_batch():
    """the numbers of shared tiles need a slot per SM for tiles of as many columns as max_batch has, up to 64: 7 MB for 16, 29 MB for 64"""
    import torch
    d, used = M.model_dir("tiny-llama"), {}
    for batch in (16, 64, 16, 64):      # (the first model of a process brings the kernels' own memory along)
        before = torch.cuda.mem_get_info()[0]
        cm = capi.CudaModel(d, max_batch=batch)
        used[batch] = before - torch.cuda.mem_get_info()[0]
        cm.close()
    slot = 148 * 6 * 128 * 4
    assert used[64] - used[16] > 0.8 * slot * (64 - 16), used
