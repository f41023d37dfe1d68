"""GPU parity of the products of token batches that run on the CUDA cores (ps_k_matmul_qb on GGUF rows, ps_k_matmul_ob on octet copies)
where their shapes change, and their way out.  Oracle: the plain-C restatement of the reference; tolerance zero."""
import time

import numpy as np
import pytest

from powerserve_b200 import capi, gguf, synth
from tests import _libs as L
from tests import _model as M

pytestmark = pytest.mark.gpu
OCTETS = 1000   # option mt_min: no batch is so wide, so that all run on the octet copies, as where the tensor cores' records find no room


def _shape(quant, dim, ffn, heads, vocab):
    return synth.ModelShape("products", "llama", dim, ffn, 1, heads, heads, dim // heads, vocab, False, 0, 1e4, 1e-5, quant, n_ctx=64)


@pytest.mark.parametrize("quant", [gguf.GGML_Q8_0, gguf.GGML_Q4_0])
def test_a_warp_that_gives_up_ends_the_call(quant, tmp_path):
    """octet copies and records of the tensor cores: one warp of every CTA takes its first piece as not arrived; the call says so and the next one has all bits"""
    d = synth.write_model_dir(str(tmp_path / "m"), _shape(quant, 256, 512, 4, 512), seed=3)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=8)
    assert cm.be.counter("mv32_ok") == 1
    tokens = synth.random_prompt(512, 5, seed=1)
    want = om.forward(tokens)
    for mt_min, warp in ((OCTETS, 0), (OCTETS, 3), (2, 0), (2, 3)):
        cm.be.set_option("mt_min", mt_min)
        cm.be.set_option("give_up_warp", warp)
        with pytest.raises(capi.PsCudaError, match="copy of a batch product"):
            cm.forward(tokens)
        cm.be.set_option("give_up_warp", -1)
        cm.reset()
        L.assert_bit_equal(cm.forward(tokens), want, f"after warp {warp} gave up")
        cm.reset()
    om.close()
    cm.close()


def _product(be, t, w, K, N, x, bs):
    """on ps_k_matmul_qb, whatever the format and the size"""
    be.set_option("mk_min", 1000)
    ref = np.zeros(N * bs, np.float32)
    L.oracle().ps_or_matmul(t, L.vptr(w), K, N, L.fptr(x), bs, L.fptr(ref))
    wd = be.register_weight(w, t, K, N)
    xd, dd = be.upload(x), be.empty(N * bs)
    be.matmul(dd, wd, t, K, N, xd, bs)
    got = dd.numpy()
    xd.free()
    dd.free()
    be.unregister_weight(w)
    return got, ref


@pytest.mark.parametrize("t", [L.Q8_0, L.Q4_0])
@pytest.mark.parametrize("blocks", [1, 3, 4, 6])
def test_infinite_scale_in_the_last_block(t, blocks):
    """a damaged file's scale: an infinity stays one, whatever the number of blocks (groups of four are filled up with zeros)"""
    be = capi.CudaBackend(capi.ModelDesc(256, 512, 1, 4, 4, 64, 512, 64, 1e-5, 64, 0, 1e4, 1.0, 1.0, 0, 8, 0, 1))
    rng = np.random.default_rng(blocks)
    K, N, bs = 32 * blocks, 21, 5
    w = synth.random_blocks(rng, t, N, K, 0.1).reshape(N, blocks, -1)
    w[::2, -1, :2] = np.frombuffer(np.float16(np.inf).tobytes(), np.uint8)
    w[::2, -1, 2:] = 1 if t == L.Q8_0 else 0x99     # quants of one sign: every lane's sum is positive
    got, ref = _product(be, t, np.ascontiguousarray(w.reshape(-1)), K, N, (1 + rng.random(K * bs)).astype(np.float32), bs)
    assert np.isinf(ref.reshape(bs, N)[:, ::2]).all() and np.isfinite(ref.reshape(bs, N)[:, 1::2]).all()
    L.assert_bit_equal(got, ref, f"type {t}, {blocks} blocks")
    be.close()


@pytest.mark.parametrize("quant", [gguf.GGML_Q8_0, gguf.GGML_Q4_0])
def test_infinite_scale_in_the_head(quant, tmp_path, monkeypatch):
    """the same on octet copies, and on the tensor cores' records: rows of the head whose last of five blocks has an infinite scale; a logit is infinite where its eight lanes agree"""
    def damaged(shape, seed=0, plain=synth.generate_tensors):
        tensors = plain(shape, seed)
        raw = next(d for n, _, _, d in tensors if n == "output.weight").view(np.uint8).reshape(2048, 5, -1)
        raw[:, 4, :2] = np.frombuffer(np.float16(np.inf).tobytes(), np.uint8)
        return tensors

    monkeypatch.setattr(synth, "generate_tensors", damaged)
    d = synth.write_model_dir(str(tmp_path / "m"), _shape(quant, 160, 320, 5, 2048), seed=3)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=8)
    assert cm.be.counter("mv32_ok") == 1
    for bs in (2, 4, 8):
        tokens = synth.random_prompt(2048, bs, seed=bs)
        om.reset()
        want = om.forward(tokens)
        for mt_min in (OCTETS, 2):
            cm.be.set_option("mt_min", mt_min)
            cm.reset()
            got = cm.forward(tokens)
            assert np.isinf(want).any() and np.array_equal(want, got, equal_nan=True)
    om.close()
    cm.close()


# 200 KB of shared memory: eight columns up to K = 22 656 (32-element blocks) or 23 552 (256), four up to 45 440 or 47 360, two beyond
@pytest.mark.parametrize("t,K", [(L.Q8_0, 22656), (L.Q8_0, 22688), (L.Q8_0, 45472), (L.Q4_0, 45504), (L.Q6_K, 23808), (L.Q4_K, 47616)])
@pytest.mark.parametrize("bs", [2, 3, 4, 8])
def test_long_rows(t, K, bs):
    be = capi.CudaBackend(capi.ModelDesc(256, K, 1, 4, 4, 64, 512, 64, 1e-5, 64, 0, 1e4, 1.0, 1.0, 0, 8, 0, 1))
    rng = np.random.default_rng(K + bs)
    w = synth.random_blocks(rng, t, 41, K, K ** -0.5).reshape(-1)
    got, ref = _product(be, t, w, K, 41, rng.standard_normal(K * bs).astype(np.float32), bs)
    L.assert_bit_equal(got, ref, f"type {t} K {K} bs {bs}")
    be.close()


@pytest.mark.parametrize("quant", [gguf.GGML_Q8_0, gguf.GGML_Q4_0])
@pytest.mark.parametrize("ffn", [5152, 11040, 23008, 31008])
def test_long_octets(quant, ffn, tmp_path):
    """the down product on octet copies: beside eight staged columns there is room for the octets of four, two or one warp, or for none (then
    ps_k_matmul_qb takes it); two and four columns leave more"""
    d = synth.write_model_dir(str(tmp_path / "m"), _shape(quant, 256, ffn, 4, 512), seed=ffn)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=8)
    cm.be.set_option("mt_min", OCTETS)
    assert cm.be.counter("mv32_ok") == 1
    for bs in (2, 3, 8):
        tokens = synth.random_prompt(512, bs, seed=bs)
        om.reset()
        cm.reset()
        L.assert_bit_equal(cm.forward(tokens), om.forward(tokens), f"ffn {ffn} bs {bs}")
    assert cm.be.counter("mt_launches") == 0
    om.close()
    cm.close()


@pytest.mark.parametrize("t", [L.Q4_K, L.Q5_K, L.Q6_K])
@pytest.mark.parametrize("bs", [2, 4, 7])
def test_rows_of_a_thread(t, bs):
    """one row a thread up to 147 CTAs of 32 rows, two beyond, and two where the columns leave room for few CTAs an SM"""
    be = capi.CudaBackend(capi.ModelDesc(256, 14336, 1, 4, 4, 64, 512, 64, 1e-5, 64, 0, 1e4, 1.0, 1.0, 0, 8, 0, 1))
    rng = np.random.default_rng(bs)
    for K, N in [(512, 4704), (512, 4705), (256, 17), (14336, 2400)]:
        w = synth.random_blocks(rng, t, N, K, K ** -0.5).reshape(-1)
        got, ref = _product(be, t, w, K, N, rng.standard_normal(K * bs).astype(np.float32), bs)
        L.assert_bit_equal(got, ref, f"type {t} {K} x {N} bs {bs}")
    be.close()


def test_rows_too_long_for_eight_octets_of_q8_0(tmp_path):
    """rows of 14336 Q8_0 weights: eight columns' activations leave no room for a single octet, four leave room for one, whose CTAs of one warp take two to three
    times as long as the kernel on the GGUF bytes.  72 tokens are the most at which the octet kernel would take four columns by its number of
    warps alone, at 80 it never does: the portions' times are to be alike, and all bits the same."""
    shape = synth.ModelShape("q8-long-rows", "llama", 1024, 14336, 1, 16, 2, 64, 264, False, 0, 1e4, 1e-5, gguf.GGML_Q8_0, n_ctx=128)
    d = synth.write_model_dir(str(tmp_path), shape, seed=12)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=80)
    cm.be.set_option("mt_min", OCTETS)
    took = {}
    for n in (72, 80):
        tokens = synth.random_prompt(264, n, seed=n)
        om.reset()
        cm.reset()
        L.assert_bit_equal(cm.forward(tokens), om.forward(tokens), f"{n} tokens")
        best = 1e9
        for _ in range(20):
            cm.reset()
            t0 = time.perf_counter()
            cm.forward(tokens, lm_head=False)
            best = min(best, time.perf_counter() - t0)
        took[n] = best
    assert cm.be.counter("mt_launches") == 0
    om.close()
    cm.close()
    assert took[72] < 1.25 * took[80], took


@pytest.mark.parametrize("quant", [gguf.GGML_Q4_0, gguf.GGML_Q8_0])
@pytest.mark.parametrize("dim,ffn", [(1536, 1536), (1024, 2816)])
def test_four_and_eight_columns_a_warp(tmp_path, quant, dim, ffn):
    """portions on both sides of the rule: CTAs of four columns that fit the SMs, that would share them, that have more warps than those of eight"""
    shape = synth.ModelShape("columns", "llama", dim, ffn, 1, dim // 64, 2, 64, 264, False, 0, 1e4, 1e-5, quant, n_ctx=128)
    d = synth.write_model_dir(str(tmp_path), shape, seed=13)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=80)
    cm.be.set_option("mt_min", OCTETS)
    for n in (5, 12, 32, 48, 65, 72):
        tokens = synth.random_prompt(264, n, seed=n)
        om.reset()
        cm.reset()
        L.assert_bit_equal(cm.forward(tokens), om.forward(tokens), f"{n} tokens")
    assert cm.be.counter("mt_launches") == 0
    om.close()
    cm.close()
