"""float32 mode on the tensor cores: products whose activations go in three bfloat16 parts (pa_k_tc_gemm3).  Oracles: the plain numpy restatements, the fp32-FMA tiles
(option arch_tc 0) and their distance from them.  Widths that do not end on a k block of 64 or an output tile of 128, token counts around tiles of 16, 32
and 64, routed rows, activations of every size, and weights that keep a model off this path."""
import numpy as np
import pytest

from powerserve_b200 import arch, arch_synth
from tests import _nufusun_ref, _vanapel_ref

pytestmark = pytest.mark.gpu


def build(d, family, width, ff, touch=lambda t: None):
    if family == "vanapel":
        layers = [arch_synth.vanapel_attention_layer(6, 2, 44, 44, window=40, ff=ff, limit=7.0), arch_synth.vanapel_latent_layer(6, 44, 8, 40, 72, 260, ff=ff, limit=7.0)]
        cfg = arch_synth.vanapel_config(width, 330, layers, groups=1)
        t, ref = arch_synth.vanapel_weights(cfg, seed=width), _vanapel_ref
    else:
        cfg = arch_synth.nufusun_config(width, 330, [arch_synth.nufusun_layer(6, 2, 44, 44, bias_max=64.0, experts=5, top=2, ff=ff, limit=7.0)])
        t, ref = arch_synth.nufusun_weights(cfg, seed=width), _nufusun_ref
    touch(t)
    arch_synth.write_model_dir(d, cfg, t)
    return cfg, t, ref


@pytest.mark.parametrize("family,width,ff", [("vanapel", 264, 200), ("vanapel", 1032, 648), ("nufusun", 264, 200), ("nufusun", 512, 136)])
def test_no_further_from_exact_than_fma(tmp_path, family, width, ff):
    """fp32 sums of K products are within about sqrt(K) 2^-24 of the exact ones on random data; both paths stay below 4e-5 through a model, and the parts' path
    is not the further one (20 % for the luck of single values)"""
    d = str(tmp_path / "m")
    cfg, t, ref = build(d, family, width, ff)
    toks = [int(v) for v in np.random.default_rng(1).integers(0, 330, 150)]
    want = ref.forward(cfg, t, toks)
    m = arch.load_model(d, dtype="float32", max_batch=150, n_ctx=160)

    def run(n):
        m.reset()
        out = [m.forward(toks[lo:lo + n]) for lo in range(0, len(toks), n)]
        return np.concatenate(out)

    err = {}
    assert m.be.counter("arch_tiled") == 1
    for tc in (0, 1):
        m.be.set_option("arch_tc", tc)
        launches = m.be.counter("arch_split_launches")
        got = run(150)
        assert (m.be.counter("arch_split_launches") > launches) == bool(tc)
        e = np.sqrt(((got - want) ** 2).mean(-1)) / np.sqrt((want ** 2).mean(-1))
        assert e.max() < 4e-5
        err[tc] = e.mean()
    assert err[1] < 1.2 * err[0] + 1e-9, err
    for n in (2, 15, 16, 17, 33, 50, 65):        # portions: the same bits whatever tile a token comes in
        part = run(n)
        whole = 150 // n * n if 150 % n == 1 else 150    # (a single token has kernels of its own)
        assert (part[:whole].view(np.uint32) == got[:whole].view(np.uint32)).all(), n
    m.close()


@pytest.mark.parametrize("size", [1e-30, 1e30])
def test_activations_of_every_size(tmp_path, size):
    """an embedding scaled by 2^+-100: the parts keep their places below and above the usual exponents"""
    scale = np.float32(2.0 ** round(np.log2(size)))
    d = str(tmp_path / "m")

    def touch(t):
        t["final.norm"] = np.asarray(t["final.norm"], np.float32) * 0 + scale

    build(d, "vanapel", 264, 200, touch)
    toks = [int(v) for v in np.random.default_rng(1).integers(0, 330, 40)]
    m = arch.load_model(d, dtype="float32", max_batch=64, n_ctx=64)
    got = {}
    for tc in (0, 1):
        m.be.set_option("arch_tc", tc)
        m.reset()
        got[tc] = m.forward(toks).astype(np.float64)
    m.close()
    assert np.isfinite(got[0]).all() and np.sqrt(((got[1] - got[0]) ** 2).sum() / (got[0] ** 2).sum()) < 1e-5


def test_weights_that_are_not_finite(tmp_path):
    """an infinite weight: zero parts would make no number of it, so the model stays on the FMA tiles"""
    def touch(t):
        w = np.array(t["l0.mlp.down"])
        w[3, 5] = np.inf if w.dtype.kind == "f" else 0x7F80
        t["l0.mlp.down"] = w

    d = str(tmp_path / "m")
    build(d, "vanapel", 264, 200, touch)
    toks = [int(v) for v in np.random.default_rng(1).integers(0, 330, 40)]
    m = arch.load_model(d, dtype="float32", max_batch=64, n_ctx=64)
    assert m.be.counter("arch_tiled") == 0      # (and the blocks are given back)
    got = []
    for tc in (0, 1):
        m.be.set_option("arch_tc", tc)
        m.reset()
        got.append(m.forward(toks))
    m.close()
    assert np.array_equal(got[0], got[1], equal_nan=True)


@pytest.mark.parametrize("K", [512, 2048, 8192])
@pytest.mark.parametrize("kind", ["one binade", "ten binades", "ten binades, weights of both signs"])
def test_products_of_one_sign(tmp_path, K, kind):
    """logits of positive activations (the layer's own outputs are zeros).  Tensor-core accumulation truncates, which has a direction: an accumulator's four upper MMAs lose less than
    an ulp of 1/4, 2/4, 3/4 and all of a k block's sum, 2.5 * 2^-23 of it, and on average half of that.  With weights of both signs it averages out, and the FMA tiles are further off"""
    cfg = arch_synth.vanapel_config(K, 330, [arch_synth.vanapel_attention_layer(4, 2, 32, 32, window=40, ff=128, limit=7.0)], groups=1)
    t = arch_synth.vanapel_weights(cfg, seed=1)
    rng = np.random.default_rng(K)
    t["l0.mix.o"], t["l0.mlp.down"] = np.zeros_like(t["l0.mix.o"]), np.zeros_like(t["l0.mlp.down"])
    spread = 1.0 if kind == "one binade" else 2.0 ** (-10 * rng.random((330, K)))
    t["embed"] = _vanapel_ref.bf16_round((1 + rng.random((330, K))) * spread)
    if "both" not in kind:
        t["head"] = _vanapel_ref.bf16_round((np.abs(rng.standard_normal((330, K))) + 0.1) / K)
    d = str(tmp_path / "m")
    arch_synth.write_model_dir(d, cfg, t)
    toks = [int(v) for v in rng.integers(0, 330, 64)]
    want = _vanapel_ref.forward(cfg, t, toks)
    m = arch.load_model(d, dtype="float32", max_batch=64, n_ctx=80)
    rms = {}
    for tc in (0, 1):
        m.be.set_option("arch_tc", tc)
        m.reset()
        off = (m.forward(toks) - want) / np.sqrt((want ** 2).mean(-1, keepdims=True))
        rms[tc] = np.sqrt((off ** 2).mean())
        if tc:
            assert abs(off.mean()) < 2.5 * 2.0 ** -23 / 2 + 2.0 ** -25      # and the norm's own rounding
    m.close()
    assert rms[1] < (rms[0] if "both" in kind else 1.5 * rms[0]), rms
