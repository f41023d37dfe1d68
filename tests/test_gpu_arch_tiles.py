"""GPU parity of the fp32 tile products of layer-list batches (powerserve_b200/csrc/ps_arch_kernels.cuh) where K is cut over a cluster: two to
eight cuts and K in one piece, sums that do not end on a step, matrices whose rows do not fill a tile, batches on both sides of 32- and 64-row tiles, first
halves of feed-forwards with and without a gate at both heights, three norm groups.  Oracles: the plain numpy restatements; tolerances as in the tests of
the models."""
import numpy as np
import pytest

from powerserve_b200 import arch, arch_synth
from tests import _pidenex_ref, _vanapel_ref

pytestmark = pytest.mark.gpu


def model(d, family, width, ff, groups=1):
    if family == "vanapel":
        layers = [arch_synth.vanapel_attention_layer(6, 2, 44, 44, window=40, ff=ff, limit=7.0), arch_synth.vanapel_latent_layer(6, 44, 8, 40, 72, 260, ff=ff, limit=7.0)]
        cfg = arch_synth.vanapel_config(width, 130, layers, groups=groups)
        t, ref = arch_synth.vanapel_weights(cfg, seed=width), _vanapel_ref
    else:                                                            # feed-forwards without a gate
        layers = [arch_synth.pidenex_attention_layer(6, 2, 44, window=40, pool=8, ff=ff), arch_synth.pidenex_attention_layer(6, 2, 44, window=40, ff=ff)]
        cfg = arch_synth.pidenex_config(width, 130, layers)
        t, ref = arch_synth.pidenex_weights(cfg, seed=width), _pidenex_ref
    arch_synth.write_model_dir(d, cfg, t)
    toks = [int(v) for v in np.random.default_rng(1).integers(0, 130, 150)]
    return toks, ref.forward(cfg, t, toks)


# K = width, feed-forward.  The first half of a feed-forward has ceil(ff / 64) tiles a cut and 64 tokens, and takes 64 rows from 148 tiles on:
# 264 x 1048: 17 tiles in two cuts, 32 rows; 1032 x 264: 5 in eight, 32 rows; 1032 x 1288: 21 in eight, 64 rows; 248 x 3208: 51 uncut, 32 rows up to 128
# tokens and 64 rows for 150
@pytest.fixture(scope="module", params=[("vanapel", 264, 1048, 3), ("vanapel", 1032, 264, 1), ("vanapel", 1032, 1288, 1), ("vanapel", 248, 3208, 1), ("pidenex", 1032, 264, 1),
                                        ("pidenex", 1032, 1288, 1), ("pidenex", 248, 3208, 1)])
def pair(request, tmp_path_factory):
    d = str(tmp_path_factory.mktemp("tiles") / "m")
    toks, ref = model(d, *request.param)
    m = arch.load_model(d, dtype="float32", max_batch=150, n_ctx=160)
    yield m, toks, ref
    m.close()


@pytest.mark.parametrize("tc", [0, 1])  # the tiles, and the tensor cores, which take these products where their operand blocks are resident
@pytest.mark.parametrize("cuts", [[150], [64], [65, 31], [33, 2], [32, 128]])
def test_portions(pair, cuts, tc):
    m, toks, ref = pair
    m.be.set_option("arch_tc", tc)
    launches = m.be.counter("arch_split_launches")
    m.reset()
    lo, k, out = 0, 0, []
    while lo < len(toks):
        n = min(cuts[k % len(cuts)], len(toks) - lo)
        out.append(m.forward(toks[lo:lo + n]))
        lo, k = lo + n, k + 1
    got = np.concatenate(out)
    err = np.sqrt(((got - ref) ** 2).mean(-1)) / np.maximum(np.sqrt((ref ** 2).mean(-1)), 1e-6)
    assert err.max() < 4e-5, (cuts, err.max())
    assert (m.be.counter("arch_split_launches") > launches) == bool(tc)


@pytest.mark.parametrize("family,width,ff", [("vanapel", 248, 3208), ("pidenex", 248, 3208), ("vanapel", 1032, 264)])
def test_rounded_operands(tmp_path, family, width, ff):
    """the same tiles on bfloat16 operands (option arch_tc 0), uncut"""
    d = str(tmp_path / "m")
    toks, ref = model(d, family, width, ff)
    m = arch.load_model(d, dtype="bfloat16", max_batch=150, n_ctx=160)
    m.be.set_option("arch_tc", 0)
    for n in (150, 75):
        m.reset()
        got = np.concatenate([m.forward(toks[lo:lo + n]) for lo in range(0, 150, n)])
        err = np.sqrt(((got - ref) ** 2).mean(-1)) / np.maximum(np.sqrt((ref ** 2).mean(-1)), 1e-6)
        assert err.max() < 5e-2 and np.median(err) < 1.5e-2, (n, err.max(), np.median(err))
    m.close()
