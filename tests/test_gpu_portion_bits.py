"""GPU: a token's logits have the same bits however its prompt is cut into portions (of two tokens or more: a single token has kernels of its own).
The tile products add over k, the attention over the keys, in an order that neither the portion's size nor its place decides: windows that
begin anywhere in a tile of keys, portions on both sides of 32- and 64-row tiles, K in one piece and cut over a cluster.  Tolerance zero."""
import numpy as np
import pytest

from powerserve_b200 import arch, arch_synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tc", [0, 1])  # products on tiles of fp32 FMAs, and on the tensor cores
@pytest.mark.parametrize("dtype,width,ff", [("bfloat16", 264, 200), ("float32", 264, 200), ("float32", 1032, 648)])
def test_portions(tmp_path, dtype, width, ff, tc):
    layers = [arch_synth.vanapel_attention_layer(6, 2, 44, 44, window=40, ff=ff, limit=7.0), arch_synth.vanapel_latent_layer(6, 44, 8, 40, 72, 260, ff=ff, limit=7.0)]
    cfg = arch_synth.vanapel_config(width, 130, layers, groups=1)
    d = str(tmp_path / "m")
    arch_synth.write_model_dir(d, cfg, arch_synth.vanapel_weights(cfg, seed=width))
    toks = [int(v) for v in np.random.default_rng(1).integers(0, 130, 150)]
    m = arch.load_model(d, dtype=dtype, max_batch=150, n_ctx=160)
    m.be.set_option("arch_tc", tc)
    want = m.forward(toks)
    assert (m.be.counter("arch_split_launches") > 0) == (tc == 1 and dtype == "float32")
    for cuts in ([64], [65, 31], [33, 2], [100, 7]):
        m.reset()
        lo, k, out = 0, 0, []
        while lo < len(toks):
            n = min(cuts[k % len(cuts)], len(toks) - lo)
            if len(toks) - lo - n == 1:
                n += 1
            out.append(m.forward(toks[lo:lo + n]))
            lo, k = lo + n, k + 1
        got = np.concatenate(out)
        same = (got.view(np.uint32) == want.view(np.uint32)).all(-1)
        assert same.all(), (cuts, np.flatnonzero(~same)[:8], np.abs(got - want).max())
    m.close()
