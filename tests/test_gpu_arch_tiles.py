"""GPU parity of the fp32 tile products of layer-list batches (powerserve_b200/csrc/ps_arch_kernels.cuh) where K is cut over a cluster: two to
eight cuts, sums that do not end on a step, matrices whose rows do not fill a tile, batches on both sides of 32- and 64-row tiles, three norm
groups.  Oracle: the plain numpy restatement; float32 tolerance as in the tests of the models.."""
import numpy as np
import pytest

from powerserve_b200 import arch, arch_synth
from tests import _vanapel_ref as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[(264, 1048, 3), (1032, 264, 1)])   # K = width, feed-forward: 2 to 8 cuts with a rest
def pair(request, tmp_path_factory):
    width, ff, groups = request.param
    layers = [arch_synth.vanapel_attention_layer(6, 2, 44, 44, window=40, ff=ff, limit=7.0), arch_synth.vanapel_latent_layer(6, 44, 8, 40, 72, 260, ff=ff, limit=7.0)]
    cfg = arch_synth.vanapel_config(width, 130, layers, groups=groups)
    t = arch_synth.vanapel_weights(cfg, seed=width)
    d = str(tmp_path_factory.mktemp("tiles") / "m")
    arch_synth.write_model_dir(d, cfg, t)
    toks = [int(v) for v in np.random.default_rng(1).integers(0, 130, 150)]
    ref = R.forward(cfg, t, toks)
    m = arch.load_model(d, dtype="float32", max_batch=150, n_ctx=160)
    yield m, toks, ref
    m.close()


@pytest.mark.parametrize("cuts", [[150], [64], [65, 31], [33, 2], [32, 128]])
def test_portions(pair, cuts):
    m, toks, ref = pair
    m.reset()
    lo, k, out = 0, 0, []
    while lo < len(toks):
        n = min(cuts[k % len(cuts)], len(toks) - lo)
        out.append(m.forward(toks[lo:lo + n]))
        lo, k = lo + n, k + 1
    got = np.concatenate(out)
    err = np.sqrt(((got - ref) ** 2).mean(-1)) / np.maximum(np.sqrt((ref ** 2).mean(-1)), 1e-6)
    assert err.max() < 4e-5, (cuts, err.max())
