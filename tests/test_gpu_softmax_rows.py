"""Soft-max of a batch's rows in shared memory (pa_k_softmax_rows) and in place (pa_k_mix_softmax): with and without a mix of heads, heads that are no multiple of four or eight, windows, chunks,
pooled blocks, rows on both sides of the lines between the two. Oracles: the kernel in place (option arch_smx_rows 0), whose rows are added up in the same order, bit for bit, and the plain numpy restatements."""
import numpy as np
import pytest

from powerserve_b200 import arch, arch_synth
from tests import _dozotar_ref, _nufusun_ref, _pidenex_ref, _vanapel_ref

pytestmark = pytest.mark.gpu


def _model(family, heads, kv):
    if family == "vanapel":
        layers = [arch_synth.vanapel_attention_layer(heads, kv, 16, 16, window=40, ff=96, limit=7.0), arch_synth.vanapel_latent_layer(heads, 16, 8, 16, 72, 64, ff=96, limit=7.0)]
        cfg = arch_synth.vanapel_config(128, 330, layers, groups=1)
        return cfg, arch_synth.vanapel_weights(cfg, seed=heads), _vanapel_ref
    if family == "pidenex":     # a window, and means of the blocks before it
        layers = [arch_synth.pidenex_attention_layer(heads, kv, 16, window=40, pool=8, ff=96), arch_synth.pidenex_attention_layer(heads, kv, 16, window=24, pool=5, ff=96)]
        cfg = arch_synth.pidenex_config(128, 330, layers)
        return cfg, arch_synth.pidenex_weights(cfg, seed=heads), _pidenex_ref
    if family == "dozotar":     # chunks
        cfg = arch_synth.dozotar_config(128, 330, [arch_synth.dozotar_attention_layer(heads, kv, 16, 16, chunk=48, ff=96)])
        return cfg, arch_synth.dozotar_weights(cfg, seed=heads), _dozotar_ref
    cfg = arch_synth.nufusun_config(128, 330, [arch_synth.nufusun_layer(heads, kv, 16, 16, bias_max=64.0, ff=96)])
    return cfg, arch_synth.nufusun_weights(cfg, seed=heads), _nufusun_ref


@pytest.mark.parametrize("family,heads,kv,n,portions", [
    ("nufusun", 6, 2, 640, (100, 640)),      # mixed: many rows, 512 keys and more in shared memory, the first portions in place
    ("nufusun", 18, 2, 600, (90, 300)),
    ("vanapel", 6, 2, 150, (1, 7, 150)),     # no mix: shared memory at every size, a window of 40
    ("vanapel", 10, 2, 600, (33, 600)),
    ("pidenex", 6, 2, 150, (7, 33, 150)),
    ("dozotar", 6, 2, 150, (7, 33, 150)),
])
def test_rows_in_shared_memory(tmp_path, family, heads, kv, n, portions):
    d = str(tmp_path / "m")
    cfg, t, ref = _model(family, heads, kv)
    arch_synth.write_model_dir(d, cfg, t)
    toks = [int(v) for v in np.random.default_rng(heads).integers(0, 330, n)]
    want = ref.forward(cfg, t, toks)
    m = arch.load_model(d, dtype="float32", max_batch=n, n_ctx=n + 8)
    for p in portions + (16,):
        got = {}
        for rows in (0, 1):
            m.be.set_option("arch_smx_rows", rows)
            m.reset()
            got[rows] = np.concatenate([m.forward(toks[lo:lo + p]) for lo in range(0, n, p)])
        assert (got[1].view(np.uint32) == got[0].view(np.uint32)).all(), (p, np.abs(got[1] - got[0]).max())
        err = np.sqrt(((got[1] - want) ** 2).mean(-1)) / np.sqrt((want ** 2).mean(-1))
        assert err.max() < 4e-5, (p, err.max(), int(err.argmax()))   # the bound that float32 mode is held to against these oracles
    m.close()
