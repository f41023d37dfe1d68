"""Soft-max of a batch's rows in shared memory (pa_k_softmax_rows) and in place (pa_k_mix_softmax): with and without a mix of heads, heads that are no multiple of four or eight, windows, rows
on both sides of the lines between the two. Oracle: portions small enough for the in-place kernel, whose rows' arithmetic is the same, and the plain numpy restatements."""
import numpy as np
import pytest

from powerserve_b200 import arch, arch_synth
from tests import _nufusun_ref, _vanapel_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("family,heads,kv,n,portions", [
    ("nufusun", 6, 2, 640, (100, 640)),      # mixed: many rows, 512 keys and more in shared memory, the first portions in place
    ("nufusun", 18, 2, 600, (90, 300)),
    ("vanapel", 6, 2, 150, (1, 7, 150)),     # no mix: shared memory at every size, a window of 40
    ("vanapel", 10, 2, 600, (33, 600)),
])
def test_rows_in_shared_memory(tmp_path, family, heads, kv, n, portions):
    d = str(tmp_path / "m")
    if family == "vanapel":
        layers = [arch_synth.vanapel_attention_layer(heads, kv, 16, 16, window=40, ff=96, limit=7.0), arch_synth.vanapel_latent_layer(heads, 16, 8, 16, 72, 64, ff=96, limit=7.0)]
        cfg = arch_synth.vanapel_config(128, 330, layers, groups=1)
        t, ref = arch_synth.vanapel_weights(cfg, seed=heads), _vanapel_ref
    else:
        cfg = arch_synth.nufusun_config(128, 330, [arch_synth.nufusun_layer(heads, kv, 16, 16, bias_max=64.0, ff=96)])
        t, ref = arch_synth.nufusun_weights(cfg, seed=heads), _nufusun_ref
    arch_synth.write_model_dir(d, cfg, t)
    toks = [int(v) for v in np.random.default_rng(heads).integers(0, 330, n)]
    want = ref.forward(cfg, t, toks)
    m = arch.load_model(d, dtype="float32", max_batch=n, n_ctx=n + 8)
    for p in portions + (16,):
        m.reset()
        got = np.concatenate([m.forward(toks[lo:lo + p]) for lo in range(0, n, p)])
        err = np.sqrt(((got - want) ** 2).mean(-1)) / np.sqrt((want ** 2).mean(-1))
        assert err.max() < 4e-5, (p, err.max(), int(err.argmax()))   # the bound that float32 mode is held to against these oracles
    m.close()
