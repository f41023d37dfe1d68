"""GPU parity of the batch P.V kernel that copies cache rows by 16-byte lines (rows of a length that four divides, and one that it does not) and of the
session kernels that take eight positions or dims a warp, at chunk edges and head sizes of one to eight chunks.  Oracle: the plain-C restatement of the
reference; tolerance zero."""
import time

import pytest

from powerserve_b200 import capi, gguf, synth
from tests import _libs as L
from tests import _model as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads,kv_heads,head_size,n_ctx", [(2, 1, 32, 254), (3, 1, 96, 250), (2, 2, 256, 256)])
def test_portions_and_sessions(tmp_path, heads, kv_heads, head_size, n_ctx):
    shape = synth.ModelShape("rows", "llama", heads * head_size, 128, 1, heads, kv_heads, head_size, 264, False, 0, 1e4, 1e-5, gguf.GGML_Q8_0, n_ctx=n_ctx)
    d = synth.write_model_dir(str(tmp_path), shape, seed=7)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=70)
    tokens = synth.random_prompt(264, 240, seed=1)
    for n in (31, 33, 70, 62, 9):                                    # chunks of 32 positions: fewer, exactly and more than the copies in flight, and rests
        L.assert_bit_equal(cm.forward(tokens[:n]), om.forward(tokens[:n]), f"{n} tokens")
        tokens = tokens[n:]
    prompts = [synth.random_prompt(264, n, seed=n) for n in (2, 8, 9, 32, 65)]
    sids = [0] + [cm.session_create() for _ in prompts[1:]]
    for sid, p in zip(sids, prompts):
        cm.session_select(sid)
        cm.reset()
        cm.prefill(p, 16)
    lg, _ = cm.forward_sessions(sids, [int(p[-1]) for p in prompts])
    for col, p in enumerate(prompts):
        om.reset()
        L.assert_bit_equal(lg[col], om.forward(p)[-1], f"session of {len(p)}")
    om.close()
    cm.close()


@pytest.mark.parametrize("heads,kv_heads", [(4, 4), (4, 2), (8, 2), (6, 2)])
def test_session_rows_of_every_group_size(tmp_path, heads, kv_heads):
    """one, two, three and four query heads a kv head; fewer, exactly and more than the four chunks of positions whose loads fly together"""
    shape = synth.ModelShape("groups", "llama", heads * 64, 128, 1, heads, kv_heads, 64, 264, False, 0, 1e4, 1e-5, gguf.GGML_Q8_0, n_ctx=320)
    d = synth.write_model_dir(str(tmp_path), shape, seed=9)
    om, cm = M.OracleModel(d), capi.CudaModel(d, max_batch=64)
    prompts = [synth.random_prompt(264, n, seed=n) for n in (31, 32, 127, 128, 129, 160, 257, 300)]
    sids = [0] + [cm.session_create() for _ in prompts[1:]]
    for sid, p in zip(sids, prompts):
        cm.session_select(sid)
        cm.reset()
        cm.prefill(p, 16)
    lg, _ = cm.forward_sessions(sids, [int(p[-1]) for p in prompts])
    for col, p in enumerate(prompts):
        om.reset()
        L.assert_bit_equal(lg[col], om.forward(p)[-1], f"session of {len(p)}")
    om.close()
    cm.close()


def test_sessions_with_a_head_per_kv_head_keep_their_loads_in_flight(tmp_path):
    """Four sessions at 1000 positions, 16 kv heads with a query head each, two layers, against the same at 8 positions: measured 177 us more when each
    load waits for the one before, and about 50 when they overlap; the bound lies between."""
    shape = synth.ModelShape("mha", "llama", 1024, 1024, 2, 16, 16, 64, 264, False, 0, 1e4, 1e-5, gguf.GGML_Q8_0, n_ctx=1280)
    cm = capi.CudaModel(synth.write_model_dir(str(tmp_path), shape, seed=10), max_batch=128)
    sids = [0] + [cm.session_create() for _ in range(3)]
    took = {}
    for n in (8, 1000):
        for sid in sids:
            cm.session_select(sid)
            cm.reset()
            cm.prefill(synth.random_prompt(264, n + 1, seed=sid), 128)
        best = 1e9
        for _ in range(40):
            t0 = time.perf_counter()
            cm.forward_sessions(sids, [1] * 4, want_logits=False)
            best = min(best, time.perf_counter() - t0)
        took[n] = best * 1e6
    cm.close()
    assert took[1000] - took[8] < 120, took
