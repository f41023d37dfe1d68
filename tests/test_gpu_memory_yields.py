"""Second weight copies that only make batches faster yield to memory that is asked for later: sessions and operator-table buffers of the same model, and other models.  Results: for block
formats the same bits without the copy; float32 layer lists within the bound of both paths.  GPU memory is filled up by plain allocations that nothing touches."""
import ctypes as C

import numpy as np
import pytest

from powerserve_b200 import arch, arch_synth, capi, gguf, synth
from tests import _libs as L

pytestmark = pytest.mark.gpu
MB = 1 << 20


class Filler:
    """takes the device's memory down to less than `left` bytes"""

    def __init__(self, left):
        import torch

        self.torch, self.held = torch, []
        rt = C.CDLL(next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line))
        pool = C.c_void_p()     # (what lies unused in the stream-ordered pool would be given to a plain allocation that finds no room)
        assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0 and torch.cuda.synchronize() is None and rt.cudaMemPoolTrimTo(pool, C.c_size_t(0)) == 0
        size = 64 << 30
        while size >= 2 * MB:
            free = torch.cuda.mem_get_info()[0]
            if free < left:
                break
            try:
                self.held.append(torch.cuda.caching_allocator_alloc(min(size, max(2 * MB, (free - left // 2) // (2 * MB) * 2 * MB))))
            except torch.OutOfMemoryError:
                size //= 2
        self.free = torch.cuda.mem_get_info()[0]

    def close(self):
        for p in self.held:
            self.torch.cuda.caching_allocator_delete(p)
        self.torch.cuda.empty_cache()


@pytest.fixture()
def blocks(tmp_path):
    """records of 33 MB, sessions of 17"""
    shape = synth.ModelShape("yield", "llama", 1024, 4096, 2, 16, 4, 64, 1000, False, 0, 1e4, 1e-5, gguf.GGML_Q8_0, n_ctx=4096)
    cm = capi.CudaModel(synth.write_model_dir(str(tmp_path / "m"), shape, seed=3), max_batch=32)
    yield cm
    cm.close()


def _both(cm, toks):
    got = []
    for mt_min in (1000, 2):
        cm.be.set_option("mt_min", mt_min)
        cm.reset()
        got.append(cm.forward(toks))
    L.assert_bit_equal(got[1], got[0], "with the records and without")
    return got[0]


def test_a_session_takes_the_place_of_the_records(blocks):
    toks = synth.random_prompt(1000, 20, seed=1)
    want = _both(blocks, toks)
    ids = [blocks.session_create()]
    blocks.session_destroy(ids.pop())
    assert blocks.be.counter("mt_ok") == 1
    fill = Filler(12 * MB)
    try:
        ids.append(blocks.session_create())
        assert blocks.be.counter("mt_ok") == 0
        blocks.session_select(ids[0])
        L.assert_bit_equal(blocks.forward(toks), want, "in the new session")
        free = fill.torch.cuda.mem_get_info()[0]
        for _ in range(6):      # no more room: refused, and nothing of an attempt stays
            with pytest.raises(capi.PsCudaError, match="cudaMalloc"):
                for _ in range(4):
                    ids.append(blocks.session_create())
        assert len(ids) <= 3 and fill.torch.cuda.mem_get_info()[0] >= free - 17 * MB * (len(ids) - 1) - 2 * MB
        blocks.session_select(0)
        blocks.reset()
        L.assert_bit_equal(blocks.forward(toks), want, "after a refused one")
    finally:
        fill.close()
    blocks.session_destroy(ids[0])


def test_another_context_takes_their_place(blocks):
    toks = synth.random_prompt(1000, 20, seed=2)
    want = _both(blocks, toks)
    other = capi.CudaBackend(capi.ModelDesc(256, 512, 1, 4, 4, 64, 512, 64, 1e-5, 64, 0, 1e4, 1.0, 1.0, 0, 8, 0, 1))
    w = np.zeros(20 * MB // 4, np.float32)
    fill = Filler(12 * MB)
    try:
        other.register_weight(w, 0, w.size, 1)
        assert blocks.be.counter("mt_ok") == 0
        blocks.reset()
        L.assert_bit_equal(blocks.forward(toks), want, "afterwards")
    finally:
        fill.close()
    other.close()


def test_a_second_bind_keeps_one_copy(blocks):
    toks = synth.random_prompt(1000, 20, seed=1)
    want = _both(blocks, toks)
    blocks.be._ck(blocks.be.L.ps_cuda_bind_model(blocks.be.h, C.byref(blocks._w)))
    assert blocks.be.counter("mt_ok") == 1
    L.assert_bit_equal(_both(blocks, toks), want, "bound again")


def test_buffers_of_the_operator_table_take_their_place(blocks):
    fill = Filler(12 * MB)
    try:
        buf = blocks.be.empty(20 * MB // 4)
        assert blocks.be.counter("mt_ok") == 0
        buf.free()
    finally:
        fill.close()


@pytest.mark.parametrize("whose", ["own", "other"])
def test_float32_layer_lists(tmp_path, whose):
    """operand blocks of 110 MB, sessions of 34"""
    cfg = arch_synth.vanapel_config(2048, 2000, [arch_synth.vanapel_attention_layer(8, 4, 64, 64, window=16384, ff=8192, limit=7.0)], groups=1)
    d = str(tmp_path / "m")
    arch_synth.write_model_dir(d, cfg, arch_synth.vanapel_weights(cfg, seed=1))
    m = arch.load_model(d, dtype="float32", max_batch=32, n_ctx=16384)
    other = capi.CudaBackend(capi.ModelDesc(256, 512, 1, 4, 4, 64, 512, 64, 1e-5, 64, 0, 1e4, 1.0, 1.0, 0, 8, 0, 1))
    w = np.zeros(16 * MB // 4, np.float32)
    toks = synth.random_prompt(2000, 20, seed=1)
    got = {}
    for tc in (0, 1):
        m.be.set_option("arch_tc", tc)
        m.reset()
        got[tc] = m.forward(toks)
    assert m.be.counter("arch_tiled") == 1
    fill = Filler(24 * MB if whose == "own" else 8 * MB)
    try:
        if whose == "own":
            sid = m.session_create()
            m.session_select(sid)
        else:
            other.register_weight(w, 0, w.size, 1)
            m.reset()
        assert m.be.counter("arch_tiled") == 0
        L.assert_bit_equal(m.forward(toks), got[0], "the FMA tiles")
    finally:
        fill.close()
    other.close()
    m.close()
