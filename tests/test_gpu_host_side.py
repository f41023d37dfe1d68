"""The host side of a call: logits arrays whose memory the device writes, and switches between sessions, whose pointer tables go with them.  Oracles: the
same call into memory of the caller's, and the same operations on one cache; tolerance zero."""
import ctypes as C
import gc
import threading

import numpy as np
import pytest

from powerserve_b200 import capi, gguf, synth
from tests import _libs as L

pytestmark = pytest.mark.gpu
SHAPE = synth.ModelShape("host", "llama", 256, 512, 2, 4, 2, 64, 1000, False, 0, 1e4, 1e-5, gguf.GGML_Q4_K, n_ctx=128)


@pytest.fixture()
def model(tmp_path):
    cm = capi.CudaModel(synth.write_model_dir(str(tmp_path), SHAPE, seed=4), max_batch=16)
    yield cm
    cm.close()


def _into_own_memory(cm, tokens):
    out = np.empty((len(tokens), 1000), np.float32)
    t, p = np.asarray(tokens, np.int32), np.arange(cm.position, cm.position + len(tokens), dtype=np.int32)
    i32p = C.POINTER(C.c_int32)
    cm.be._ck(cm.be.L.ps_cuda_forward(cm.be.h, t.ctypes.data_as(i32p), p.ctypes.data_as(i32p), len(tokens), 1, out.ctypes.data))
    return out


def test_logits_arrays_are_the_callers(model):
    """arrays keep their values whatever comes after, views keep the memory, buffers come back, and more arrays than buffers are ordinary ones"""
    toks = synth.random_prompt(1000, 12, seed=1)
    want = []
    for k in range(6):
        model.reset()
        want.append(_into_own_memory(model, toks[k:k + 1 + k]))
    kept = []
    for k in range(6):
        model.reset()
        kept.append(model.forward(toks[k:k + 1 + k])[-1:, :500])
        assert model.be.logits_pool.made <= model.be.logits_pool.MOST
    for k in range(6):
        L.assert_bit_equal(kept[k], want[k][-1:, :500], f"array {k}")
    kept[0][:] = 0      # the caller may write to it
    del kept
    gc.collect()
    assert len(model.be.logits_pool.free) == model.be.logits_pool.made
    model.reset()
    last = model.forward(toks[:2])
    model.close()       # an array outlives its model
    L.assert_bit_equal(last[:1], want[0], "after close")


def test_pool_without_room(model):
    pool = capi._LogitsPool(model.be.L)
    small = [pool.array(1, 10), pool.array(1, 10)]
    assert pool.made == 2 and pool.array(1, 10).base is None          # ordinary memory
    del small
    gc.collect()
    big = pool.array(1, 1000)                                         # takes the place of a smaller buffer
    assert pool.made == 2 and len(pool.free) == 1 and big.base is not None
    assert pool.array(1, (pool.LARGEST >> 2) + 1).base is None
    pool.close()
    del big
    gc.collect()
    assert pool.free == []


def test_slots_after_a_switch(model):
    """copies and moves of cache slots reach the set that is selected, the step kernel and the captured steps too"""
    toks = synth.random_prompt(1000, 40, seed=2)

    def run():
        model.forward(toks[:9], lm_head=False)
        model.forward_tree(toks[9:14], [9, 10, 10, 11, 11], lm_head=False)
        model.be.kv_rollback(5)
        model.be.kv_advance(2)
        model.be.kv_copy_slot(9, 0)
        model.be.kv_copy_slot(10, 2)
        out = [model.forward(toks[14:15])]
        model.be.set_option("persist", 1)
        out.append(model.forward(toks[15:16]))
        model.be.set_option("persist", 0)
        return out + [model.forward(toks[16:17]), model.decode_greedy(toks[17], 3)]

    want = run()
    sids = [model.session_create() for _ in range(2)]
    for sid in sids:
        model.session_select(sid)
        for a, b in zip(run(), want):
            L.assert_bit_equal(np.asarray(a), np.asarray(b), f"session {sid}")
    model.session_select(0)
    model.reset()
    for a, b in zip(run(), want):
        L.assert_bit_equal(np.asarray(a), np.asarray(b), "session 0 again")
    model.session_destroy(sids[0])
    with pytest.raises(capi.PsCudaError, match="unknown session"):
        model.session_select(sids[0])


def test_page_locked_memory_of_any_thread(model):
    """made and freed by threads that have chosen no device; what is no such memory, or no device, is refused"""
    lib, got = model.be.L, []

    def make():
        p = C.c_void_p()
        got.append((lib.ps_cuda_host_alloc_on(0, 4096, C.byref(p)), p.value))

    def free():
        got.append(lib.ps_cuda_host_free(got[0][1]))

    for f in (make, free, free):
        t = threading.Thread(target=f)
        t.start()
        t.join()
    assert got[0][0] == 0 and got[1] == 0 and got[2] != 0
    p = C.c_void_p()
    assert lib.ps_cuda_host_alloc_on(99, 4096, C.byref(p)) != 0 and lib.ps_cuda_host_alloc_on(-1, 4096, C.byref(p)) != 0 and not p.value
    assert len(model.forward(synth.random_prompt(1000, 3, seed=9))) == 3    # (an error of those calls is not the next one's)


@pytest.mark.parametrize("pinned", [[(0, 1)], [(1, 1)], [(0, 1), (2, 1)], [(0, 1), (1, 1), (2, 1)], [(0, 3)]])
def test_arrays_of_which_a_part_is_page_locked(model, pinned):
    """three pages of a caller's: the first, the middle one, the ends, all in three pieces, all in one piece"""
    import torch

    rt, toks = torch.cuda.cudart(), synth.random_prompt(1000, 3, seed=3)
    want = model.forward(toks)
    raw = np.zeros(5 * 4096, np.uint8)
    lo = -raw.ctypes.data % 4096
    out = raw[lo:lo + 12000].view(np.float32)       # 3 x 1000 logits in three pages
    torch.cuda.init()
    done = []
    try:
        for page, n in pinned:
            assert int(rt.cudaHostRegister(out.ctypes.data + 4096 * page, 4096 * n, 0)) == 0
            done.append(out.ctypes.data + 4096 * page)
        model.reset()
        t, p = np.asarray(toks, np.int32), np.arange(3, dtype=np.int32)
        i32p = C.POINTER(C.c_int32)
        model.be._ck(model.be.L.ps_cuda_forward(model.be.h, t.ctypes.data_as(i32p), p.ctypes.data_as(i32p), 3, 1, out.ctypes.data))
        L.assert_bit_equal(out.reshape(3, 1000), want, str(pinned))
    finally:
        for at in done:
            rt.cudaHostUnregister(at)
