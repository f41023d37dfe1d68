"""Page-locked buffers behind the logits arrays (capi._LogitsPool, capi._PinnedStore), over a library that counts: buffers go from model to model, a batch that grows makes
few of them, and what lies unused is bounded and can be given back."""
import ctypes as C
import gc
import threading

import numpy as np

from powerserve_b200 import capi


class FakeLib:
    """page-locked memory of ordinary memory"""

    def __init__(self):
        self.live, self.made, self.fail, self.devices = {}, 0, False, []

    def ps_cuda_host_alloc_on(self, device, n, out):
        self.devices.append(device)
        if self.fail:
            return 2
        b = C.create_string_buffer(n)
        out._obj.value = C.addressof(b)
        self.live[C.addressof(b)] = b
        self.made += 1
        return 0

    def ps_cuda_host_free(self, p):
        del self.live[p]    # (a second time: KeyError)
        return 0


def pinned(a):
    return a.base is not None


def test_the_next_model_takes_over_what_a_closed_one_had():
    L, store = FakeLib(), capi._PinnedStore()
    first = capi._LogitsPool(L, store)
    a, b = first.array(12, 32768), first.array(12, 32768)
    assert pinned(a) and pinned(b) and L.made == 2
    a[:], b[:] = 1, 2
    first.close()
    assert (a == 1).all() and (b == 2).all()    # arrays outlive the model
    del a
    gc.collect()
    second = capi._LogitsPool(L, store)
    c = second.array(10, 32768)
    assert pinned(c) and L.made == 2 and (b == 2).all()
    del b, c
    gc.collect()
    second.close()
    assert len(L.live) == len(store.idle) == 2
    store.clear(L)
    assert not L.live and store.idle == []


def test_a_growing_batch_makes_a_buffer_a_size():
    L, store = FakeLib(), capi._PinnedStore()
    pool = capi._LogitsPool(L, store)
    for n in range(1, 65):
        pool.array(n, 32768)[:] = n
    assert L.made <= 7
    held, made = pool.array(1, 32768), L.made
    for n in list(range(1, 65)) * 2:        # the result before is held
        held = pool.array(n, 32768)
        held[:] = n
    assert pinned(held) and L.made <= made + 7
    del held
    gc.collect()
    pool.close()
    assert len(store.idle) <= store.MOST and len(L.live) == len(store.idle)


def test_bounds():
    L, store = FakeLib(), capi._PinnedStore()
    pools = [capi._LogitsPool(L, store) for _ in range(9)]
    arrays = [[p.array(1, 1 << 21) for _ in range(3)] for p in pools]   # 8 MB each
    assert all([pinned(a) for a in got] == [True, True, False] for got in arrays)
    assert not pinned(pools[0].array(1, (pools[0].LARGEST >> 2) + 1))
    del arrays
    gc.collect()
    for p in pools:
        p.close()
    assert 0 < len(store.idle) <= store.MOST and sum(b[1] for b in store.idle) <= store.BYTES and len(L.live) == len(store.idle)


def test_no_page_locked_memory():
    L, store = FakeLib(), capi._PinnedStore()
    pool = capi._LogitsPool(L, store)
    L.fail = True
    assert not pinned(pool.array(2, 100)) and pool.made == 0
    L.fail = False
    assert pinned(pool.array(2, 100))
    gc.collect()
    pool.close()
    pool.close()
    assert len(L.live) == len(store.idle) == 1


def test_threads():
    """models that come and go in several threads, with arrays that are freed by any of them"""
    L, store, bad = FakeLib(), capi._PinnedStore(), []
    handed = []

    def work(k):
        rng = np.random.default_rng(k)
        for _ in range(60):
            pool = capi._LogitsPool(L, store)
            for _ in range(10):
                a = pool.array(int(rng.integers(1, 40)), 4096)
                a[:] = k
                handed.append((a, k))
                while len(handed) > 12:
                    try:
                        x, owner = handed.pop(int(rng.integers(0, 4)))
                    except IndexError:
                        break
                    if not (x == owner).all():
                        bad.append(owner)
                    del x
            pool.close()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad
    handed.clear()
    gc.collect()
    assert len(L.live) == len(store.idle) <= store.MOST


def test_buffers_are_made_on_the_models_device():
    """whatever device the calling thread has chosen, or none"""
    L, store = FakeLib(), capi._PinnedStore()
    got = []
    t = threading.Thread(target=lambda: got.append(capi._LogitsPool(L, store, device=3).array(4, 100)))
    t.start()
    t.join()
    assert pinned(got[0]) and L.devices == [3]


def test_what_has_lain_longest_makes_room():
    """models of one size come after models of another: their buffers stay, whatever lies there"""
    L, store = FakeLib(), capi._PinnedStore()
    for rows in (1, 1, 1, 16):
        pools = [capi._LogitsPool(L, store) for _ in range(3)]
        arrays = [p.array(rows, 32768) for p in pools]
        made = L.made
        del arrays
        gc.collect()
        for p in pools:
            p.close()
    assert made == 6 and sorted(b[1] for b in store.idle) == [128 << 10] + 3 * [4 << 20] and len(L.live) == 4
    pools = [capi._LogitsPool(L, store) for _ in range(3)]
    assert all(pinned(p.array(16, 32768)) for p in pools) and L.made == made
