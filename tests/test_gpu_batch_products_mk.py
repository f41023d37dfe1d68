"""GPU parity of the batch products of K-quant rows on the tensor cores (ps_k_matmul_mk): one to four column tiles a CTA, rows and columns that do not fill a tile,
rows of one and of many super-blocks, sums at the end of the exact range, scales that are not finite, and the kernel for narrower batches.  Oracle: the plain-C restatement of
the reference; tolerance zero."""
import numpy as np
import pytest

from powerserve_b200 import capi, synth
from tests import _libs as L

pytestmark = pytest.mark.gpu
TYPES = [L.Q4_K, L.Q5_K, L.Q6_K]


@pytest.fixture(scope="module")
def be():
    b = capi.CudaBackend(capi.ModelDesc(256, 4608, 1, 4, 4, 64, 512, 64, 1e-5, 64, 0, 1e4, 1.0, 1.0, 0, 70, 0, 1))
    yield b
    b.close()


def _product(be, t, w, K, N, x, bs):
    ref = np.zeros(N * bs, np.float32)
    L.oracle().ps_or_matmul(t, L.vptr(w), K, N, L.fptr(x), bs, L.fptr(ref))
    wd = be.register_weight(w, t, K, N)
    xd, dd = be.upload(x), be.empty(N * bs)
    out = {}
    for mk_min in (2, 1000):
        be.set_option("mk_min", mk_min)
        launches = be.counter("mk_launches")
        be.matmul(dd, wd, t, K, N, xd, bs)
        assert be.counter("mk_launches") - launches == (mk_min == 2)
        out[mk_min] = dd.numpy()
    be.set_option("mk_min", 2)
    xd.free()
    dd.free()
    be.unregister_weight(w)
    return out, ref


@pytest.mark.parametrize("t", TYPES)
@pytest.mark.parametrize("K,N", [(256, 1), (512, 17), (768, 250), (2304, 33), (4608, 129), (1280, 2500)])
@pytest.mark.parametrize("bs", [2, 7, 8, 9, 16, 17, 33, 70])
def test_products(be, t, K, N, bs):
    rng = np.random.default_rng(K + N + bs)
    w = synth.random_blocks(rng, t, N, K, K ** -0.5).reshape(-1)
    got, ref = _product(be, t, w, K, N, rng.standard_normal(K * bs).astype(np.float32), bs)
    for m in got:
        L.assert_bit_equal(got[m], ref, f"type {t} {K} x {N} on {bs}, mk_min {m}")


@pytest.mark.parametrize("t", TYPES)
def test_largest_sums(be, t):
    """every quant, scale and activation at its extremes: Q6_K's sums reach 32 x 32 x 128 x 127 = 16 646 144, just below 2^24"""
    K, N, bs = 512, 32, 9
    rng = np.random.default_rng(1)
    w = synth.random_blocks(rng, t, N, K, 1.0).reshape(N * K // 256, -1).copy()
    n_q = {L.Q4_K: (4, 144), L.Q5_K: (4, 176), L.Q6_K: (0, 208)}[t]
    for r in range(0, len(w), 4):       # all ones / all zeros, and for Q6_K scales of -128 and 127
        w[r, n_q[0]:n_q[1]] = 0xFF
        w[r + 1, n_q[0]:n_q[1]] = 0
        if t == L.Q6_K:
            w[r, 192:208], w[r + 1, 192:208] = 0x80, 0x80
            w[r + 2, :192], w[r + 2, 192:208] = 0, 0x7F
    x = np.where(rng.random((bs, K)) < 0.5, -1.0, 1.0).astype(np.float32)
    x[:3] = 1.0
    x[3] = -1.0
    got, ref = _product(be, t, np.ascontiguousarray(w.reshape(-1)), K, N, x.reshape(-1), bs)
    for m in got:
        L.assert_bit_equal(got[m], ref, f"type {t}, mk_min {m}")


@pytest.mark.parametrize("t", TYPES)
def test_scales_that_are_not_finite(be, t):
    K, N, bs = 768, 21, 5
    rng = np.random.default_rng(3)
    w = synth.random_blocks(rng, t, N, K, 0.1).reshape(N, K // 256, -1).copy()
    at = 208 if t == L.Q6_K else 0
    w[::2, -1, at:at + 2] = np.frombuffer(np.float16(np.inf).tobytes(), np.uint8)
    w[1, 0, at:at + 2] = np.frombuffer(np.float16(np.nan).tobytes(), np.uint8)
    got, ref = _product(be, t, np.ascontiguousarray(w.reshape(-1)), K, N, rng.standard_normal(K * bs).astype(np.float32), bs)
    for m in got:
        assert np.array_equal(got[m], ref, equal_nan=True), m


@pytest.mark.parametrize("t", TYPES)
def test_a_copy_that_does_not_arrive_is_reported(be, t):
    """a product of the operator table whose copies did not arrive: whoever waits for it or fetches it is told, once, and the next product has all bits"""
    K, N, bs = 512, 40, 6
    rng = np.random.default_rng(t)
    w = synth.random_blocks(rng, t, N, K, K ** -0.5).reshape(-1)
    x = rng.standard_normal(K * bs).astype(np.float32)
    ref = np.zeros(N * bs, np.float32)
    L.oracle().ps_or_matmul(t, L.vptr(w), K, N, L.fptr(x), bs, L.fptr(ref))
    wd, xd, dd = be.register_weight(w, t, K, N), be.upload(x), be.empty(N * bs)
    for ask in (dd.numpy, be.sync):
        be.set_option("give_up_warp", 0)
        be.matmul(dd, wd, t, K, N, xd, bs)
        with pytest.raises(capi.PsCudaError, match="copy of a batch product"):
            ask()
        be.set_option("give_up_warp", -1)
        be.sync()
        be.matmul(dd, wd, t, K, N, xd, bs)
        L.assert_bit_equal(dd.numpy(), ref, f"type {t}, after a failure")
    xd.free()
    dd.free()
    be.unregister_weight(w)
