"""Device top-k (ps_cuda_sample_topk) on planted logits rows: ties, zeros of both signs, infinities, NaNs, vocabularies of less than a
slice, of many slices and of more candidates than one merge round holds.  Oracle: numpy; values and ids equal."""
import numpy as np
import pytest

from powerserve_b200 import capi, gguf, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("vocab", [256, 2048, 2056, 40000, 140000])
def test_planted_rows(vocab):
    shape = synth.ModelShape("topk", "llama", 256, 256, 1, 4, 4, 64, vocab, True, 0, 1e4, 1e-5, gguf.GGML_Q8_0, n_ctx=32)
    tensors = {n: gguf.GGUFTensor(n, t, tuple(s), np.ascontiguousarray(d).view(np.uint8).reshape(-1)) for n, t, s, d in synth.generate_tensors(shape, 1)}
    m = capi.CudaModel(desc=capi.desc_from_model_json(synth.model_json(shape), max_batch=2, n_ctx=32), tensors=tensors)
    rng = np.random.default_rng(vocab)
    rows = {"normal": rng.standard_normal(vocab), "ties": rng.integers(-3, 4, vocab) * 0.5, "zeros": np.where(rng.random(vocab) < 0.5, 0.0, -0.0),
            "ascending": np.arange(vocab), "descending": -np.arange(vocab), "few": np.where(np.arange(vocab) % 97 == 5, rng.standard_normal(vocab), -np.inf)}
    nan = rng.standard_normal(vocab)
    nan[rng.random(vocab) < 0.3] = np.nan
    nan[7] = np.inf
    rows["nan"] = nan
    m.forward_lazy([1])
    for name, row in rows.items():
        row = np.ascontiguousarray(row, np.float32)
        m.be._ck(m.be.L.ps_cuda_memcpy_h2d(m.be.h, m.be.logits_dev(), row.ctypes.data, row.nbytes))
        live = np.flatnonzero(~np.isnan(row))
        order = live[np.lexsort((live, -row[live]))]
        for k in (1, 5, 40, 64):
            vals, ids = m.sample_topk(k)
            assert list(ids) == list(order[:k]), (name, k)
            assert np.array_equal(vals, row[order[:k]]), (name, k)
    row = np.full(vocab, np.nan, np.float32)      # fewer candidates than asked for
    row[9] = 2.0
    m.be._ck(m.be.L.ps_cuda_memcpy_h2d(m.be.h, m.be.logits_dev(), row.ctypes.data, row.nbytes))
    vals, ids = m.sample_topk(3)
    assert list(ids) == [9, -1, -1] and vals[0] == 2.0 and np.all(np.isneginf(vals[1:]))
    m.close()


def test_every_k():
    """all k that a call takes, one after the other on one row: each is the front of the same order"""
    shape = synth.ModelShape("topk", "llama", 256, 256, 1, 4, 4, 64, 5000, True, 0, 1e4, 1e-5, gguf.GGML_Q8_0, n_ctx=32)
    tensors = {n: gguf.GGUFTensor(n, t, tuple(s), np.ascontiguousarray(d).view(np.uint8).reshape(-1)) for n, t, s, d in synth.generate_tensors(shape, 1)}
    m = capi.CudaModel(desc=capi.desc_from_model_json(synth.model_json(shape), max_batch=2, n_ctx=32), tensors=tensors)
    m.forward_lazy([1])
    row = (np.random.default_rng(2).integers(-40, 40, 5000) * 0.25).astype(np.float32)
    m.be._ck(m.be.L.ps_cuda_memcpy_h2d(m.be.h, m.be.logits_dev(), row.ctypes.data, row.nbytes))
    order = np.lexsort((np.arange(5000), -row))
    for k in list(range(1, 65)) + [3, 1]:
        vals, ids = m.sample_topk(k)
        assert list(ids) == list(order[:k]) and np.array_equal(vals, row[order[:k]]), k
    m.close()
