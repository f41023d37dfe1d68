"""Performance cases: what a user of this framework has it do, through the entry points a program calls, over the range of sizes
its models and callers bring.

Two model families, both through the model objects of `powerserve_b200`:

* GGUF / llama stacks (`capi.CudaModel`): one decoded token, a prompt portion, one token for many sessions, a draft tree's
  verification.  Layer shapes are those of Qwen2-0.5B (Q4_0, biases, NEOX rotation), Llama-3.2-1B and Llama-3.1-8B (Q4_K) with few
  layers, so that a model is made in a second; results of this family are defined bit by bit.
* layer-list models (`arch.LayerListModel`, bfloat16 weights): a prompt portion or one token of a Nufusun model (attention with mixed
  heads, routed experts) or a Vanapel model (windowed and latent attention, dense feed-forward), in both compute modes.

and the operator table's matrix product (`capi.CudaBackend.matmul`), for every block format a GGUF file holds.
"""
import math
import os
import shutil
import tempfile
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from powerserve_b200 import arch, arch_synth, capi, gguf, synth

QUANTS = {"q4_0": gguf.GGML_Q4_0, "q8_0": gguf.GGML_Q8_0, "q4_k": gguf.GGML_Q4_K, "q5_k": gguf.GGML_Q5_K, "q6_k": gguf.GGML_Q6_K}

# layer shapes: architecture, width, feed-forward rows, heads, kv heads, head size, tied head, rotation kind, rotation base, norm eps, biases
SHAPES = {
    "qwen2-0.5b": ("qwen2", 896, 4864, 14, 2, 64, True, 2, 1e6, 1e-6, True),
    "llama-3.2-1b": ("llama", 2048, 8192, 32, 8, 64, True, 0, 5e5, 1e-5, False),
    "llama-3.1-8b": ("llama", 4096, 14336, 32, 8, 128, False, 0, 5e5, 1e-5, False),
}


def listed():
    return [
        # the smallest call: one token of a small chat model after a short prompt, logits to the host for its own sampler
        {"name": "decode_qwen2_05b", "kind": "decode", "shape": "qwen2-0.5b", "quant": "q4_0", "out": "", "layers": 6, "vocab": 151936, "ctx": 48, "pick": "host"},
        # one token of a 1B model in a chat; the 40 best logits come back, the sampler draws from those
        {"name": "decode_llama_1b", "kind": "decode", "shape": "llama-3.2-1b", "quant": "q4_k", "out": "", "layers": 4, "vocab": 128256, "ctx": 300, "pick": "topk"},
        # one token of an 8B model deep in a document, logits to the host
        {"name": "decode_llama_8b", "kind": "decode", "shape": "llama-3.1-8b", "quant": "q4_k", "out": "", "layers": 2, "vocab": 128256, "ctx": 2048, "pick": "host"},
        # a short question as one portion
        {"name": "prefill_qwen2_05b", "kind": "prefill", "shape": "qwen2-0.5b", "quant": "q4_0", "out": "", "layers": 6, "vocab": 16384, "ctx": 0, "batch": 32, "head": False},
        # a ragged portion whose logits are all wanted (scoring a text)
        {"name": "score_llama_1b", "kind": "prefill", "shape": "llama-3.2-1b", "quant": "q4_k", "out": "", "layers": 4, "vocab": 16384, "ctx": 128, "batch": 77, "head": True},
        # a full portion of a long prompt
        {"name": "prefill_llama_8b", "kind": "prefill", "shape": "llama-3.1-8b", "quant": "q4_k", "out": "", "layers": 2, "vocab": 8192, "ctx": 1920, "batch": 128, "head": False},
        # a server's step: one token for each of 64 conversations, four steps
        {"name": "sessions_llama_8b", "kind": "sessions", "shape": "llama-3.1-8b", "quant": "q4_k", "out": "", "layers": 2, "vocab": 32768, "ctx": 200, "batch": 64, "steps": 4},
        # speculative decoding: the target checks a drafted tree of 12 tokens
        {"name": "verify_llama_8b", "kind": "verify", "shape": "llama-3.1-8b", "quant": "q4_k", "out": "", "layers": 2, "vocab": 32768, "ctx": 1000, "batch": 12},
        # a matrix of a Q4_K_M file (its Q6_K ones) by way of the operator table
        {"name": "matmul_q6_k", "kind": "matmul", "quant": "q6_k", "k": 4096, "n": 4096, "batch": 32},
        # a portion and a token of a layer-list model with routed experts
        {"name": "prefill_nufusun", "kind": "layers", "arch": "nufusun", "dtype": "bfloat16", "width": 2048, "heads": 16, "kv_heads": 4, "head_size": 128, "ff": 2816,
         "layers": 1, "vocab": 4096, "ctx": 768, "batch": 256},
        {"name": "decode_nufusun", "kind": "layers", "arch": "nufusun", "dtype": "bfloat16", "width": 2048, "heads": 16, "kv_heads": 4, "head_size": 128, "ff": 2816,
         "layers": 1, "vocab": 32000, "ctx": 1024, "batch": 1},
        # a ragged portion through windowed and latent attention, without rounding
        {"name": "prefill_vanapel_f32", "kind": "layers", "arch": "vanapel", "dtype": "float32", "width": 1024, "heads": 16, "kv_heads": 4, "head_size": 64, "ff": 2048,
         "layers": 2, "vocab": 4096, "ctx": 300, "batch": 150},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "prefill", "prefill", "prefill", "sessions", "verify", "matmul", "layers", "layers"])
    if kind == "matmul":
        quant = rng.choice(sorted(QUANTS))
        unit = 256 if quant.endswith("_k") else 32
        return {"kind": kind, "quant": quant, "k": unit * _log(rng, 512 // unit, 8192 // unit), "n": _log(rng, 256, 8192), "batch": _log(rng, 1, 128)}
    if kind == "layers":
        name = rng.choice(["nufusun", "vanapel"])
        width, heads, kv, hs, ff = rng.choice([(1024, 16, 4, 64, 1024), (1024, 8, 2, 128, 2048), (1536, 12, 4, 128, 2048), (2048, 16, 4, 128, 2816)])
        batch = 1 if rng.random() < 0.4 else _log(rng, 2, 256)
        f32 = rng.random() < 0.3
        return {"kind": kind, "arch": name, "dtype": "float32" if f32 else "bfloat16", "width": width, "heads": heads, "kv_heads": kv, "head_size": hs, "ff": ff,
                "layers": 2 if name == "vanapel" else 1, "vocab": rng.choice([2048, 4096, 8000]), "ctx": _log(rng, 2, 1024), "batch": min(batch, 128) if f32 else batch}
    shape = rng.choice(sorted(SHAPES))
    quant = rng.choice(["q4_0", "q4_0", "q8_0"]) if shape == "qwen2-0.5b" else "q4_k"
    out = "q6_k" if quant == "q4_k" and kind in ("decode", "prefill") and rng.random() < 0.15 else ""   # a Q4_K_M file's head
    case = {"kind": kind, "shape": shape, "quant": quant, "out": out, "layers": rng.choice([1, 2, 3]) if shape != "llama-3.1-8b" else rng.choice([1, 2]),
            "vocab": rng.choice([4096, 16384, 32768]), "ctx": _log(rng, 1, 2048)}
    if kind == "decode":
        case["pick"] = rng.choice(["host", "topk"])
    elif kind == "prefill":
        case["ctx"] = rng.choice([0, _log(rng, 1, 1920)])
        case["batch"] = _log(rng, 2, 128)
        case["head"] = rng.random() < 0.4
        if out:     # a mixed file takes the operator table: keep it within the largest listed case
            case["batch"], case["layers"] = min(case["batch"], 24), 1
    elif kind == "sessions":
        case["ctx"] = _log(rng, 8, 300)
        case["batch"] = _log(rng, 2, 64)
        case["steps"] = rng.choice([1, 2, 3])
    else:
        case["ctx"] = _log(rng, 8, 1900)
        case["batch"] = _log(rng, 2, 32)
    return case


# ---------------------------------------------------------------------------------------------------------------- what a case is made of
def _shape(case, n_ctx):
    a, dim, ffn, nh, nkv, hs, tied, rope, base, eps, bias = SHAPES[case["shape"]]
    return synth.ModelShape(case["shape"], a, dim, ffn, case["layers"], nh, nkv, hs, case["vocab"], tied and not case["out"], rope, base, eps, QUANTS[case["quant"]],
                            n_ctx=n_ctx, qkv_bias=bias, output_type=QUANTS[case["out"]] if case["out"] else None)


def _n_ctx(case):
    return -(-(case["ctx"] + case.get("batch", 1) * (1 if case["kind"] != "sessions" else 0) + case.get("steps", 1) + 8) // 256) * 256


def _tensors(case, seed):
    return {n: gguf.GGUFTensor(n, t, tuple(s), np.ascontiguousarray(d).view(np.uint8).reshape(-1)) for n, t, s, d in synth.generate_tensors(_shape(case, _n_ctx(case)), seed)}


def _rng(seed, what):
    return np.random.Generator(np.random.SFC64([int(seed) & 0x7FFFFFFF, what]))


def _tokens(case, seed):
    """tokens of the call's past and of the call: (past [ctx], now [batch]) or per session (past [batch][len], now [batch][steps])"""
    r, v = _rng(seed, 1000), case["vocab"]
    if case["kind"] == "sessions":
        past = [r.integers(0, v, max(1, case["ctx"] - int(r.integers(0, case["ctx"] // 2 + 1))), dtype=np.int32) for _ in range(case["batch"])]
        return past, r.integers(0, v, (case["batch"], case["steps"]), dtype=np.int32)
    return r.integers(0, v, case["ctx"], dtype=np.int32), r.integers(0, v, case.get("batch", 1), dtype=np.int32)


def _tree(case, seed):
    """parents of a drafted tree's nodes (node 0 is the root), their depths and the mask [n][n] of the nodes each one sees"""
    r, n = _rng(seed, 2000), case["batch"]
    parent = [-1] + [int(r.integers(max(0, i - 4), i)) for i in range(1, n)]
    mask, depth = np.zeros((n, n), np.uint8), [0] * n
    for i in range(n):
        if i:
            depth[i] = depth[parent[i]] + 1
            mask[i] = mask[parent[i]]
        mask[i, i] = 1
    return depth, mask


def _layer_config(case):
    W, H, G, hs, ff, n = (case[k] for k in ("width", "heads", "kv_heads", "head_size", "ff", "layers"))
    if case["arch"] == "nufusun":
        return arch_synth.nufusun_config(W, case["vocab"], [arch_synth.nufusun_layer(H, G, hs, hs, bias_max=1024.0, experts=8, top=2, ff=ff, limit=7.0) for _ in range(n)])
    kinds = [arch_synth.vanapel_attention_layer(H, G, hs, hs, window=512, ff=ff, limit=7.0), arch_synth.vanapel_latent_layer(H, hs, 32, hs, 3 * W // 8, W // 4, ff=ff, limit=7.0)]
    return arch_synth.vanapel_config(W, case["vocab"], (kinds * n)[:n], groups=4)


def _layer_weights(cfg, seed):
    """bfloat16 bit patterns of every tensor of a layer-list model: uniform within a binade for the matrices, normal for the vectors"""
    jobs = []
    W, V = cfg["width"], cfg["vocab"]
    nuf = cfg["architecture"] == "Nufusun"

    def mat(name, o, i, gain=1.0):
        jobs.append((name, (o, i), gain / math.sqrt(i), None))

    def vec(name, shape, std, mean=0.0):
        jobs.append((name, shape if isinstance(shape, tuple) else (shape,), std, mean))

    nrm = 0.0 if nuf else 1.0
    mat("embed", V, W, math.sqrt(W))
    mat("head", V, W)
    vec("final.norm", W, 0.1, nrm)
    for i, l in enumerate(cfg["layers"]):
        p, m, f = "l%d." % i, l["mixer"], l["mlp"]
        H, dv = m["heads"], m["vdim"]
        vec(p + "norm1", W, 0.1, nrm)
        if nuf:
            G, dq = m["kv_heads"], m["dim"]
            for n, o, g in (("q", H * dq, 2.0), ("k", G * dq, 2.0), ("v", G * dv, 1.0)):
                mat(p + "mix." + n, o, W, g)
                vec(p + "mix.%s.b" % n, o, 0.1)
            vec(p + "mix.o.b", W, 0.1)
            vec(p + "mix.rel", (32, H), 0.7)
            vec(p + "mix.talk", (H, H), 0.2, "eye")
            vec(p + "mix.temp", H, 0.2, 1.0)
            mat(p + "mlp.router", 8, W, 2.0)
            for e in range(8):
                mat(p + "mlp.e%d.gate" % e, f["expert"]["ff"], W, 1.5)
                mat(p + "mlp.e%d.up" % e, f["expert"]["ff"], W, 1.5)
                mat(p + "mlp.e%d.down" % e, W, f["expert"]["ff"])
        else:
            vec(p + "norm1b", W, 0.1, 0.5)
            vec(p + "norm2", W, 0.1, 1.0)
            vec(p + "norm2b", W, 0.1, 0.5)
            vec(p + "mix.sink", H, 1.0)
            if l["type"] == "attention":
                G, dq = m["kv_heads"], m["dim"]
                mat(p + "mix.q", H * dq, W)
                mat(p + "mix.k", G * dq, W)
                mat(p + "mix.v", G * dv, W)
                vec(p + "mix.r1", H, 0.1, 0.3)
                vec(p + "mix.r2", H, 0.2, 0.8)
            else:
                dn, dr, rq, rk = m["dim"], m["rot_dim"], m["q_rank"], m["kv_rank"]
                mat(p + "mix.dq", rq, W)
                vec(p + "mix.dq.norm", rq, 0.1, 1.0)
                mat(p + "mix.uq", H * (dn + dr), rq, 2.0)
                mat(p + "mix.dkv", rk + dr, W, 2.0)
                vec(p + "mix.dkv.norm", rk, 0.1, 1.0)
                mat(p + "mix.uk", H * dn, rk, 2.0)
                mat(p + "mix.uv", H * dv, rk)
            mat(p + "mlp.gate", f["ff"], W, 1.5)
            mat(p + "mlp.up", f["ff"], W, 1.5)
            mat(p + "mlp.down", W, f["ff"])
        mat(p + "mix.o", W, H * dv)

    def make(job):
        k, (name, shape, scale, mean) = job
        r = _rng(seed, 3000 + k)
        if mean is None:    # |w| uniform in [2^e, 2^(e + 1)), so that std is about `scale`
            e = int(math.floor(math.log2(scale / 1.1))) + 127
            bits = np.frombuffer(r.bytes(2 * shape[0] * shape[1]), np.uint16).reshape(shape)
            return name, (bits & np.uint16(0x807F)) | np.uint16(e << 7)
        v = r.standard_normal(shape).astype(np.float32) * np.float32(scale)
        v = v + (np.eye(shape[0], dtype=np.float32) if mean == "eye" else np.float32(mean))
        if name.endswith(("r1", "r2")):
            v = np.abs(v) + np.float32(0.05)
        return name, (np.ascontiguousarray(v).view(np.uint32) >> 16).astype(np.uint16).reshape(shape)

    with ThreadPoolExecutor(8) as ex:
        return dict(ex.map(make, enumerate(jobs)))


# ---------------------------------------------------------------------------------------------------------------- state and run
class _Context:
    """a model or an operator table and the device buffers on it; released with the last state or output that refers to it"""

    def __init__(self, case):
        self.case, self.model, self.be, self.buffers = case, None, None, []

    def view(self, ptr, *shape):
        """device memory of the context as a torch tensor, which keeps the context"""
        return torch.as_tensor(_View(self, ptr, shape), device="cuda")

    def __del__(self):
        try:
            for b in self.buffers:
                b.free()
            if self.model is not None:
                self.model.close()
            elif self.be is not None:
                self.be.close()
        except Exception:   # the interpreter is on its way out
            pass


class _View:
    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": tuple(shape), "typestr": "<f4", "version": 3}


class _State:
    pass


def prepare(case, seed):
    s, c = _State(), _Context(case)
    s.case, s.own, s.model = case, c, None
    if case["kind"] == "matmul":
        t, K, N, bs = QUANTS[case["quant"]], case["k"], case["n"], case["batch"]
        s.be = c.be = capi.CudaBackend(capi.desc_from_model_json(synth.model_json(synth.PRESETS["slice-8b"]), max_batch=128, n_ctx=256))
        s.host = _matmul_weight(case, seed)
        s.w = s.be.register_weight(s.host, t, K, N)
        s.x, s.y = s.be.upload(_matmul_input(case, seed)), s.be.empty(N * bs)
        c.buffers = [s.x, s.y]
        s.out = c.view(s.y.ptr, bs, N)
        s.be.sync()
        return s
    past, s.now = _tokens(case, seed)
    if case["kind"] == "layers":
        cfg = _layer_config(case)
        d = tempfile.mkdtemp(prefix="perf_case_", dir="/dev/shm" if os.path.isdir("/dev/shm") else None)
        try:
            arch_synth.write_model_dir(d, cfg, _layer_weights(cfg, seed))
            s.model = c.model = arch.load_model(d, dtype=case["dtype"], max_batch=256, n_ctx=_n_ctx(case))
        finally:
            shutil.rmtree(d, ignore_errors=True)
        chunk = 256
    else:
        s.model = c.model = capi.CudaModel(desc=capi.desc_from_model_json(synth.model_json(_shape(case, _n_ctx(case))), max_batch=128, n_ctx=_n_ctx(case), qkv_bias=SHAPES[case["shape"]][10]),
                                 tensors=_tensors(case, seed))
        chunk = 128
    if case["kind"] == "sessions":
        s.ids, s.lens = [0] + [s.model.session_create() for _ in range(case["batch"] - 1)], [len(p) for p in past]
        past = dict(zip(s.ids, past))
    for sid, p in (past if case["kind"] == "sessions" else {0: past}).items():
        s.model.session_select(sid)
        for lo in range(0, len(p), chunk):
            s.model.forward(p[lo:lo + chunk], lm_head=False)
    if case["kind"] == "verify":
        depth, s.mask = _tree(case, seed)
        s.pos = [case["ctx"] + d for d in depth]
    if case["kind"] != "sessions":
        s.logits = c.view(s.model.be.logits_dev(), case.get("batch", 1), case["vocab"])
    if case["kind"] in ("decode", "prefill", "verify"):
        s.rows = _rows(s, case.get("batch", 1), case["ctx"])
    return s


def _rows(s, n, ctx):
    """the cache rows of the call's tokens in every layer: K [n][kv], V [kv][n]"""
    a = SHAPES[s.case["shape"]]
    kvd, n_ctx, got = a[4] * a[5], _n_ctx(s.case), []
    for L in range(s.case["layers"]):
        got.append(s.own.view(s.model.be.kv_k(L), n_ctx, kvd)[ctx:ctx + n])
        got.append(s.own.view(s.model.be.kv_v(L), kvd, n_ctx)[:, ctx:ctx + n])
    return got


def run(s):
    c, m = s.case, s.model
    if c["kind"] == "matmul":
        s.be.matmul(s.y, s.w, QUANTS[c["quant"]], c["k"], c["n"], s.x, c["batch"])
        return s.out
    if c["kind"] == "sessions":
        for t in range(c["steps"]):     # greedy picks come back, at the end all logits
            logits, ids = m.forward_sessions(s.ids, s.now[:, t], want_logits=t == c["steps"] - 1)
        for sid in s.ids:               # the conversations are where they were, for the next pass
            m.session_select(sid)
            m.be.kv_rollback(c["steps"])
        return {"logits": logits, "ids": ids}
    m.be.kv_truncate(c["ctx"])          # what an earlier pass appended
    if c["kind"] == "verify":
        return {"logits": m.forward_tree(s.now, s.pos, s.mask), "cache": s.rows}
    if c["kind"] == "decode":
        if c["pick"] == "host":
            return {"logits": m.forward(s.now), "cache": s.rows}
        m.forward_lazy(s.now)
        best, ids = m.sample_topk(40)
        return {"best": best, "ids": ids, "logits": s.logits, "cache": s.rows}
    if c["kind"] == "layers":
        if c["batch"] == 1:
            return m.forward(s.now)
        m.forward_lazy(s.now)
        return s.logits
    if c["head"]:
        m.forward_lazy(s.now)
        return {"logits": s.logits, "cache": s.rows}
    m.forward(s.now, lm_head=False)
    return {"cache": s.rows}


# ---------------------------------------------------------------------------------------------------------------- bytes and operations
def work(case):
    if case["kind"] == "matmul":
        K, N, bs = case["k"], case["n"], case["batch"]
        return {"bytes": gguf.row_bytes(QUANTS[case["quant"]], K) * N + 4 * bs * (K + N), "flops": 2 * K * N * bs}
    bs, ctx, V = case.get("batch", 1), case["ctx"], case["vocab"]
    if case["kind"] == "layers":
        cfg, w, act, kv, attn = _layer_config(case), 0, 0, 0, 0
        W = cfg["width"]
        for l in cfg["layers"]:
            m = l["mixer"]
            H, dv = m["heads"], m["vdim"]
            if l["type"] == "attention":
                mix, row, sees = (H * m["dim"] + m["kv_heads"] * (m["dim"] + dv) + H * dv) * W, m["kv_heads"] * (m["dim"] + dv), min(ctx, (m.get("mask") or {}).get("size", ctx))
                attn += 2 * H * (m["dim"] + dv) * (min(sees, ctx) + (bs + 1) / 2) * bs
            else:
                rq, rk, dn, dr = m["q_rank"], m["kv_rank"], m["dim"], m["rot_dim"]
                mix, row, sees = rq * W + H * (dn + dr) * rq + (rk + dr) * W + H * (dn + dv) * rk + H * dv * W, rk + dr, ctx
                attn += 2 * H * (2 * rk + dr) * (ctx + (bs + 1) / 2) * bs
            if cfg["architecture"] == "Nufusun":
                ff = l["mlp"]["expert"]["ff"]
                w += mix + min(8, 2 * bs) * 3 * ff * W
                act += mix + 2 * 3 * ff * W
            else:
                w += mix + 3 * l["mlp"]["ff"] * W
                act += mix + 3 * l["mlp"]["ff"] * W
            kv += 4 * row * (sees + bs)
        return {"bytes": 2 * (w + V * W) + kv + 4 * bs * V, "flops": 2 * bs * (act + V * W) + attn}
    _, dim, ffn, nh, nkv, hs, _, _, _, _, _ = SHAPES[case["shape"]]
    L, head = case["layers"], case["kind"] != "prefill" or case["head"]
    params = L * (dim * hs * (2 * nh + 2 * nkv) + 3 * dim * ffn)
    steps = case.get("steps", 1)
    wb = (gguf.row_bytes(QUANTS[case["quant"]], 256 * 1024) / (256 * 1024)) * params
    wb += gguf.row_bytes(QUANTS[case["out"] or case["quant"]], dim) * V * head
    own = 1 if case["kind"] in ("sessions", "decode") else (bs + 1) / 2
    past = 0.75 * ctx if case["kind"] == "sessions" else ctx
    kv = L * 2 * nkv * hs * 4 * (past * (bs if case["kind"] == "sessions" else 1) + bs)
    attn = L * 4 * nh * hs * (past + own) * bs
    return {"bytes": steps * (wb + kv) + 4 * bs * V * head, "flops": steps * (2 * bs * (params + V * dim * head) + attn)}


def tolerance(case):
    if case["kind"] != "layers":
        return "exact"      # block formats: results are defined bit by bit, whatever the batch a token comes in
    # measured as the largest difference between the fp32-FMA products and the tensor-core ones (sums in another order), times four.
    # bfloat16 operands are rounded after every product, so an ulp of an fp32 sum becomes 2^-9 of a value here and there: 9e-5 in a
    # model of one Nufusun block, 3e-3 in one of two Vanapel layers with a norm on both sides of each sublayer.  float32: both orders
    # agree to the bit today; the sums' own error against 64 bits is 2.5e-6.
    if case["dtype"] == "float32":
        return {"rel": 1e-5}
    return {"rel": 5e-4} if case["arch"] == "nufusun" else {"rel": 1.2e-2}


# ---------------------------------------------------------------------------------------------------------------- the same in 64 bits
_DEV = "cuda" if torch.cuda.is_available() else "cpu"


def _blocks(raw, nbytes):
    return torch.from_numpy(np.array(raw, np.uint8).reshape(-1, nbytes)).to(_DEV)


def _f16(b):
    return b.contiguous().view(torch.float16).double()


def _dequant(raw, t, K, N):
    """[N][K] of a GGUF matrix in 64 bits"""
    B = _blocks(raw, gguf.TYPE_INFO[t][1])
    if t in (gguf.GGML_Q4_0, gguf.GGML_Q8_0):
        d, q = _f16(B[:, :2]), B[:, 2:]
        v = torch.cat([q & 15, q >> 4], 1).double() - 8 if t == gguf.GGML_Q4_0 else q.contiguous().view(torch.int8).double()
        return (v * d).reshape(N, K)
    if t == gguf.GGML_Q6_K:
        ql, qh, sc, d = B[:, :128].reshape(-1, 2, 64), B[:, 128:192].reshape(-1, 2, 32), B[:, 192:208].contiguous().view(torch.int8).double(), _f16(B[:, 208:210])
        lo = [ql[:, :, :32] & 15, ql[:, :, 32:] & 15, ql[:, :, :32] >> 4, ql[:, :, 32:] >> 4]
        q = torch.stack([lo[k] | (((qh >> (2 * k)) & 3) << 4) for k in range(4)], 2).double() - 32     # [nb][2][4][32]
        return (q.reshape(-1, 16, 16) * sc[:, :, None] * d[:, :, None]).reshape(N, K)
    d, dmin, s = _f16(B[:, 0:2]), _f16(B[:, 2:4]), B[:, 4:16]
    sc = torch.cat([s[:, 0:4] & 63, (s[:, 8:12] & 15) | ((s[:, 0:4] >> 6) << 4)], 1).double()
    mn = torch.cat([s[:, 4:8] & 63, (s[:, 8:12] >> 4) | ((s[:, 4:8] >> 6) << 4)], 1).double()
    qs = B[:, -128:].reshape(-1, 4, 1, 32)
    q = torch.cat([qs & 15, qs >> 4], 2).reshape(-1, 8, 32)
    if t == gguf.GGML_Q5_K:
        bit = torch.arange(8, device=_DEV, dtype=torch.uint8)[None, :, None]
        q = q | (((B[:, 16:48][:, None, :] >> bit) & 1) << 4)
    return (q.double() * (sc * d)[:, :, None] - (mn * dmin)[:, :, None]).reshape(N, K)


def _rounded(x, t):
    """activations as the block formats take them: one signed byte per element and a scale per block"""
    x = x.float()
    if t in (gguf.GGML_Q4_0, gguf.GGML_Q8_0):
        b = x.reshape(x.shape[0], -1, 32)
        d = b.abs().amax(-1, keepdim=True) / 127
        q = torch.round(b * torch.where(d > 0, 1 / d, torch.zeros_like(d)))
        return (q.double() * d.half().double()).reshape(x.shape)
    b = x.reshape(x.shape[0], -1, 256)
    top = torch.gather(b, -1, b.abs().argmax(-1, keepdim=True))
    inv = torch.where(top != 0, -127 / top, torch.zeros_like(top))
    q = torch.clamp(torch.round(inv * b), max=127)
    return (q.double() * torch.where(inv != 0, 1 / inv, torch.zeros_like(inv)).double()).reshape(x.shape)


def _matmul_weight(case, seed):
    return synth.random_blocks(np.random.default_rng(seed), QUANTS[case["quant"]], case["n"], case["k"], case["k"] ** -0.5)


def _matmul_input(case, seed):
    return _rng(seed, 1).standard_normal((case["batch"], case["k"]), dtype=np.float32)


def _softmax_rows(s, ok, extra=None):
    """soft-max over the visible keys; `extra`: the logit of one more term in the denominator"""
    s = s.masked_fill(~ok, -math.inf)
    top = s.amax(-1, keepdim=True)
    if extra is not None:
        top = torch.maximum(top, extra)
    e = torch.exp(s - top)
    return e / (e.sum(-1, keepdim=True) + (torch.exp(extra - top) if extra is not None else 0))


def _exact_llama(case, seed):
    T, (_, dim, ffn, nh, nkv, hs, _, rope, base, eps, bias) = _tensors(case, seed), SHAPES[case["shape"]]

    def mat(x, name):
        t = T[name]
        return _rounded(x, t.ggml_type) @ _dequant(t.data, t.ggml_type, t.shape[0], t.shape[1]).T

    def vec(name):
        return torch.from_numpy(T[name].data.view(np.float32).copy()).to(_DEV).double()

    def norm(x, name):
        return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * vec(name)

    past, now = _tokens(case, seed)
    if case["kind"] == "sessions":
        seqs = [np.concatenate([p, q]) for p, q in zip(past, now)]
    else:
        seqs = [np.concatenate([past, now])]
    spans, lo = [], 0
    for q in seqs:
        spans.append((lo, lo + len(q)))
        lo += len(q)
    tok = torch.from_numpy(np.concatenate(seqs).astype(np.int64)).to(_DEV)
    pos = torch.cat([torch.arange(b - a, device=_DEV) for a, b in spans]).double()
    masks = [torch.ones(b - a, b - a, dtype=torch.bool, device=_DEV).tril() for a, b in spans]
    if case["kind"] == "verify":
        depth, m = _tree(case, seed)
        pos[case["ctx"]:] = case["ctx"] + torch.tensor(depth, device=_DEV, dtype=torch.float64)
        masks[0][case["ctx"]:, case["ctx"]:] = torch.from_numpy(m).to(_DEV).bool()
    ang = pos[:, None, None] * base ** (-2.0 * torch.arange(hs // 2, device=_DEV).double() / hs)
    cs, sn = torch.cos(ang), torch.sin(ang)

    def turn(x):
        u, v = (x[..., :hs // 2], x[..., hs // 2:]) if rope & 2 else (x[..., 0::2], x[..., 1::2])
        u, v = u * cs - v * sn, u * sn + v * cs
        return torch.cat([u, v], -1) if rope & 2 else torch.stack([u, v], -1).reshape(x.shape)

    e = T["token_embd.weight"]
    rb = gguf.row_bytes(e.ggml_type, dim)
    uniq, inv = torch.unique(tok, return_inverse=True)
    x = _dequant(e.data.reshape(-1, rb)[uniq.cpu().numpy()], e.ggml_type, dim, len(uniq))[inv]
    cache = []
    for L in range(case["layers"]):
        p = "blk.%d." % L
        h = norm(x, p + "attn_norm.weight")
        q, k, v = (mat(h, p + "attn_%s.weight" % c) + (vec(p + "attn_%s.bias" % c) if bias else 0) for c in "qkv")
        q, k, v = turn(q.reshape(-1, nh, hs)), turn(k.reshape(-1, nkv, hs)), v.reshape(-1, nkv, hs)
        cache += [k.reshape(-1, nkv * hs), v.reshape(-1, nkv * hs).T]
        y = torch.empty_like(q)
        for (a, b), ok in zip(spans, masks):
            for g in range(nkv):
                r = nh // nkv
                s = torch.einsum("ihd,jd->hij", q[a:b, g * r:(g + 1) * r], k[a:b, g]) / math.sqrt(hs)
                y[a:b, g * r:(g + 1) * r] = torch.einsum("hij,jd->ihd", _softmax_rows(s, ok), v[a:b, g])
        x = x + mat(y.reshape(-1, nh * hs), p + "attn_output.weight")
        h = norm(x, p + "ffn_norm.weight")
        g = mat(h, p + "ffn_gate.weight")
        x = x + mat(g / (1 + torch.exp(-g)) * mat(h, p + "ffn_up.weight"), p + "ffn_down.weight")
    head = "output.weight" if "output.weight" in T else "token_embd.weight"
    if case["kind"] == "sessions":
        return {"logits": mat(norm(x[[b - 1 for _, b in spans]], "output_norm.weight"), head), "ids": None}
    n, ctx = len(now), case["ctx"]
    got = {"cache": [t[ctx:] if i % 2 == 0 else t[:, ctx:] for i, t in enumerate(cache)]}
    if case["kind"] != "prefill" or case["head"]:
        got["logits"] = mat(norm(x[-n:], "output_norm.weight"), head)
    if case["kind"] == "decode" and case["pick"] == "topk":
        got["best"], got["ids"] = torch.topk(got["logits"][0], 40).values, None
    return got


def _exact_layers(case, seed):
    cfg = _layer_config(case)
    T = {k: (torch.from_numpy(v.astype(np.int32) << 16).view(torch.float32)).to(_DEV).double() for k, v in _layer_weights(cfg, seed).items()}
    eps, W = cfg["norm"]["eps"], cfg["width"]
    past, now = _tokens(case, seed)
    tok = torch.from_numpy(np.concatenate([past, now]).astype(np.int64)).to(_DEV)
    n = len(tok)
    dist = torch.arange(n, device=_DEV)[:, None] - torch.arange(n, device=_DEV)[None, :]
    nuf = cfg["architecture"] == "Nufusun"
    parts = 1 if nuf else cfg["norm"]["groups"]

    def norm(x, name):
        p = x.reshape(n, parts, -1)
        return (p / torch.sqrt((p * p).mean(-1, keepdim=True) + eps)).reshape(n, -1) * (T[name] + (1.0 if nuf else 0.0))

    def unit(v):
        return v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)

    def gated(z, gate, up, down, limit):
        g, u = torch.clamp(z @ gate.T, max=limit), torch.clamp(z @ up.T, -limit, limit)
        return (g / (1 + torch.exp(-1.702 * g)) * (u + 1)) @ down.T

    x = T["embed"][tok]
    for i, l in enumerate(cfg["layers"]):
        p, m, f = "l%d." % i, l["mixer"], l["mlp"]
        H, dv = m["heads"], m["vdim"]
        h = norm(x, p + "norm1")
        if l["type"] == "attention":
            G, dq = m["kv_heads"], m["dim"]
            q, k, v = h @ T[p + "mix.q"].T, h @ T[p + "mix.k"].T, h @ T[p + "mix.v"].T
            if nuf:
                q, k, v = q + T[p + "mix.q.b"], k + T[p + "mix.k.b"], v + T[p + "mix.v.b"]
            q, k, v = q.reshape(n, H, dq), k.reshape(n, G, dq), v.reshape(n, G, dv).repeat_interleave(H // G, 1)
            if not nuf:
                q, k = unit(q), unit(k)
            s = torch.einsum("ihd,jhd->hij", q, k.repeat_interleave(H // G, 1)) * m["scale"]
            if nuf:
                rel = T[p + "mix.rel"]
                B, half = rel.shape[0], rel.shape[0] // 2
                far = np.arange(n, dtype=np.float32)
                with np.errstate(divide="ignore"):
                    b = half + np.floor(np.log(far / np.float32(half)) / np.float32(math.log(m["bias_max"] / half)) * np.float32(B - half))
                bucket = torch.from_numpy(np.where(far < half, far, np.minimum(b, B - 1)).astype(np.int64)).to(_DEV)
                s = s * T[p + "mix.temp"][:, None, None] + rel[bucket[dist.clamp(min=0)]].permute(2, 0, 1)
                s = torch.einsum("hg,gij->hij", T[p + "mix.talk"], s)
                sink, ok = torch.zeros(1, 1, 1, device=_DEV, dtype=torch.float64), dist >= 0
            else:
                s = s - T[p + "mix.r1"][:, None, None] * torch.log1p(T[p + "mix.r2"][:, None, None] * dist.clamp(min=0).double())
                sink, ok = T[p + "mix.sink"][:, None, None], (dist >= 0) & (dist < m["mask"]["size"])
        else:
            dn, dr, rk, D = m["dim"], m["rot_dim"], m["kv_rank"], m["rot"]["dims"]
            a = torch.arange(n, device=_DEV).double()[:, None, None] * m["rot"]["base"] ** (-2.0 * torch.arange(D // 2, device=_DEV).double() / D)

            def turn(t):
                u, w = t[..., :D // 2], t[..., D // 2:D]
                return torch.cat([u * torch.cos(a) - w * torch.sin(a), w * torch.cos(a) + u * torch.sin(a), t[..., D:]], -1)

            q = ((unit(h @ T[p + "mix.dq"].T) * T[p + "mix.dq.norm"]) @ T[p + "mix.uq"].T).reshape(n, H, dn + dr)
            t = h @ T[p + "mix.dkv"].T
            c = unit(t[:, :rk]) * T[p + "mix.dkv.norm"]
            k, v = (c @ T[p + "mix.uk"].T).reshape(n, H, dn), (c @ T[p + "mix.uv"].T).reshape(n, H, dv)
            s = (torch.einsum("ihd,jhd->hij", q[..., :dn], k) + torch.einsum("ihd,jd->hij", turn(q[..., dn:]), turn(t[:, None, rk:])[:, 0])) * m["scale"]
            sink, ok = T[p + "mix.sink"][:, None, None], dist >= 0
        y = torch.einsum("hij,jhd->ihd", _softmax_rows(s, ok, sink), v).reshape(n, H * dv) @ T[p + "mix.o"].T
        if nuf:
            score = torch.sigmoid(h @ T[p + "mlp.router"].T)
            best = torch.topk(score, 2, -1).indices
            y = y + T[p + "mix.o.b"]
            for e in range(8):
                z = score[:, e:e + 1] * h
                mine = (best == e).any(-1, keepdim=True)
                y = y + mine * gated(z, T[p + "mlp.e%d.gate" % e], T[p + "mlp.e%d.up" % e], T[p + "mlp.e%d.down" % e], f["expert"]["limit"])
            x = x + y
        else:
            x = x + norm(y, p + "norm1b")
            x = x + norm(gated(norm(x, p + "norm2"), T[p + "mlp.gate"], T[p + "mlp.up"], T[p + "mlp.down"], f["limit"]), p + "norm2b")
    return norm(x, "final.norm")[-case["batch"]:] @ T["head"].T


def exact(case, seed):
    if case["kind"] == "matmul":
        t, K, N = QUANTS[case["quant"]], case["k"], case["n"]
        x = torch.from_numpy(_matmul_input(case, seed)).to(_DEV)
        return _rounded(x, t) @ _dequant(_matmul_weight(case, seed), t, K, N).T
    return _exact_layers(case, seed) if case["kind"] == "layers" else _exact_llama(case, seed)
