"""The work that users of this library have it do, as cases that can be timed and compared.

Five kinds of case, each through the public entry points a program calls:

  matmul    pib_quantize_act / pib_norm_quantize_act + pib_gemv: one quantised weight matrix times the 1..16 tokens of a decode or verification batch
  prompt    pib_quantize_act_rows + pib_gemm: one Q4_K matrix times the tokens of a prompt pass
  step      llama_decode of 1..16 tokens of one sequence behind a prompt, llama architecture: a draft step, a plain decode step or a verification batch
  ingest    llama_decode of a whole prompt, llama architecture, Q4_K
  layers    llama_decode on two layers of a layer-list model (attention with distance slopes and with distance buckets, dense feed-forwards, bfloat16
            operands): prompts of several sequences in one batch, then steps of one decoded token of each
"""
import ctypes as C
import json
import math
import os
import shutil
import struct
import tempfile

import numpy as np
import torch

from pipeinfer_b200 import design_bench, lib as pib, llama

Q4_0, Q8_0, Q3_K, Q4_K, Q5_K, Q6_K = pib.TYPE_Q4_0, pib.TYPE_Q8_0, pib.TYPE_Q3_K, pib.TYPE_Q4_K, pib.TYPE_Q5_K, pib.TYPE_Q6_K
TYPE = {"q4_0": Q4_0, "q8_0": Q8_0, "q3_k": Q3_K, "q4_k": Q4_K, "q5_k": Q5_K, "q6_k": Q6_K}
EPS = 1e-5


def listed():
    return [
        # query | key | value projection of the 1.1B draft, one token: the smallest call of a draft step, all latency
        {"name": "matmul_q4k_draft_b1", "kind": "matmul", "type": "q4_k", "N": 2560, "K": 2048, "b": 1, "norm": True},
        # gate | up of the 70B-shaped target, a verification batch of four tokens: the launch that reads most weights
        {"name": "matmul_q4k_gate_up_b4", "kind": "matmul", "type": "q4_k", "N": 57344, "K": 8192, "b": 4, "norm": True},
        # its down projection at a wide verification batch (three drafted branches), a ragged token count
        {"name": "matmul_q4k_down_b13", "kind": "matmul", "type": "q4_k", "N": 8192, "K": 28672, "b": 13, "norm": False},
        # gate | up of the 7B Q4_0 target, a verification batch of seven
        {"name": "matmul_q4_0_gate_up_b7", "kind": "matmul", "type": "q4_0", "N": 22016, "K": 4096, "b": 7, "norm": True},
        # output matrix of a Q4_K_M file (Q6_K rows), three tokens
        {"name": "matmul_q6k_head_b3", "kind": "matmul", "type": "q6_k", "N": 32000, "K": 8192, "b": 3, "norm": True},
        # a short prompt through the 70B target's query | key | value projection
        {"name": "prompt_q4k_qkv_40", "kind": "prompt", "N": 10240, "K": 8192, "b": 40},
        # a full prompt pass of 256 tokens through its gate | up
        {"name": "prompt_q4k_gate_up_256", "kind": "prompt", "N": 57344, "K": 8192, "b": 256},
        # one step of the 1.1B-shaped Q4_K draft behind 300 tokens, with its logits
        {"name": "step_draft", "kind": "step", "type": "q4_k", "layers": 22, "embd": 2048, "heads": 32, "kv_heads": 4, "ff": 5632, "vocab": 32000, "past": 300, "b": 1},
        # a verification batch of four tokens on 7B-shaped Q4_0 layers behind 200 tokens
        {"name": "step_verify_q4_0_b4", "kind": "step", "type": "q4_0", "layers": 8, "embd": 4096, "heads": 32, "kv_heads": 32, "ff": 11008, "vocab": 32000, "past": 200, "b": 4},
        # a 700-token prompt through 4096-wide Q4_K layers, the logits of its last token
        {"name": "ingest_w4096_700", "kind": "ingest", "layers": 4, "embd": 4096, "heads": 32, "kv_heads": 32, "ff": 11008, "vocab": 32000, "tokens": 700},
        # prompts of three sequences in one batch through two 2048-wide layers of a layer-list model
        {"name": "layers_prompts_w2048", "kind": "layers", "width": 2048, "heads": 16, "window": 1024, "ff": 5632, "vocab": 8000, "seqs": 3, "tokens": 517, "steps": 0},
        # four requests from start to end through the same layers: short prompts in one batch, then 24 steps of one token each
        {"name": "layers_requests_w2048_4", "kind": "layers", "width": 2048, "heads": 16, "window": 1024, "ff": 5632, "vocab": 8000, "seqs": 4, "tokens": 90, "steps": 24},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matmul", "matmul", "matmul", "prompt", "prompt", "step", "ingest", "layers", "layers"])
    if kind == "matmul":
        t = rng.choice(["q4_k", "q4_k", "q4_k", "q4_0", "q8_0", "q6_k", "q5_k", "q3_k"])
        while True:
            N, K = 16 * _log(rng, 64, 3584), 256 * _log(rng, 4, 112)
            if N * K <= 57344 * 8192:
                break
        return {"kind": "matmul", "type": t, "N": N - rng.choice([0, 0, 0, 5]), "K": K, "b": rng.randint(1, 16), "norm": K <= 14848 and rng.random() < 0.5}
    if kind == "prompt":
        while True:
            N, K = 16 * _log(rng, 64, 3584), 256 * _log(rng, 8, 112)
            if N * K <= 57344 * 8192:
                break
        return {"kind": "prompt", "N": N - rng.choice([0, 0, 0, 3]), "K": K, "b": _log(rng, 17, 256)}
    if kind == "step":
        embd, heads, kv, ff = rng.choice([(2048, 32, 4, 5632), (1024, 8, 8, 2816), (4096, 32, 32, 11008), (2048, 16, 16, 5632), (4096, 32, 8, 14336)])
        return {"kind": "step", "type": rng.choice(["q4_k", "q4_k", "q4_0", "q8_0"]), "layers": rng.randint(2, 8 if embd > 2048 else 22), "embd": embd, "heads": heads, "kv_heads": kv,
                "ff": ff, "vocab": 32000, "past": rng.randint(20, 900), "b": _log(rng, 1, 16)}
    if kind == "ingest":
        embd, heads, kv, ff = rng.choice([(2048, 32, 4, 5632), (1024, 8, 8, 2816), (4096, 32, 32, 11008), (2048, 16, 16, 5632), (4096, 32, 8, 14336)])
        return {"kind": "ingest", "layers": rng.randint(2, 3), "embd": embd, "heads": heads, "kv_heads": kv, "ff": ff, "vocab": 32000, "tokens": _log(rng, 34, 700)}
    width, heads, ff = rng.choice([(1024, 8, 2816), (2048, 16, 5632), (2048, 16, 4000)])
    c = {"kind": "layers", "width": width, "heads": heads, "window": rng.choice([512, 1024]), "ff": ff, "vocab": rng.choice([4000, 8000])}
    if rng.random() < 0.5:
        return dict(c, seqs=rng.randint(1, 4), tokens=_log(rng, 20, 500), steps=0)
    return dict(c, seqs=rng.randint(1, 8), tokens=rng.randint(20, 200), steps=rng.randint(4, 18))


# ---- quantised blocks as the reference's files hold them ----------------------------------------------------------------------------
def _gen(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1000003 + salt) % (1 << 62))
    return g


def _scale(n, mean, g):
    """block scales spread around `mean`, as fp16"""
    return ((torch.rand(n, device="cuda", generator=g) + 0.5) * mean).to(torch.float16)


def _blocks(t, N, K, seed):
    """[N, K / block, block bytes] on the device: every byte pattern is a valid block, the scales give weights of about 0.02 around zero"""
    g = _gen(seed, 1)
    el, by = pib.BLOCK[t]
    w = torch.randint(0, 256, (N, K // el, by), dtype=torch.uint8, device="cuda", generator=g)

    def put(at, mean):
        w[:, :, at:at + 2] = _scale((N, K // el), mean, g).view(torch.uint8).reshape(N, K // el, 2)
    if t == Q4_0:
        put(0, 0.0043)
    elif t == Q8_0:
        put(0, 0.00027)
    elif t in (Q4_K, Q5_K):
        put(0, 1.2e-4 if t == Q4_K else 0.6e-4)
        put(2, 9.0e-4)
    elif t == Q6_K:
        put(208, 1.5e-5)
    else:
        put(108, 4.5e-4)
    return w


def _f16(w, at):
    return w[..., at:at + 2].contiguous().view(torch.float16).double()


def _dequant(t, w):
    """float64 weights of blocks [rows, nb, bytes]: the formulas of the file format"""
    R, nb = w.shape[:2]
    i = w.to(torch.int32)
    if t == Q4_0:
        q = i[..., 2:18]
        return ((torch.cat([q & 15, q >> 4], -1) - 8).double() * _f16(w, 0)).reshape(R, -1)
    if t == Q8_0:
        return (w[..., 2:34].contiguous().view(torch.int8).double() * _f16(w, 0)).reshape(R, -1)
    if t in (Q4_K, Q5_K):
        s = i[..., 4:16]
        sc = torch.cat([s[..., 0:4] & 63, (s[..., 8:12] & 15) | ((s[..., 0:4] >> 6) << 4)], -1)
        mn = torch.cat([s[..., 4:8] & 63, (s[..., 8:12] >> 4) | ((s[..., 4:8] >> 6) << 4)], -1)
        by = 16 if t == Q4_K else 48
        q = i[..., by:by + 128].reshape(R, nb, 4, 1, 32)
        q = torch.cat([q & 15, q >> 4], 3).reshape(R, nb, 8, 32)
        if t == Q5_K:
            q = q + 16 * ((i[..., 16:48].unsqueeze(2) >> torch.arange(8, device=w.device).reshape(8, 1)) & 1)
        d, m = _f16(w, 0).unsqueeze(-1) * sc.double().unsqueeze(-1), _f16(w, 2).unsqueeze(-1) * mn.double().unsqueeze(-1)
        return (d * q.double() - m).reshape(R, -1)
    if t == Q6_K:
        ql, qh = i[..., 0:128].reshape(R, nb, 2, 2, 32), i[..., 128:192].reshape(R, nb, 2, 1, 32)
        low = torch.cat([ql & 15, ql >> 4], 3)
        q = low | (((qh >> (2 * torch.arange(4, device=w.device).reshape(4, 1))) & 3) << 4)
        sc = w[..., 192:208].contiguous().view(torch.int8).double().reshape(R, nb, 16, 1)
        return ((q - 32).double().reshape(R, nb, 16, 16) * sc * _f16(w, 208).unsqueeze(-1)).reshape(R, -1)
    h, q, s = i[..., 0:32].reshape(R, nb, 1, 1, 32), i[..., 32:96].reshape(R, nb, 2, 1, 32), i[..., 96:108]
    j = torch.arange(4, device=w.device).reshape(4, 1)
    v = ((q >> (2 * j)) & 3) - 4 * (1 - ((h >> (4 * torch.arange(2, device=w.device).reshape(2, 1, 1) + j)) & 1))
    lo = torch.cat([s[..., 0:8] & 15, s[..., 0:8] >> 4], -1)
    hi = torch.cat([(s[..., 8:12] >> (2 * k)) & 3 for k in range(4)], -1)
    sc = ((lo | (hi << 4)) - 32).double().unsqueeze(-1)
    return (v.double().reshape(R, nb, 16, 16) * sc * _f16(w, 108).unsqueeze(-1)).reshape(R, -1)


def _activations(b, K, norm, seed):
    """the residual stream in front of a norm (a few large channels), or what a gated product leaves (heavy tails)"""
    g = _gen(seed, 2)
    x = torch.randn(b, K, device="cuda", generator=g)
    if norm:
        x[:, torch.randint(0, K, (max(1, K // 512),), device="cuda", generator=g)] *= 12.0
        return x * 3.0, 1.0 + 0.2 * torch.randn(K, device="cuda", generator=g)
    return x * torch.randn(b, K, device="cuda", generator=g), None


def _quantised(t, x):
    """float64 values of the activations as the matmul of weight type t reads them (8-bit blocks, scales formed in fp32)"""
    b, K = x.shape
    if t in (Q4_0, Q8_0):
        v = x.reshape(b, -1, 32)
        a = v.abs().amax(-1, keepdim=True)
        q = torch.round(v * torch.where(a > 0, 127.0 / a, torch.zeros_like(a))).clamp(-128, 127)
        return (q.double() * (a / 127.0).to(torch.float16).double()).reshape(b, K)
    v = x.reshape(b, -1, 256)
    i = v.abs().argmax(-1, keepdim=True)
    s = -128.0 / v.gather(-1, i)
    return (torch.round(s * v).clamp(max=127).double() * (1.0 / s).double()).reshape(b, K)


class _Matrix:
    """an uploaded weight matrix and the buffers of a program that multiplies with it"""

    def __init__(self, c, seed):
        self.L = pib.load().L
        pib.load().init(0)
        t, N, K, b = TYPE[c.get("type", "q4_k")], c["N"], c["K"], c["b"]
        self.norm, self.gemm, self.N, self.K, self.b = c.get("norm", False), c["kind"] == "prompt", N, K, b
        blocks = _blocks(t, N, K, seed)
        torch.cuda.synchronize()
        self.w = self.L.pib_weight_from_device(t, blocks.data_ptr(), N, K)
        if not self.w:
            raise pib.PibError(self.L.pib_last_error().decode())
        self.family = t if t in (Q4_0, Q8_0) else Q4_K
        self.x, self.nw = _activations(b, K, self.norm, seed)
        self.act = torch.empty(self.L.pib_act_bytes(self.family, K, b), dtype=torch.uint8, device="cuda")
        self.y = torch.empty(b, N, device="cuda")
        if self.gemm:
            self.L.pib_gemm_scratch_bytes.restype, self.L.pib_gemm_scratch_bytes.argtypes = C.c_size_t, [C.c_int64, C.c_int]
            self.L.pib_gemm.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
            self.L.pib_quantize_act_rows.argtypes = self.L.pib_quantize_act.argtypes
            self.scratch = torch.empty(self.L.pib_gemm_scratch_bytes(K, b), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()

    def run(self):
        L, x, act, y = self.L, self.x.data_ptr(), self.act.data_ptr(), self.y.data_ptr()
        if self.gemm:
            rc = L.pib_quantize_act_rows(self.family, x, self.b, self.K, act, None) or L.pib_gemm(self.w, act, self.b, y, self.scratch.data_ptr(), None)
        else:
            rc = (L.pib_norm_quantize_act(self.family, 1, x, self.nw.data_ptr(), EPS, self.b, self.K, act, None, None) if self.norm
                  else L.pib_quantize_act(self.family, x, self.b, self.K, act, None)) or L.pib_gemv(self.w, act, self.b, y, 0, None)
        if rc:
            raise pib.PibError(L.pib_last_error().decode())
        return self.y

    def __del__(self):
        if getattr(self, "w", None):
            self.L.pib_weight_free(self.w)


# ---- whole calls --------------------------------------------------------------------------------------------------------------------
class _Decoder:
    """a context behind its prompt and the batch that it decodes next: each run takes the sequences back to where they were and decodes the batch again"""

    def __init__(self, ctx, prompts, batch, rows, again):
        self.ctx, self.L, self.rows, self.again = ctx, ctx.L, rows, again
        for s, toks in prompts:
            b, keep = llama.make_batch(toks, list(range(len(toks))), [[s]] * len(toks), 0, ctx.max_seq)
            self._decode(b)
        self.batch, self.keep = llama.make_batch(*batch, 1, ctx.max_seq)
        self.prompts = prompts

    def _decode(self, b):
        if self.L.llama_decode(self.ctx.ctx, b) != 0:
            raise pib.PibError(self.L.pib_last_error().decode())

    def run(self):
        for s, p in self.again:
            self.L.llama_kv_cache_seq_rm(self.ctx.ctx, s, p, -1)
        self.batch.batch_id += 1
        self._decode(self.batch)
        out = np.empty((len(self.rows), self.ctx.n_vocab), np.float32)
        for k, i in enumerate(self.rows):
            out[k] = np.ctypeslib.as_array(self.L.llama_get_logits_ith(self.ctx.ctx, i), shape=(self.ctx.n_vocab,))
        return out

    def __del__(self):
        if getattr(self, "ctx", None):
            self.ctx.close()


class _Requests:
    """requests from start to end on a model whose sequences cannot be taken back: prompts of several sequences in one batch, then `steps` decoded tokens of
    each (given ones, so that every run feeds the same), then the sequences end; the logits of every sequence's last token after each call"""

    def __init__(self, ctx, prompts, steps):
        self.ctx, self.L, self.S = ctx, ctx.L, len(prompts)
        lens = [len(p) for p in prompts]
        ends = [sum(lens[:s + 1]) - 1 for s in range(self.S)]
        calls = [([t for p in prompts for t in p], [i for n in lens for i in range(n)], [[s] for s, n in enumerate(lens) for _ in range(n)], ends)]
        calls += [(row, [n + k for n in lens], [[s] for s in range(self.S)], list(range(self.S))) for k, row in enumerate(steps)]
        self.calls = [llama.make_batch(*c[:3], 1, ctx.max_seq) + (c[3],) for c in calls]

    def run(self):
        ctx, L = self.ctx, self.L
        out = np.empty((len(self.calls), self.S, ctx.n_vocab), np.float32)
        for k, (batch, _, rows) in enumerate(self.calls):
            batch.batch_id += 1
            if L.llama_decode(ctx.ctx, batch) != 0:
                raise pib.PibError(L.pib_last_error().decode())
            for s, i in enumerate(rows):
                out[k, s] = np.ctypeslib.as_array(L.llama_get_logits_ith(ctx.ctx, i), shape=(ctx.n_vocab,))
        for s in range(self.S):
            L.llama_kv_cache_seq_rm(ctx.ctx, s, -1, -1)
        return out

    def __del__(self):
        if getattr(self, "ctx", None):
            self.ctx.close()


def _tokens(seed, salt, n, vocab):
    return [int(v) for v in np.random.default_rng([seed & 0xFFFFFFFF, salt]).integers(3, vocab, n)]


def _llama(c, seed):
    n = c.get("past", 0) + c.get("b", c.get("tokens", 0))
    # bigram flavour: the residual stream is dominated by the token, as in the benchmark's models
    ctx = llama.Context(None, n_ctx=256 * -(-(n + 32) // 256), max_seq=8,
                        synthetic=(c["layers"], c["embd"], c["heads"], c["kv_heads"], c["ff"], c["vocab"], TYPE[c.get("type", "q4_k")], 1, 1, 1.0))
    if c["kind"] == "step":
        P, b = c["past"], c["b"]
        return _Decoder(ctx, [(0, _tokens(seed, 1, P, c["vocab"]))], (_tokens(seed, 2, b, c["vocab"]), list(range(P, P + b)), [[0]] * b), list(range(b)), [(0, P)])
    T = c["tokens"]
    return _Decoder(ctx, [], (_tokens(seed, 1, T, c["vocab"]), list(range(T)), [[0]] * T), [T - 1], [(0, 0)])


def _layers_config(c):
    base = design_bench.gusedra_config(c["width"], c["vocab"], 1, c["heads"], c["window"], c["ff"], 4, 2, 64, 64)
    dense = {"kind": "dense", "ff": c["ff"]}
    return dict(base, layers=[dict(l, mlp=dense) for l in base["layers"][:2]])


BUCKETS = 32


def _layers_weights(c, seed):
    """name -> bfloat16 tensor on the device (the same model for every seed of the tokens)"""
    cfg, W, D = _layers_config(c), {}, c["width"]
    g = _gen(7, 3)

    def mat(name, r, k):
        W[name] = (torch.randn(r, k, device="cuda", generator=g) * (1.4 / math.sqrt(k))).bfloat16()

    def vec(name, mean, std, n=D):
        W[name] = (mean + std * torch.randn(n, device="cuda", generator=g)).bfloat16()
    W["embed"] = torch.randn(c["vocab"], D, device="cuda", generator=g).bfloat16()
    mat("head", c["vocab"], D)
    vec("final.norm", 1, 0.25), vec("final.norm.b", 0, 0.2)
    for i, jl in enumerate(cfg["layers"]):
        p, m = "l%d." % i, jl["mixer"]
        for n in ("norm1", "norm1b", "norm2", "norm2b"):
            vec(p + n, 1, 0.25), vec(p + n + ".b", 0, 0.2)
        vec(p + "ls1", 1, 0.25), vec(p + "ls2", 1, 0.25)
        H, G, d = m["heads"], m["kv_heads"], m["dim"]
        mat(p + "mix.q", H * d, D), mat(p + "mix.k", G * d, D), mat(p + "mix.v", G * d, D), mat(p + "mix.o", D, H * d)
        if jl["type"] == "attention":
            W[p + "mix.sink"] = (torch.rand(H, device="cuda", generator=g) * 3 - 1).bfloat16()
        else:
            W[p + "mix.rel"] = torch.randn(BUCKETS, H, device="cuda", generator=g).bfloat16()
            mat(p + "mix.g", H * d, D)
        mat(p + "mlp.up", c["ff"], D), mat(p + "mlp.down", D, c["ff"])
    return W


def _layers_tokens(c, seed):
    """prompts of unlike lengths, about c["tokens"] each, and the tokens decoded behind them"""
    return ([_tokens(seed, 1 + s, max(1, c["tokens"] - 13 * s), c["vocab"]) for s in range(c["seqs"])],
            [_tokens(seed, 1000 + k, c["seqs"], c["vocab"]) for k in range(c["steps"])])


def _layers(c, seed):
    W = _layers_weights(c, seed)
    folder = tempfile.mkdtemp(prefix="pib_layers_")
    try:
        head, off = {}, 0
        for name, w in W.items():
            head[name] = {"dtype": "BF16", "shape": list(w.shape), "data_offsets": [off, off + 2 * w.numel()]}
            off += 2 * w.numel()
        hj = json.dumps(head).encode()
        hj += b" " * (-len(hj) % 8)
        with open(os.path.join(folder, "model.safetensors"), "wb") as f:
            f.write(struct.pack("<Q", len(hj)) + hj)
            for w in W.values():
                f.write(w.view(torch.int16).cpu().numpy())
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(_layers_config(c), f)
        prompts, steps = _layers_tokens(c, seed)
        n = sum(len(p) for p in prompts) + c["seqs"] * c["steps"]
        ctx = llama.Context(None, n_ctx=256 * -(-(n + 64) // 256), max_seq=8, model_dir=folder, state_slots=8)
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    return _Requests(ctx, prompts, steps)


def prepare(c, seed):
    if c["kind"] in ("matmul", "prompt"):
        return _Matrix(c, seed)
    return _llama(c, seed) if c["kind"] in ("step", "ingest") else _layers(c, seed)


def run(state):
    return state.run()


# ---- what a pass cannot do without ----------------------------------------------------------------------------------------------------
def _bits(t):
    el, by = pib.BLOCK[t]
    return by / el


def work(c):
    if c["kind"] in ("matmul", "prompt"):
        N, K, b = c["N"], c["K"], c["b"]
        return {"bytes": N * K * _bits(TYPE[c.get("type", "q4_k")]) + 4.0 * b * (N + K), "flops": 2.0 * N * K * b}
    if c["kind"] in ("step", "ingest"):
        t, E, F, V = TYPE[c.get("type", "q4_k")], c["embd"], c["ff"], c["vocab"]
        G = E // c["heads"] * c["kv_heads"]
        n, past = (c["b"], c["past"]) if c["kind"] == "step" else (c["tokens"], 0)
        out = n if c["kind"] == "step" else 1                     # rows of logits that are read
        per = E * (2 * E + 2 * G + 3 * F)
        seen = n * past + n * (n + 1) // 2
        return {"bytes": (c["layers"] * per + V * E) * _bits(t) + c["layers"] * 4.0 * G * (past + n) + n * E * _bits(t) + 4.0 * out * V,
                "flops": 2.0 * n * c["layers"] * per + 2.0 * out * V * E + 4.0 * c["layers"] * E * seen}
    prompts, _ = _layers_tokens(c, 0)
    D, H, F, V, d, steps, S = c["width"], c["heads"], c["ff"], c["vocab"], 128, c["steps"], c["seqs"]
    G = max(1, H // 4)
    per = [D * (2 * H * d + 2 * G * d + 2 * F), D * (3 * H * d + 2 * G * d + 2 * F)]
    rows = sum(len(p) for p in prompts)
    seen = sum(sum(min(i + 1, c["window"]) for i in range(len(p))) for p in prompts)
    later = sum(sum(min(len(p) + k + 1, c["window"]) for k in range(steps)) for p in prompts)
    kv = 4.0 * 2 * G * d * 2                                       # both layers' cells of one token
    return {"bytes": 2.0 * (1 + steps) * (sum(per) + V * D) + kv * (rows + S * steps + later) + 4.0 * S * (1 + steps) * V + 2.0 * D * (rows + S * steps),
            "flops": 2.0 * (rows + S * steps) * sum(per) + 2.0 * S * (1 + steps) * V * D + 4.0 * 2 * H * d * (seen + later)}


def tolerance(c):
    if c["kind"] == "matmul":
        return {"rel": 1e-5, "max": 2e-4}
    if c["kind"] == "prompt":
        return {"rel": 1.5e-3, "max": 1e-2}
    if c["kind"] in ("step", "ingest"):
        return {"rel": 3.5e-3, "max": 4e-2}
    return {"rel": 1e-2, "max": 0.2}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------------------------
def exact(c, seed):
    if c["kind"] in ("matmul", "prompt"):
        return _exact_matmul(c, seed)
    if c["kind"] in ("step", "ingest"):
        return None                                               # these models' weights are drawn inside the library
    return _exact_layers(c, seed)


def _exact_matmul(c, seed):
    t, N, K, b = TYPE[c.get("type", "q4_k")], c["N"], c["K"], c["b"]
    x, nw = _activations(b, K, c.get("norm", False), seed)
    if nw is not None:
        x = (x * (1.0 / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True).float() + EPS))) * nw
    xq, blocks = _quantised(t, x), _blocks(t, N, K, seed)
    return torch.cat([xq @ _dequant(t, blocks[r:r + 2048]).T for r in range(0, N, 2048)], 1)


def _ln(x, w, b):
    v = x - x.mean(-1, keepdim=True)
    return v / torch.sqrt((v * v).mean(-1, keepdim=True) + EPS) * w + b


def _bucket_of(n, B, D):
    half = B // 2
    if n < half:
        return n
    return min(B - 1, half + math.floor(math.log(n / half) / math.log(D / half) * (B - half) + 1e-9))


def _exact_attention(h, W, p, jl):
    m, T = jl["mixer"], h.shape[0]
    H, G, d = m["heads"], m["kv_heads"], m["dim"]
    q = (h @ W[p + "q"].T).reshape(T, H, d)
    k, v = ((h @ W[p + n].T).reshape(T, G, d).repeat_interleave(H // G, 1) for n in ("k", "v"))
    s = torch.einsum("thd,jhd->htj", q, k) * m["scale"]
    dist = torch.arange(T, device=h.device).reshape(T, 1) - torch.arange(T, device=h.device)
    seen = (dist >= 0) & ((dist < m["mask"]["size"]) | (torch.arange(T, device=h.device) < m["mask"].get("keep_first", 0)))
    if jl["type"] == "attention":
        slope = torch.tensor([2.0 ** (-8.0 * (i + 1) / H) for i in range(H)], dtype=torch.float64, device=h.device)
        s = s - slope.reshape(H, 1, 1) * dist
        sink = W[p + "sink"].reshape(H, 1, 1).expand(H, T, 1)
        w = torch.softmax(torch.cat([s.masked_fill(~seen, -math.inf), sink], -1), -1)[..., :T]
    else:
        of = torch.tensor([_bucket_of(n, BUCKETS, m["bias_max"]) for n in range(T)], device=h.device)
        s = s + W[p + "rel"][of[dist.clamp(min=0)]].permute(2, 0, 1)
        w = torch.softmax(s.masked_fill(~seen, -math.inf), -1)
    o = torch.einsum("htj,jhd->thd", w, v).reshape(T, H * d)
    if jl["type"] != "attention":
        o = o * torch.sigmoid(h @ W[p + "g"].T)
    return o @ W[p + "o"].T


def _exact_layers(c, seed):
    cfg, W = _layers_config(c), {k: v.double() for k, v in _layers_weights(c, seed).items()}
    prompts, steps = _layers_tokens(c, seed)
    out = torch.empty(1 + c["steps"], c["seqs"], c["vocab"], dtype=torch.float64, device="cuda")
    for s, p in enumerate(prompts):
        x = W["embed"][torch.tensor(p + [row[s] for row in steps], device="cuda")]
        for i, jl in enumerate(cfg["layers"]):
            q = "l%d." % i
            h = _exact_attention(_ln(x, W[q + "norm1"], W[q + "norm1.b"]), W, q + "mix.", jl)
            x = x + cfg["residual_mult"] * W[q + "ls1"] * _ln(h, W[q + "norm1b"], W[q + "norm1b.b"])
            h = torch.relu(_ln(x, W[q + "norm2"], W[q + "norm2.b"]) @ W[q + "mlp.up"].T) ** 2 @ W[q + "mlp.down"].T
            x = x + cfg["residual_mult"] * W[q + "ls2"] * _ln(h, W[q + "norm2b"], W[q + "norm2b.b"])
        out[:, s] = _ln(x[len(p) - 1:], W["final.norm"], W["final.norm.b"]) @ W["head"].T
    return out
