#!/usr/bin/env python
"""Generate the committed golden fixtures by RUNNING THE COMPILED REFERENCE (oracle/_ref, built by oracle/Makefile
from its sources).  Run only where those are; the outputs are
committed so that every test can check the oracle -- and the CUDA path -- against what the reference produced.

  python tests/golden/make_goldens.py

Writes, under tests/golden/:
  tiny_{q8_0,q4_0,q4_k}.gguf    2-layer llama-arch GQA models (random init, quantised by the reference `quantize --pure`)
  kernels.npz                   K1-K3: reference weight blocks, activation blocks, dequantised rows, mul_mat results
  decode_<type>.script / .logits.bin / .kv.txt    R2/R6: a llama.h call trace and what the reference returned
  kvops.script / kvops.kv.txt   R6: 400 random KV ops replayed through the reference's llama_kv_cache_seq_* wrappers
  speculative_q8_0.json         S1-S6: token ids generated by the reference `speculative` under the mini-MPI shim
                                (3 ranks) and by `main` (1 rank) on the same model
"""
import json
import os
import re
import subprocess
import sys

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.abspath(os.path.join(HERE, "..", ".."))
sys.path.insert(0, ROOT)
from oracle import oracle_py as op  # noqa: E402

REF = os.path.join(ROOT, "oracle", "_ref")
TINY = dict(n_layer=2, n_embd=256, n_head=4, n_head_kv=2, n_ff=256, n_vocab=384)
N_CTX, MAX_SEQ = 48, 8


def make_models():
    for q in ("q8_0", "q4_0", "q4_k"):
        out = os.path.join(HERE, "tiny_%s.gguf" % q)
        subprocess.run([sys.executable, os.path.join(ROOT, "tools", "make_gguf.py"), "--out", out,
                        "--n-layer", str(TINY["n_layer"]), "--n-embd", str(TINY["n_embd"]),
                        "--n-head", str(TINY["n_head"]), "--n-head-kv", str(TINY["n_head_kv"]),
                        "--n-ff", str(TINY["n_ff"]), "--n-vocab", str(TINY["n_vocab"]),
                        "--quant", q, "--flavour", "bigram", "--eps", "1.0", "--seed", "4321"], check=True)
    # a 1-layer draft for the speculative golden
    subprocess.run([sys.executable, os.path.join(ROOT, "tools", "make_gguf.py"), "--out",
                    os.path.join(HERE, "tiny_draft_q8_0.gguf"), "--n-layer", "1", "--n-embd", "128", "--n-head", "2",
                    "--n-head-kv", "2", "--n-ff", "256", "--n-vocab", str(TINY["n_vocab"]), "--quant", "q8_0",
                    "--flavour", "bigram", "--eps", "1.0", "--seed", "777", "--agree", "0.7"], check=True)


def kernel_goldens():
    r = op.Ref()
    rng = np.random.default_rng(2024)
    out = {}
    for name, wt in op.TYPE_NAMES.items():
        N, K, b = 12, 512, 5
        w = (rng.standard_normal((N, K)) * 0.04).astype(np.float32)
        x = (rng.standard_normal((b, K)) * 2.0).astype(np.float32)
        x[1, 32:64] = 0.0            # an all-zero Q8_0 block (id = 0 branch)
        x[2, 0:256] = 0.0            # an all-zero Q8_K super-block (d = 0 branch)
        x[3] *= 1e-3
        x[4, 7] = 300.0              # one outlier: every other value of its block rounds towards 0
        wq = r.quantize_weights(wt, w)
        out[name + "_w"] = wq
        out[name + "_x"] = x
        out[name + "_act"] = r.quantize_act(wt, x)
        out[name + "_deq"] = r.dequantize(wt, wq, K)
        out[name + "_y"] = r.mul_mat(wt, wq, x)
    # the test-quantize-fns data pattern (tests/test-quantize-fns.cpp:26-30): 0.1 + 2*cos(i + offset)
    n = 4096
    a = (0.1 + 2.0 * np.cos(np.arange(n, dtype=np.float32) + 0.0)).astype(np.float32)
    bvec = (0.1 + 2.0 * np.cos(np.arange(n, dtype=np.float32) + 1.0)).astype(np.float32)
    for name, wt in op.TYPE_NAMES.items():
        wq = r.quantize_weights(wt, a[None, :])
        out["cos_" + name + "_y"] = r.mul_mat(wt, wq, bvec[None, :])
        out["cos_" + name + "_w"] = wq
    out["cos_a"], out["cos_b"] = a, bvec
    np.savez_compressed(os.path.join(HERE, "kernels.npz"), **out)


def decode_script(n_vocab, seed):
    rng = np.random.default_rng(seed)
    allseq = list(range(MAX_SEQ))
    ops = []
    ops.append(("D", rng.integers(3, n_vocab, 7).tolist(), list(range(7)), [allseq] * 7))
    ops.append(("KV",))
    ops += [("RM", 1, 7, -1), ("RM", 2, 7, -1)]
    ops.append(("D", rng.integers(3, n_vocab, 5).tolist(), [7, 8, 9, 8, 9], [[1, 2], [1], [1], [2], [2]]))
    ops.append(("KV",))
    ops += [("RM", 2, 8, -1), ("CP", 1, 0, 7, 9), ("RM", 1, 9, -1), ("KV",)]
    for i in range(1, MAX_SEQ):
        ops += [("RM", i, 7, 9), ("CP", 0, i, 7, 9)]
    ops.append(("KV",))
    ops.append(("D", rng.integers(3, n_vocab, 1).tolist(), [9], [[0]]))
    ops += [("KEEP", 0), ("KV",)]
    ops.append(("D", rng.integers(3, n_vocab, 3).tolist(), [10, 11, 12], [[0, 3], [0, 3], [3]]))
    ops.append(("KV",))
    # a 16-token verification batch, then fill the cache until there is no slot left (rc = -1 in this fork)
    ops.append(("D", rng.integers(3, n_vocab, 16).tolist(), list(range(13, 29)), [[0]] * 16))
    ops.append(("KV",))
    ops.append(("D", rng.integers(3, n_vocab, 16).tolist(), list(range(29, 45)), [[0]] * 16))
    ops.append(("D", rng.integers(3, n_vocab, 8).tolist(), list(range(45, 53)), [[0]] * 8))
    ops.append(("KV",))
    ops += [("RM", 0, 20, 30), ("KV",)]
    ops.append(("D", rng.integers(3, n_vocab, 4).tolist(), [20, 21, 22, 23], [[0], [0], [0, 5], [5]]))
    ops.append(("KV",))
    return ops


def kvops_script(seed, n_ops=400):
    rng = np.random.default_rng(seed)
    ops = []
    pos_next = 0
    for _ in range(n_ops):
        c = rng.integers(0, 10)
        if c < 3:
            n = int(rng.integers(1, 6))
            seqs = [sorted(set(rng.integers(0, MAX_SEQ, int(rng.integers(1, 4))).tolist())) for _ in range(n)]
            ops.append(("D", rng.integers(3, TINY["n_vocab"], n).tolist(), [pos_next + i for i in range(n)], seqs))
            pos_next += n
        elif c < 6:
            p0 = int(rng.integers(-1, max(pos_next, 1)))
            p1 = int(rng.integers(-1, max(pos_next, 1) + 2))
            ops.append(("RM", int(rng.integers(-1, MAX_SEQ)), p0, p1))
        elif c < 9:
            p0 = int(rng.integers(-1, max(pos_next, 1)))
            p1 = int(rng.integers(-1, max(pos_next, 1) + 2))
            ops.append(("CP", int(rng.integers(0, MAX_SEQ)), int(rng.integers(0, MAX_SEQ)), p0, p1))
        else:
            ops.append(("KEEP", int(rng.integers(0, MAX_SEQ))))
        ops.append(("KV",))
        if pos_next > 36:
            ops.append(("RM", -1, -1, -1))
            pos_next = 0
    return ops


def write_script(path, ops):
    with open(path, "w") as f:
        for o in ops:
            if o[0] == "D":
                f.write("D %d\n" % len(o[1]))
                for t, p, s in zip(o[1], o[2], o[3]):
                    f.write("%d %d %d %s\n" % (t, p, len(s), " ".join(map(str, s))))
            else:
                f.write(" ".join(map(str, o)) + "\n")


def run_ref(model, script, prefix, n_ctx=N_CTX, max_seq=MAX_SEQ, threads=2):
    subprocess.run([os.path.join(REF, "ref_decode_dump"), model, str(n_ctx), str(max_seq), script, prefix, str(threads)],
                   check=True, stdout=subprocess.DEVNULL, stderr=subprocess.DEVNULL)


def decode_goldens():
    for i, q in enumerate(("q8_0", "q4_0", "q4_k")):
        script = os.path.join(HERE, "decode_%s.script" % q)
        write_script(script, decode_script(TINY["n_vocab"], 100 + i))
        run_ref(os.path.join(HERE, "tiny_%s.gguf" % q), script, os.path.join(HERE, "decode_%s" % q))
    script = os.path.join(HERE, "kvops.script")
    write_script(script, kvops_script(5))
    run_ref(os.path.join(HERE, "tiny_q8_0.gguf"), script, os.path.join(HERE, "kvops"))
    os.unlink(os.path.join(HERE, "kvops.logits.bin"))     # only the bookkeeping is pinned by this one


FALCON = {   # name: (quant, n_head_kv, second norm) -- 7B layout (MQA, one norm) and 40B/180B layout (8 KV heads there, two norms)
    "falcon_q4_0": ("q4_0", 1, False),
    "falcon40_q8_0": ("q8_0", 2, True),
}


def falcon_goldens():
    """falcon architecture (build_falcon, llama.cpp:4106): LayerNorm + bias, NeoX RoPE, fused QKV, GELU MLP in parallel
    with attention.  Same call trace as the llama fixtures; the reference decides what the logits are."""
    for i, (name, (q, hkv, norm2)) in enumerate(FALCON.items()):
        out = os.path.join(HERE, "tiny_%s.gguf" % name)
        subprocess.run([sys.executable, os.path.join(ROOT, "tools", "make_gguf.py"), "--arch", "falcon", "--out", out,
                        "--n-layer", "2", "--n-embd", "256", "--n-head", "4", "--n-head-kv", str(hkv), "--n-ff", "1024",
                        "--n-vocab", str(TINY["n_vocab"]), "--quant", q, "--flavour", "bigram", "--eps", "1.0",
                        "--seed", str(9000 + i)] + (["--norm2"] if norm2 else []), check=True)
        script = os.path.join(HERE, "decode_%s.script" % name)
        write_script(script, decode_script(TINY["n_vocab"], 200 + i))
        run_ref(out, script, os.path.join(HERE, "decode_%s" % name))


def q6k_goldens():
    """Q6_K / Q5_K (output.weight, attn_v, ffn_down of Q4_K_M files): reference quantiser, dequantiser and dot product"""
    for wt, fname, seed in ((op.TYPE_Q6_K, "kernels_q6k.npz", 2025), (op.TYPE_Q5_K, "kernels_q5k.npz", 2026), (op.TYPE_Q3_K, "kernels_q3k.npz", 2027)):
        _kquant_golden(wt, fname, seed)


def _kquant_golden(wt, fname, seed):
    r = op.Ref()
    rng = np.random.default_rng(seed)
    N, K, b = 12, 512, 5
    w = (rng.standard_normal((N, K)) * 0.04).astype(np.float32)
    x = (rng.standard_normal((b, K)) * 2.0).astype(np.float32)
    x[2, 0:256] = 0.0
    x[4, 7] = 300.0
    wq = r.quantize_weights(wt, w)
    np.savez_compressed(os.path.join(HERE, fname), w=wq, x=x, act=r.quantize_act(wt, x), deq=r.dequantize(wt, wq, K),
                        y=r.mul_mat(wt, wq, x))


def q4km_goldens():
    """a Q4_K_M file as the reference's quantize makes it (Q4_K + Q6_K tensors in one model) and its decode trace"""
    out = os.path.join(HERE, "tiny_q4_k_m.gguf")
    subprocess.run([sys.executable, os.path.join(ROOT, "tools", "make_gguf.py"), "--out", out, "--n-layer", "4", "--n-embd", "256",
                    "--n-head", "4", "--n-head-kv", "2", "--n-ff", "512", "--n-vocab", str(TINY["n_vocab"]), "--quant", "q4_k_m",
                    "--flavour", "bigram", "--eps", "1.0", "--seed", "4444"], check=True)
    script = os.path.join(HERE, "decode_q4_k_m.script")
    write_script(script, decode_script(TINY["n_vocab"], 400))
    run_ref(out, script, os.path.join(HERE, "decode_q4_k_m"))
    # Q4_K_S: attn_v and ffn_down of the first layers in Q5_K (llama.cpp:7925, 7950-7957) -- the type 70B-class Q4_K_M files
    # keep attn_v in (:7927-7933 applies to MODEL_70B only, which a small fixture cannot be)
    out = os.path.join(HERE, "tiny_q4_k_s.gguf")
    subprocess.run([sys.executable, os.path.join(ROOT, "tools", "make_gguf.py"), "--out", out, "--n-layer", "4", "--n-embd", "256",
                    "--n-head", "4", "--n-head-kv", "2", "--n-ff", "512", "--n-vocab", str(TINY["n_vocab"]), "--quant", "q4_k_s",
                    "--flavour", "bigram", "--eps", "1.0", "--seed", "4445"], check=True)
    script = os.path.join(HERE, "decode_q4_k_s.script")
    write_script(script, decode_script(TINY["n_vocab"], 401))
    run_ref(out, script, os.path.join(HERE, "decode_q4_k_s"))


def q3km_goldens():
    """a Q3_K_M file as the reference's quantize makes it -- the type of the authors' 70B target (scripts/dolphin_tinyllama_8_nodes.sh):
    token_embd, attn_q / attn_k, ffn_gate / ffn_up in Q3_K, attn_v / attn_output / ffn_down in Q4_K or Q5_K, output.weight in Q6_K
    (llama.cpp:7900-7970) -- and its decode trace"""
    out = os.path.join(HERE, "tiny_q3_k_m.gguf")
    subprocess.run([sys.executable, os.path.join(ROOT, "tools", "make_gguf.py"), "--out", out, "--n-layer", "4", "--n-embd", "256",
                    "--n-head", "4", "--n-head-kv", "2", "--n-ff", "512", "--n-vocab", str(TINY["n_vocab"]), "--quant", "q3_k_m",
                    "--flavour", "bigram", "--eps", "1.0", "--seed", "4446"], check=True)
    script = os.path.join(HERE, "decode_q3_k_m.script")
    write_script(script, decode_script(TINY["n_vocab"], 402))
    run_ref(out, script, os.path.join(HERE, "decode_q3_k_m"))


def q56_goldens():
    """files whose token embedding is Q5_K (Q5_K_M: Q5_K + Q6_K tensors) and Q6_K (pure Q6_K), and their decode traces"""
    for quant, seed, sseed in (("q5_k_m", "4447", 403), ("q6_k", "4448", 404)):
        out = os.path.join(HERE, "tiny_%s.gguf" % quant)
        subprocess.run([sys.executable, os.path.join(ROOT, "tools", "make_gguf.py"), "--out", out, "--n-layer", "4", "--n-embd", "256",
                        "--n-head", "4", "--n-head-kv", "2", "--n-ff", "512", "--n-vocab", str(TINY["n_vocab"]), "--quant", quant,
                        "--flavour", "bigram", "--eps", "1.0", "--seed", seed], check=True)
        script = os.path.join(HERE, "decode_%s.script" % quant)
        write_script(script, decode_script(TINY["n_vocab"], sseed))
        run_ref(out, script, os.path.join(HERE, "decode_%s" % quant))


# ---- fixtures at the shapes the benchmark runs (head_dim 128, grouped-query attention, long caches, 94-word sequence sets) ----
WIDE = {   # name: (quant, n_embd, n_head, n_head_kv, n_ff): head_dim 128; group 8 (the 70B / 120B layout) and group 1 (7B)
    "wide_q4_k": ("q4_k", 1024, 8, 1, 512),
    "wide_q4_0": ("q4_0", 512, 4, 4, 512),
}
WIDE_MAX_SEQ = 3002        # -np 3: 1000 partitions of 3 ids + seq 0 + 1 (speculative.cpp:140-145) -> 94 words per cell


def wide_script(n_vocab, seed, n_prompt=208):
    """what a PipeInfer run does to the cache, at benchmark-like sizes: a long prompt in one batch (13 chunks of 16 here),
    partitions seeded from sequence 0, three speculative tree batches in partitions that live in different words of the
    sequence set, the commit sweep, a non-speculative token, a 16-token batch, and a second round on top of 290 cells."""
    rng = np.random.default_rng(seed)
    tok = lambda n: rng.integers(3, n_vocab, n).tolist()
    parts = [(1, 2, 3), (1501, 1502, 1503), (2998, 2999, 3000)]
    ops = [("D", tok(n_prompt), list(range(n_prompt)), [[0]] * n_prompt), ("KV",)]
    P = n_prompt
    for a, b, c in parts:
        for i in (a, b, c):
            ops.append(("CP", 0, i, -1, -1))
    ops.append(("KV",))
    a, b, c = parts[0]      # 5-token tree: trunk, two branches
    ops.append(("D", tok(5), [P, P + 1, P + 2, P + 1, P + 2], [[a, b, c], [a, b], [a], [c], [c]]))
    a, b, c = parts[1]      # 6 tokens, three branches off the first token
    ops.append(("D", tok(6), [P, P + 1, P + 2, P + 1, P + 1, P + 2], [[a, b, c], [a], [a], [b], [c], [c]]))
    a, b, c = parts[2]      # 9 tokens (two n-tiles in the matmul), a chain with one side branch
    ops.append(("D", tok(9), [P + i for i in range(8)] + [P + 3], [[a, b]] * 3 + [[a]] * 5 + [[b]]))
    ops.append(("KV",))
    # commit partition 0's trunk to sequence 0 and sweep it to every id in use (speculative.cpp:420-470, 603-612)
    ops += [("RM", 0, P, -1), ("CP", parts[0][0], 0, P, P + 3)]
    for pa in parts:
        for i in pa:
            ops += [("RM", i, P, -1), ("CP", 0, i, -1, -1)]
    ops.append(("KV",))
    P += 3
    ops.append(("D", tok(1), [P], [[0]]))                                   # the non-speculative run
    ops.append(("D", tok(16), list(range(P + 1, P + 17)), [[0]] * 16))
    P += 17
    ops.append(("D", tok(64), list(range(P, P + 64)), [[0, 1502, 3000]] * 64))       # four more chunks, ids in three words
    P += 64
    ops.append(("KV",))
    ops.append(("D", tok(4), [P, P + 1, P + 1, P + 2], [[1502, 3000], [1502], [3000], [3000]]))
    ops.append(("D", tok(2), [P, P + 1], [[0], [0]]))
    ops.append(("KV",))
    return ops


def wide_goldens():
    for i, (name, (q, E, H, HKV, FF)) in enumerate(WIDE.items()):
        out = os.path.join(HERE, "%s.gguf" % name)
        subprocess.run([sys.executable, os.path.join(ROOT, "tools", "make_gguf.py"), "--out", out, "--n-layer", "2",
                        "--n-embd", str(E), "--n-head", str(H), "--n-head-kv", str(HKV), "--n-ff", str(FF),
                        "--n-vocab", str(TINY["n_vocab"]), "--quant", q, "--flavour", "bigram", "--eps", "3.0",
                        "--seed", str(6100 + i)], check=True)
        script = os.path.join(HERE, "decode_%s.script" % name)
        write_script(script, wide_script(TINY["n_vocab"], 600 + i))
        run_ref(out, script, os.path.join(HERE, "decode_%s" % name), n_ctx=1024, max_seq=WIDE_MAX_SEQ, threads=4)
    # the same grouped-query model with a 6144-cell cache and 300 + cells in use: the long-context attention path
    script = os.path.join(HERE, "decode_wide_long.script")
    rng = np.random.default_rng(650)
    nv = TINY["n_vocab"]
    ops = [("D", rng.integers(3, nv, 300).tolist(), list(range(300)), [[0, 1, 2]] * 300), ("KV",),
           ("D", rng.integers(3, nv, 5).tolist(), [300, 301, 302, 301, 302], [[1, 2], [1], [1], [2], [2]]),
           ("RM", 2, 300, -1), ("CP", 1, 0, 300, 303), ("KV",),
           ("D", rng.integers(3, nv, 16).tolist(), list(range(303, 319)), [[0]] * 16), ("KV",)]
    write_script(script, ops)
    run_ref(os.path.join(HERE, "wide_q4_k.gguf"), script, os.path.join(HERE, "decode_wide_long"), n_ctx=6144, max_seq=8, threads=4)


# ---- the one-GPU 1.1B model at its real shape: TinyLlama-1.1B architecture, Q8_0 (1.17 GB: not committed; tools/make_gguf.py
# --direct regenerates it bit for bit from the seed, the sha256 of the file is part of the fixture) ----
C1 = dict(n_layer=22, n_embd=2048, n_head=32, n_head_kv=4, n_ff=5632, n_vocab=32000, quant="q8_0", seed=11,
          emb_scale=0.05)     # embedding / output rows of std 0.05: logits of a realistic size (std ~2), every layer matters


def c1_model(path):
    subprocess.run([sys.executable, os.path.join(ROOT, "tools", "make_gguf.py"), "--direct", "--out", path,
                    "--n-layer", str(C1["n_layer"]), "--n-embd", str(C1["n_embd"]), "--n-head", str(C1["n_head"]),
                    "--n-head-kv", str(C1["n_head_kv"]), "--n-ff", str(C1["n_ff"]), "--n-vocab", str(C1["n_vocab"]),
                    "--quant", C1["quant"], "--seed", str(C1["seed"]), "--emb-scale", str(C1["emb_scale"])], check=True)


def file_sha256(path):
    import hashlib
    h = hashlib.sha256()
    with open(path, "rb") as f:
        for blk in iter(lambda: f.read(1 << 24), b""):
            h.update(blk)
    return h.hexdigest()


def c1_script():
    rng = np.random.default_rng(1100)
    nv = C1["n_vocab"]
    tok = lambda n: rng.integers(3, nv, n).tolist()
    return [("D", tok(6), list(range(6)), [[0, 1, 2]] * 6), ("D", tok(1), [6], [[0]]),
            ("D", tok(3), [6, 7, 7], [[1, 2], [1], [2]]), ("RM", 2, 6, -1), ("CP", 1, 0, 6, 8), ("KV",),
            ("D", tok(1), [8], [[0]]), ("D", tok(2), [9, 10], [[0], [0]]), ("D", tok(1), [11], [[0]]),
            ("CP", 0, 3, -1, -1), ("D", tok(4), [12, 13, 14, 13], [[0, 3], [0], [0], [3]]), ("D", tok(1), [15], [[0]]), ("KV",)]


def c1_goldens():
    path = "/tmp/pib_c1_tinyllama_q8_0.gguf"
    c1_model(path)
    script = os.path.join(HERE, "decode_c1_tinyllama_q8_0.script")
    write_script(script, c1_script())
    run_ref(path, script, os.path.join(HERE, "decode_c1_tinyllama_q8_0"), n_ctx=64, max_seq=8, threads=8)
    json.dump({"sha256": file_sha256(path), "bytes": os.path.getsize(path), "shape": C1},
              open(os.path.join(HERE, "c1_tinyllama_q8_0.json"), "w"), indent=1)
    os.unlink(path)


def speculative_golden(target="tiny_q8_0.gguf", out="speculative_q8_0.json"):
    prompt = "the quick brown fox"
    pf = os.path.join(HERE, "prompt.txt")
    open(pf, "w").write(prompt)
    tgt = os.path.join(HERE, target)
    dft = os.path.join(HERE, "tiny_draft_q8_0.gguf")
    common = ["-f", pf, "-n", "24", "-c", "256", "--temp", "-1", "--repeat-last-n", "0", "--ignore-eos", "-t", "2"]
    r = subprocess.run([os.path.join(REF, "main"), "-m", tgt] + common, stdout=subprocess.PIPE, stderr=subprocess.DEVNULL)
    main_text = r.stdout.decode("utf-8", "replace")
    pre = "/tmp/pib_spec_golden"
    subprocess.run([os.path.join(REF, "mpirun_shim"), "-np", "3", "--timeout", "120", "--out-prefix", pre,
                    os.path.join(REF, "speculative"), "-m", tgt, "-md", dft] + common +
                   ["--draft", "4", "-np", "1", "--mpi-layer-split", "0.5,0.5/1.0"], check=True)
    spec_text = open(pre + ".0.out", "rb").read().decode("utf-8", "replace")
    err = open(pre + ".0.err", "rb").read().decode("utf-8", "replace")
    stats = {k: float(v) for k, v in re.findall(r"(n_predict|n_drafted|n_accept)\s*=\s*([0-9.]+)", err)}
    json.dump({"prompt": prompt, "main_text": main_text, "speculative_text": spec_text, "stats": stats,
               "args": common + ["--draft", "4", "-np", "1", "--mpi-layer-split", "0.5,0.5/1.0"]},
              open(os.path.join(HERE, out), "w"), indent=1)
    os.unlink(pf)


if __name__ == "__main__":
    op.build(ref=True)
    if sys.argv[1:] == ["q4km"]:
        q4km_goldens()
        sys.exit(0)
    if sys.argv[1:] == ["q6k"]:
        q6k_goldens()
        sys.exit(0)
    if sys.argv[1:] == ["q3k"]:
        _kquant_golden(op.TYPE_Q3_K, "kernels_q3k.npz", 2027)
        q3km_goldens()
        speculative_golden("tiny_q3_k_m.gguf", "speculative_q3_k_m.json")        # the authors' program on the authors' file type
        sys.exit(0)
    if sys.argv[1:] == ["q56"]:
        q56_goldens()
        sys.exit(0)
    if sys.argv[1:] == ["falcon"]:
        falcon_goldens()
        sys.exit(0)
    if sys.argv[1:] == ["wide"]:
        wide_goldens()
        sys.exit(0)
    if sys.argv[1:] == ["c1"]:
        c1_goldens()
        sys.exit(0)
    make_models()
    kernel_goldens()
    decode_goldens()
    speculative_golden()
    speculative_golden("tiny_q3_k_m.gguf", "speculative_q3_k_m.json")
    falcon_goldens()
    q6k_goldens()
    q4km_goldens()
    q3km_goldens()
    q56_goldens()
    wide_goldens()
    c1_goldens()
    print("goldens written to", HERE)
