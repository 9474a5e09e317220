"""RoPE, KV store and attention of a decode batch (csrc/attention.cu) against the reference's order of operations restated in numpy, bit for bit: cells left over behind
the last multiple of 32, rounds of cells held in registers or not, value rows staged in shared memory or not, the batch's cells at the end of the range, inside it and on
both sides of the staged rows, masked cells that hold anything."""
import ctypes as C
import ctypes.util

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOK, POS, MAXB = 64, 128, 16                       # offsets of a descriptor's tokens and positions (csrc/desc.cuh)


@pytest.fixture(scope="module")
def fn():
    from pipeinfer_b200 import lib as pib
    L = pib.load()
    L.init(0)
    f = L.L._Z13pib_attentionPKfS0_PKhPK6float2iiP6__halfS7_S2_PKiiiiiiPfS9_P11CUstream_st
    f.argtypes = [C.c_void_p] * 4 + [C.c_int] * 2 + [C.c_void_p] * 4 + [C.c_int] * 5 + [C.c_void_p] * 3
    return L, f


@pytest.fixture(scope="module")
def exp16():
    """fp16(expf(x)) of every fp16 x with the host's expf, the reference's table"""
    m = C.CDLL(ctypes.util.find_library("m"))
    m.expf.restype, m.expf.argtypes = C.c_float, [C.c_float]
    x = np.arange(65536, dtype=np.uint16).view(np.float16).astype(np.float32)
    with np.errstate(over="ignore"):
        return np.array([m.expf(v) for v in x.tolist()], np.float32).astype(np.float16)


def fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c.astype(np.float64)).astype(np.float32)


def tree(acc):
    """[..., 32] partial sums -> ((0 + 2) + (1 + 3)) over the vectors of eight, halves, two horizontal additions; fp32"""
    v = acc.reshape(acc.shape[:-1] + (4, 8))
    r = (v[..., 0, :] + v[..., 2, :]) + (v[..., 1, :] + v[..., 3, :])
    t = r[..., :4] + r[..., 4:]
    return (t[..., 0] + t[..., 1]) + (t[..., 2] + t[..., 3])


def one_head(q, K, V, seen, scale, exp16):
    n, hd = K.shape
    acc = np.zeros((n, 32), np.float32)
    for st in range(0, hd, 32):
        acc = fma(K[:, st:st + 32], q[None, st:st + 32], acc)
    s = np.where(seen, tree(acc) * scale, np.float32(-np.inf)).astype(np.float32)
    e = np.where(seen, exp16[(s - s.max()).astype(np.float16).view(np.uint16)].astype(np.float32), np.float32(0))
    inv = np.float32(1.0 / e.astype(np.float64).sum())
    p = (e * inv).astype(np.float16).astype(np.float32)
    V = np.where((p == 0)[:, None], np.float32(0), V)
    acc, n32 = np.zeros((32, hd), np.float32), n & ~31
    for c in range(0, n32, 32):
        acc = fma(V[c:c + 32], p[c:c + 32, None], acc)
    o = tree(acc.T).astype(np.float64)
    for c in range(n32, n):
        o = o + (V[c] * p[c]).astype(np.float64)
    return o.astype(np.float32)


@pytest.mark.parametrize("hd,H,G,n,b,cell0,n_ctx", [
    (64, 4, 2, 32, 1, 31, 64), (64, 4, 1, 33, 3, 20, 512), (64, 8, 2, 63, 16, 40, 512), (64, 4, 4, 257, 2, 255, 512), (64, 4, 1, 300, 1, 299, 512), (64, 4, 2, 511, 4, 100, 512),
    (64, 4, 1, 513, 1, 512, 1024), (64, 2, 1, 705, 3, 702, 1024), (64, 2, 1, 736, 2, 734, 1024), (64, 2, 2, 930, 5, 700, 1000), (64, 2, 1, 1100, 2, 300, 1301), (64, 2, 2, 420, 2, 390, 3400),
    (128, 2, 1, 32, 1, 30, 64), (128, 4, 4, 129, 2, 127, 256), (128, 2, 1, 300, 1, 299, 512), (128, 2, 2, 385, 3, 382, 512), (128, 2, 1, 700, 2, 200, 1024),
    (128, 32, 4, 95, 16, 79, 256), (128, 32, 4, 290, 8, 250, 512), (128, 16, 4, 415, 16, 380, 640)])      # from 149 (head, token) pairs on 256 threads
@pytest.mark.parametrize("mode,sep", [(0, False), (2, True)])
def test_decode_attention_bits(fn, exp16, hd, H, G, n, b, cell0, n_ctx, mode, sep):
    L, f = fn
    rng = np.random.default_rng(n * 31 + hd + b)
    E, GQA = H * hd, G * hd
    rows = rng.standard_normal((b, E + 2 * GQA)).astype(np.float32) * np.float32(1.5)
    kc, vc = rng.standard_normal((n_ctx, GQA)).astype(np.float16), rng.standard_normal((n_ctx, GQA)).astype(np.float16)
    pos = rng.integers(0, 900, b).astype(np.int32)
    ang = rng.uniform(0, 6.28, (964, hd // 2))
    rope = np.stack([np.cos(ang), np.sin(ang)], -1).astype(np.float32)
    seen = rng.random((b, n)) < 0.8
    seen[:, cell0:cell0 + b] = np.tril(np.ones((b, b), bool))
    hidden = [c for c in (0, n // 2, n - 1) if not cell0 <= c < cell0 + b]
    seen[:, hidden] = False
    kc[hidden], vc[hidden] = np.nan, np.inf                         # cells no row sees hold anything
    desc = np.zeros(8192, np.uint8)
    desc[:8].view(np.int32)[:] = (b, cell0)
    desc[POS:POS + 4 * b].view(np.int32)[:] = pos
    mask = np.ones((b, n_ctx), np.uint8)
    mask[:, :n] = ~seen
    dev = [L.to_device(a) for a in (rows[:, :E + GQA].copy() if sep else rows, rows[:, E + GQA:].copy(), desc, rope, kc, vc, mask, np.array([0, 0, n], np.int32), np.full((b, E), np.nan, np.float32))]
    q, v, dd, rp, kd, vd, md, sc, out = dev
    L.check(f(q, v if sep else None, dd, rp, 964, mode, kd, vd, md, sc, b, H, G, hd, n_ctx, out, None, None))
    L.check(L.L.pib_stream_sync(None))

    def rotate(x):                                                   # [b][heads][hd] -> fp16, unfused multiplies
        y, cs = np.empty(x.shape, np.float16), rope[pos][:, None]
        i0, i1 = (slice(0, hd // 2), slice(hd // 2, hd)) if mode & 2 else (slice(0, hd, 2), slice(1, hd, 2))
        y[..., i0] = x[..., i0] * cs[..., 0] - x[..., i1] * cs[..., 1]
        y[..., i1] = x[..., i0] * cs[..., 1] + x[..., i1] * cs[..., 0]
        return y
    Q = rotate(rows[:, :E].reshape(b, H, hd)).astype(np.float32)
    kc[cell0:cell0 + b] = rotate(rows[:, E:E + GQA].reshape(b, G, hd)).reshape(b, GQA)
    vc[cell0:cell0 + b] = rows[:, E + GQA:].astype(np.float16)
    K, V = kc.astype(np.float32).reshape(n_ctx, G, hd), vc.astype(np.float32).reshape(n_ctx, G, hd)
    scale = np.float32(1.0) / np.sqrt(np.float32(hd))
    with np.errstate(invalid="ignore"):
        want = np.stack([np.concatenate([one_head(Q[t, h], K[:n, h // (H // G)], V[:n, h // (H // G)], seen[t], scale, exp16) for h in range(H)]) for t in range(b)])
    got = L.to_host(out, (b, E), np.float32)
    gk, gv = L.to_host(kd, (n_ctx, GQA), np.float16), L.to_host(vd, (n_ctx, GQA), np.float16)
    for d in dev:
        L.L.pib_dev_free(d)
    assert np.array_equal(gk, kc, equal_nan=True) and np.array_equal(gv, vc, equal_nan=True)
    assert np.array_equal(got, want)
