"""RoPE + KV store and attention of a wide prompt pass (csrc/prompt_attn.cu) against float64, at the edges of its tiles: row and cell remainders, grouped heads,
contexts whose mask rows are not 16-byte aligned, cells no row sees (holding anything, infinities included), a value that is infinite for some rows only."""
import ctypes as C
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def fn():
    from pipeinfer_b200 import lib as pib
    L = pib.load()
    L.init(0)
    names = subprocess.run(["nm", "-D", "--defined-only", pib.SO_PATH], capture_output=True, text=True, check=True).stdout.split()
    f = getattr(L.L, next(n for n in names if "pib_prompt_attentionPK" in n))
    f.argtypes = [C.c_void_p] * 4 + [C.c_int] + [C.c_void_p] * 5 + [C.c_int] * 5 + [C.c_void_p] * 3
    return L, f


@pytest.mark.parametrize("T,H,G,hd,n_ctx,past,odd", [(1, 2, 2, 128, 64, 0, 0), (33, 4, 2, 64, 96, 0, 0), (64, 2, 1, 128, 200, 63, 0), (65, 3, 3, 64, 301, 40, 0), (256, 4, 1, 128, 700, 129, 0),
                                                     (255, 2, 2, 64, 1023, 700, 0), (70, 2, 1, 128, 256, 64, 1), (90, 4, 2, 64, 333, 100, 1)])
def test_prompt_attention(fn, T, H, G, hd, n_ctx, past, odd):
    L, f = fn
    rng = np.random.default_rng(T * 7 + hd + n_ctx)
    E, GQA, n = H * hd, G * hd, min(n_ctx, (past + T + 31) // 32 * 32)
    qkv = rng.standard_normal((T, E + 2 * GQA)).astype(np.float32) * 2
    pos = np.arange(past, past + T, dtype=np.int32)
    cell = pos.copy()
    kc = rng.standard_normal((n_ctx, GQA)).astype(np.float16)
    vc = rng.standard_normal((n_ctx, GQA)).astype(np.float16)
    ang = rng.uniform(0, 6.28, (n_ctx + 64, hd // 2))
    rope = np.stack([np.cos(ang), np.sin(ang)], -1).astype(np.float32)
    seen = np.arange(n_ctx)[None, :] <= pos[:, None]
    seen[:, :past] &= rng.random((T, past)) < 0.7
    if past > 3:
        seen[:, past // 3] = False                                   # a cell of another sequence, holding anything
        kc[past // 3], vc[past // 3] = np.nan, np.inf
    kc[past + T:], vc[past + T:] = np.inf, np.nan
    if odd:                                                          # infinite for the rows that see it, nothing for the others
        vc[past // 2, ::3] = np.inf
        seen[:, past // 2] = np.arange(T) % 5 == 0
    mask = (~seen).astype(np.uint8)
    scal = np.array([0, 0, n, n_ctx], np.int32)
    d = {k: L.to_device(v) for k, v in dict(qkv=qkv, pos=pos, cell=cell, rope=rope, kc=kc, vc=vc, mask=mask, scal=scal).items()}
    q16, out = L.alloc(T * E * 2), L.alloc(T * E * 4)
    L.check(f(d["qkv"], d["pos"], d["cell"], d["rope"], n_ctx + 64, q16, d["kc"], d["vc"], d["mask"], d["scal"], T, H, G, hd, n_ctx, out, None, None))
    got = L.to_host(out, (T, E), np.float32).reshape(T, H, hd)
    kd, vd = L.to_host(d["kc"], kc.shape, np.float16), L.to_host(d["vc"], vc.shape, np.float16)

    def rot(x):                                                      # fp32 products and sums, rounded to fp16 once, as the decode path
        x0, x1, cs = x[..., 0::2], x[..., 1::2], rope[pos][:, None, :, :]
        o = np.empty(x.shape, np.float16)
        o[..., 0::2], o[..., 1::2] = x0 * cs[..., 0] - x1 * cs[..., 1], x0 * cs[..., 1] + x1 * cs[..., 0]
        return o
    q = rot(qkv[:, :E].reshape(T, H, hd))
    kc[past:past + T] = rot(qkv[:, E:E + GQA].reshape(T, G, hd)).reshape(T, GQA)
    vc[past:past + T] = qkv[:, E + GQA:].astype(np.float16)
    assert np.array_equal(kd.view(np.uint16), kc.view(np.uint16)) and np.array_equal(vd.view(np.uint16), vc.view(np.uint16))
    worst = 0.0
    with np.errstate(all="ignore"):
        for t in range(T):
            js = np.nonzero(seen[t, :n])[0]
            for h in range(H):
                k, v = (c[js, (h // (H // G)) * hd:(h // (H // G) + 1) * hd].astype(np.float64) for c in (kc, vc))
                s = (k @ q[t, h].astype(np.float64)) / np.sqrt(hd)
                p = np.exp(s - s.max())
                p /= p.sum()
                want = p @ v
                fin = np.isfinite(want)
                assert np.array_equal(fin, np.isfinite(got[t, h]))
                # weights rounded to fp16 (2^-11 of each, 2^-25 below its normal range), fp32 scores of size |s| before exp
                lim = (2.0 ** -11 + 2.0 ** -21 * (1 + np.abs(s).max())) * (p @ np.abs(v)) + 2.0 ** -24 * np.abs(v).sum(0)
                worst = max(worst, float((np.abs(got[t, h] - want) / lim)[fin].max(initial=0)))
    print("T %d H %d/%d hd %d: worst error %.3g of the bound" % (T, H, G, hd, worst))
    assert worst <= 1.0
    for p in list(d.values()) + [q16, out]:
        L.free(p)
