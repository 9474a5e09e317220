"""The Q4_K GEMM with weights in tensor memory (csrc/gemm_q4k_tc.cu) at the edges of its tiles and splits: rows that fill no 16-row tile, no accumulator or no
block, every token-block width, K shares of unequal length in a cluster.  Reference: float64 sums of the dequantised weights times
the quantised activations; both operands enter the product rounded to fp16, so the error of an output is below 2 * 2^-11 * sum |w x| (and far below in the mean)."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle_py as op
from tests.test_gpu_gemm import rand_q4k

pytestmark = pytest.mark.gpu


def reference(w, x):
    """float64 sums of the products, and the bound of an output's error"""
    (N, _), (b, K) = w.shape, x.shape
    blk = w.reshape(N, K // 256, 144).astype(np.int32)
    f16 = lambda at: w.reshape(N, K // 256, 144)[:, :, at:at + 2].copy().view(np.float16)[..., 0].astype(np.float64)
    s = blk[:, :, 4:16]
    sc = np.concatenate([s[..., 0:4] & 63, (s[..., 8:12] & 15) | ((s[..., 0:4] >> 6) << 4)], -1)
    mn = np.concatenate([s[..., 4:8] & 63, (s[..., 8:12] >> 4) | ((s[..., 4:8] >> 6) << 4)], -1)
    q = blk[:, :, 16:].reshape(N, K // 256, 4, 1, 32)
    q = np.concatenate([q & 15, q >> 4], 3).reshape(N, K // 256, 8, 32)
    W = ((f16(0)[..., None] * sc)[..., None] * q - (f16(2)[..., None] * mn)[..., None]).reshape(N, K)
    v = x.reshape(b, -1, 256)
    m = np.take_along_axis(v, np.abs(v).argmax(-1)[..., None], -1)
    iscale = np.float32(-128) / m
    X = (np.minimum(np.rint(iscale * v), 127).astype(np.float64) * (np.float32(1) / iscale).astype(np.float64)).reshape(b, K)
    return X @ W.T, 2.0 ** -10 * (np.abs(X) @ np.abs(W).T) + 1e-30


@pytest.mark.parametrize("N,K,b", [(1, 256, 1), (17, 512, 33), (129, 256, 97), (257, 1280, 129), (300, 2816, 64), (640, 3328, 65), (1000, 768, 193), (127, 1792, 32), (37900, 256, 40), (37999, 512, 64),
                                   (38000, 256, 20)])
def test_gemm_edges(oracle, N, K, b):
    from pipeinfer_b200 import load
    lib = load()
    lib.init(0)
    lib.L.pib_gemm_host.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]
    rng = np.random.default_rng(N * 3 + K + b)
    w, x = rand_q4k(rng, N, K), rng.standard_normal((b, K)).astype(np.float32)
    h = lib.weight_upload(op.TYPE_Q4_K, w, K)
    y = np.full((b, N), np.nan, np.float32)
    lib.check(lib.L.pib_gemm_host(h, x.ctypes.data, b, y.ctypes.data))
    lib.L.pib_weight_free(h)
    want, lim = reference(w, x)
    err = np.abs(y - want)
    print("N %d K %d b %d: worst error %.3g of the bound, mean %.2g" % (N, K, b, (err / lim).max(), (err / lim).mean()))
    assert np.isfinite(y).all() and (err <= lim).all() and (err / lim).mean() < 0.1


# every instance, <token columns, weight groups>; K shares in a cluster where there are few row blocks, a second launch for what is left of a round
@pytest.mark.parametrize("N,K,b", [(2048, 4096, 24), (4096, 4096, 24), (19200, 1024, 32),      # <32, 1>, two CTAs per SM
                                   (2048, 4096, 40), (19200, 1024, 64),                        # <64, 1>
                                   (19200, 1024, 90), (19200, 1024, 128),                      # <96, 1>, <128, 1>
                                   (10240, 2048, 17), (10240, 2048, 50),                       # <32, 2>, <64, 2>
                                   (10240, 2048, 96), (2048, 4096, 80), (1910, 4096, 80),      # <96, 2>, one share, four and eight (15 row blocks)
                                   (4220, 4096, 90), (4230, 4096, 90), (9460, 2048, 70), (9480, 2048, 70),      # 33 / 34 and 74 / 75 row blocks: four shares, two; two, one
                                   (10240, 2048, 128), (4096, 4096, 100),                      # <128, 2>, one share and four
                                   (10240, 2048, 188), (4096, 4096, 129), (19200, 1024, 180),  # <192, 2>, one share, four, a round and two blocks
                                   (10240, 2048, 250), (4096, 4096, 256)])                     # <256, 2>, one share and four
def test_calls_that_follow_one_another_give_the_same(N, K, b):
    """launches overlap their predecessors (programmatic launch), and a ring place is refilled while others are read: the same call over and over, never waited for, must
    leave the same bits each time, and the right ones"""
    from pipeinfer_b200 import load
    lib = load()
    lib.init(0)
    L = lib.L
    L.pib_gemm_scratch_bytes.restype, L.pib_gemm_scratch_bytes.argtypes = C.c_size_t, [C.c_int64, C.c_int]
    L.pib_gemm.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    L.pib_quantize_act_rows.argtypes = L.pib_quantize_act.argtypes
    rng = np.random.default_rng(N + b)
    blocks, xs = rand_q4k(rng, N, K), rng.standard_normal((b, K)).astype(np.float32)
    w, x = lib.weight_upload(op.TYPE_Q4_K, blocks, K), lib.to_device(xs)
    act, scr, n = lib.alloc(L.pib_act_bytes(op.TYPE_Q4_K, K, b)), lib.alloc(L.pib_gemm_scratch_bytes(K, b)), 40
    y = lib.alloc(n * b * N * 4)
    for i in range(n):
        lib.check(L.pib_quantize_act_rows(op.TYPE_Q4_K, x, b, K, act, None))
        lib.check(L.pib_gemm(w, act, b, y + i * b * N * 4, scr, None))
    got = lib.to_host(y, (n, b, N), np.float32)
    L.pib_weight_free(w)
    for p in (x, act, scr, y):
        lib.free(p)
    assert all(np.array_equal(got[0], g) for g in got[1:])
    want, lim = reference(blocks, xs)
    assert (np.abs(got[0] - want) <= lim).all()
