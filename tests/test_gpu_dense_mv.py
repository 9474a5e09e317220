"""Few rows against bfloat16 weights on the tensor cores (mv_mma_kernel, csrc/dense_mm.cu) at the edges of its tiles: weight rows that fill no tile, k that fills no
chunk and leaves warps without any, one to sixteen tokens, strided rows, outputs in pairs.  The operands are bfloat16 (products exact in fp32), so an output is off by
fp32 sums only: below (K + 8) 2^-23 sum |w x|."""
import ctypes as C

import numpy as np
import pytest

from pipeinfer_b200 import load
from tests.rapisun_oracle import bf16_round
from tests.test_gpu_dense_mm import mm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,ldx", [(1, 1, 8, 8), (2, 15, 16, 20), (4, 17, 40, 40), (8, 16, 256, 260), (9, 33, 264, 264), (16, 48, 2056, 2056), (7, 100, 1280, 1284), (13, 31, 1032, 1032)])
def test_few_rows(M, N, K, ldx):
    rng = np.random.default_rng(M + 10 * N + K)
    W, X = bf16_round(rng.standard_normal((N, K))), rng.standard_normal((M, ldx))
    Xr = bf16_round(X[:, :K])
    got, lim = mm(W, X, M, N, K, ldx=ldx).reshape(M, N), (K + 8) * 2.0 ** -23 * (np.abs(Xr) @ np.abs(W).T)
    assert (np.abs(got - Xr @ W.T) <= lim).all()
    one = mm(W, X[M - 1:], 1, N, K, ldx=ldx).reshape(N)              # a token's outputs do not depend on the rest of the batch
    assert np.array_equal(one, got[M - 1])


# (148 SMs) CTAs of 16 rows: one per SM up to 2368 rows, two up to 4736, three up to 7104; groups of weights that a warp has: K / 1024
@pytest.mark.parametrize("N,K", [(2368, 1024), (2369, 1000), (4736, 1024), (4737, 1024), (4737, 520),                    # one group: in shared memory, in registers
                                 (4737, 2048), (7104, 1032), (7105, 2048), (7105, 4104),                                # two places, used once and in turn; registers for 9 to 16 tokens
                                 (2369, 2056), (4736, 3080), (4720, 7168),                                              # three places
                                 (2368, 4096), (2368, 5128), (40, 11272)])                                             # five places
@pytest.mark.parametrize("M", [1, 8, 9, 16])
def test_weights_in_flight(M, N, K):
    """both sides of each line at which the groups of weights that a warp has in flight change (launch_mm), with more groups than places and fewer; the bound as above"""
    rng = np.random.default_rng(M + 10 * N + K)
    W, X = bf16_round(rng.standard_normal((N, K), dtype=np.float32)), bf16_round(rng.standard_normal((M, K)))
    got, again = mm(W, X, M, N, K).reshape(M, N), mm(W, X, M, N, K).reshape(M, N)
    assert np.array_equal(got, again)
    assert (np.abs(got - X @ W.T) <= (K + 8) * 2.0 ** -23 * (np.abs(X) @ np.abs(W).T)).all()


def test_weights_in_flight_of_grouped_rows():
    """rows divided over problems, each launch of a problem behind the launch wait, with places used in turn"""
    rng = np.random.default_rng(5)
    Z, N, K, M = 6, 1000, 4104, 14
    zr = [0, 3, 3, 4, 12, 12, 14]
    W, X = bf16_round(rng.standard_normal((Z, N, K), dtype=np.float32)), bf16_round(rng.standard_normal((M, K)))
    got = mm(W, X, M, N, K, Z=Z, wz=N * K, zrange=zr).reshape(M, N)
    for z in range(Z):
        r = slice(zr[z], zr[z + 1])
        assert (np.abs(got[r] - X[r] @ W[z].T) <= (K + 8) * 2.0 ** -23 * (np.abs(X[r]) @ np.abs(W[z]).T)).all()


@pytest.mark.parametrize("M,N,K", [(1, 24, 64), (16, 40, 2048)])
def test_weight_rows_of_the_launch_in_front(M, N, K):
    """W that an earlier launch makes (an attention's gathered keys): none of it is read before that launch is through, however late it is"""
    lib = load()
    lib.init(0)
    L = lib.L
    L.pib_dense_mm_made_host.argtypes = [C.c_void_p] * 3 + [C.c_int] * 3
    rng = np.random.default_rng(M + N + K)
    W, X = bf16_round(rng.standard_normal((N, K))), bf16_round(rng.standard_normal((M, K)))
    bits, x, y = (W.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16), X.astype(np.float32), np.full((M, N), np.nan, np.float32)
    for _ in range(3):
        lib.check(L.pib_dense_mm_made_host(bits.ctypes.data, x.ctypes.data, y.ctypes.data, M, N, K))
        assert (np.abs(y - X @ W.T) <= (K + 8) * 2.0 ** -23 * (np.abs(X) @ np.abs(W).T)).all()


@pytest.mark.parametrize("M,N,K", [(3, 32, 8192), (12, 48, 16384)])
def test_sums_do_not_drift(M, N, K):
    """long sums of one sign: the tensor core cuts towards zero, per 16 k and by less than an ulp of their sum, 2^-23; what is added up outside is rounded to nearest.
    So the error's mean stays within 2^-23 for any K (one accumulator for all of a warp's k was off by 2e-6 at 16384)"""
    rng = np.random.default_rng(M + K)
    W, X = bf16_round(rng.uniform(0.5, 1, (N, K))), bf16_round(rng.uniform(0.5, 1, (M, K)))
    got = mm(W, X, M, N, K).reshape(M, N).astype(np.float64)
    rel = got / (X.astype(np.float64) @ W.astype(np.float64).T) - 1
    print("K %d: mean relative error %.2g, mean size %.2g" % (K, rel.mean(), np.abs(rel).mean()))
    assert abs(rel.mean()) < 2.0 ** -23


class MM(C.Structure):
    """pib_mm (csrc/hybrid.cuh)"""
    _fields_ = [("W", C.c_void_p), ("wtype", C.c_int), ("ldw", C.c_int64), ("wz", C.c_int64), ("X", C.c_void_p), ("ldx", C.c_int64), ("xz", C.c_int64), ("xrows", C.c_void_p), ("xdiv", C.c_int),
                ("Y", C.c_void_p), ("ldy", C.c_int64), ("yz", C.c_int64), ("M", C.c_int), ("N", C.c_int), ("K", C.c_int), ("Z", C.c_int), ("zlist", C.c_void_p), ("zrange", C.c_void_p),
                ("epi", C.c_int), ("e0", C.c_float), ("e1", C.c_float), ("exact", C.c_int), ("Y2", C.c_void_p), ("ld2", C.c_int64), ("n2", C.c_int), ("rows2", C.c_void_p),
                ("x_bf16", C.c_int), ("y_bf16", C.c_int), ("w_made", C.c_int)]


@pytest.mark.parametrize("N1,N2,K", [(1024, 3712, 1000), (1024, 3744, 1024), (1024, 3744, 2048), (1024, 6080, 2056), (1024, 6096, 2048)])      # 296 / 298 and 444 / 445 CTAs, one group and more
@pytest.mark.parametrize("M", [1, 8, 9, 16])
def test_two_matmuls_in_a_launch(N1, N2, K, M):
    """both sides of the lines at which the pair's weights wait in registers or in shared memory; the bound as above"""
    lib = load()
    lib.init(0)
    f = lib.L._Z17pib_dense_mm_pairRK6pib_mmS1_P11CUstream_st
    f.argtypes = [C.c_void_p] * 3
    rng = np.random.default_rng(M + N1 + N2 + K)
    X = bf16_round(rng.standard_normal((M, K)))
    Ws = [bf16_round(rng.standard_normal((n, K), dtype=np.float32)) for n in (N1, N2)]
    x = lib.to_device(X.astype(np.float32))
    mms, dev = [], [x]
    for w in Ws:
        wd, y = lib.to_device((w.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16)), lib.to_device(np.full((M, len(w)), np.nan, np.float32))
        dev += [wd, y]
        mms.append(MM(W=wd, wtype=30, ldw=K, X=x, ldx=K, xdiv=1, Y=y, ldy=len(w), M=M, N=len(w), K=K, Z=1, n2=0x7fffffff))
    lib.check(f(C.byref(mms[0]), C.byref(mms[1]), None))
    lib.check(lib.L.pib_stream_sync(None))
    for w, m in zip(Ws, mms):
        got = lib.to_host(m.Y, (M, len(w)), np.float32)
        assert (np.abs(got - X @ w.T) <= (K + 8) * 2.0 ** -23 * (np.abs(X) @ np.abs(w).T)).all()
    for d in dev:
        lib.free(d)
