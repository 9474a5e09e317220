"""The Q4_K GEMM in three K shares (csrc/gemm_q4k_tc.cu): one and two groups of warps, both ends of the numbers of blocks that go there, shares of unequal length, rows and tokens that
fill no tile, and the neighbours that do not.  Reference and bound as in test_gpu_gemm_shapes."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle_py as op
from tests import test_gpu_gemm_shapes as shapes
from tests.test_gpu_gemm import rand_q4k

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K,b", [(9600, 4608, 24), (11520, 4608, 64), (11515, 4864, 33), (11528, 4608, 40), (9472, 4608, 40), (9601, 8192, 100), (10368, 8192, 128), (10496, 8192, 97),     # two CTAs per SM
                                   (4352, 1536, 100), (4992, 1792, 180), (4355, 2048, 256), (5120, 1280, 97), (6000, 1536, 130)])                                       # one
def test_three_shares(N, K, b):
    from pipeinfer_b200 import load
    lib = load()
    lib.init(0)
    lib.L.pib_gemm_host.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p]
    rng = np.random.default_rng(N + K + b)
    w, x = rand_q4k(rng, N, K), rng.standard_normal((b, K)).astype(np.float32)
    h = lib.weight_upload(op.TYPE_Q4_K, w, K)
    ys = []
    for _ in range(3):                                               # calls that follow one another
        y = np.full((b, N), np.nan, np.float32)
        lib.check(lib.L.pib_gemm_host(h, x.ctypes.data, b, y.ctypes.data))
        ys.append(y)
    lib.L.pib_weight_free(h)
    assert all(np.array_equal(ys[0], y) for y in ys[1:])
    for r in range(0, N, 1600):                                      # the reference in pieces of rows
        want, bound = shapes.reference(w[r:r + 1600], x)
        assert (np.abs(ys[0][:, r:r + 1600] - want) <= bound).all()


@pytest.mark.parametrize("N,K,b,shares,groups", [
    (9600, 4608, 24, 3, 1), (11520, 4608, 64, 3, 1), (11515, 4864, 33, 3, 1), (11528, 4608, 40, 1, 2), (9472, 4608, 40, 2, 1), (9601, 8192, 100, 3, 1), (10368, 8192, 128, 3, 1), (10496, 8192, 97, 1, 2),
    (4352, 1536, 100, 3, 2), (4992, 1792, 180, 3, 2), (4355, 2048, 256, 3, 2), (5120, 1280, 97, 2, 2), (6000, 1536, 130, 2, 2)])
def test_route(N, K, b, shares, groups):
    """which of the shapes above take three shares"""
    from pipeinfer_b200 import load
    lib = load()
    lib.init(0)
    lib.L.pib_gemm_shares.argtypes = [C.c_int64, C.c_int64, C.c_int, C.POINTER(C.c_int)]
    g = C.c_int()
    assert (lib.L.pib_gemm_shares(N, K, b, C.byref(g)), g.value) == (shares, groups)
    assert lib.L.pib_gemm_shares(N, K + 1, b, None) == lib.L.pib_gemm_shares(0, K, b, None) == lib.L.pib_gemm_shares(N, K, 0, None) == -1
