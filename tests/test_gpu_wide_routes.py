"""K-quant matmuls on both sides of each line at which pib_gemv changes between four and eight warps per row tile, K shares and none, one and two CTAs per SM
(csrc/gemv_mma.cu, gemv_q5k.cu, gemv_q6k.cu, gemv_q3k.cu), with token counts that fill octets of the activation planes and that do not, against the oracle."""
import numpy as np
import pytest

from oracle import oracle_py as op
from tests.test_gpu_kernels import REL_TOL

pytestmark = pytest.mark.gpu
Q3, Q4, Q5, Q6 = op.TYPE_Q3_K, op.TYPE_Q4_K, op.TYPE_Q5_K, op.TYPE_Q6_K
SCALES = {Q3: (108,), Q4: (0, 2), Q5: (0, 2), Q6: (208,)}          # fp16 numbers of a block


def blocks(rng, wt, N, K):
    w = rng.integers(0, 256, (N, K // 256, op.BLOCK[wt][1]), dtype=np.uint8)
    for at in SCALES[wt]:
        w[:, :, at:at + 2] = (rng.uniform(0.5, 1.5, (N, K // 256)) * 1e-3).astype(np.float16).view(np.uint8).reshape(N, K // 256, 2)
    return w.reshape(N, -1)


@pytest.mark.parametrize("wt,N,K,b", [
    (Q4, 2353, 1792, 1), (Q4, 2353, 2048, 8), (Q4, 2371, 2304, 9), (Q4, 7555, 2048, 7), (Q4, 7569, 2048, 16),      # 7 / 8 super-blocks, 148 / 149 and 473 / 474 tiles
    (Q4, 9471, 4096, 15), (Q4, 9485, 4096, 9), (Q4, 2361, 8448, 16), (Q4, 40, 6400, 13),                          # 592 / 593 tiles; one CTA per SM
    (Q6, 2353, 1792, 3), (Q6, 2353, 2048, 8), (Q6, 2371, 2304, 9), (Q6, 4735, 4096, 15), (Q6, 4743, 4096, 16), (Q6, 19, 4352, 1),      # 148 / 149 and 296 / 297 tiles
    (Q5, 2353, 1792, 3), (Q5, 2353, 2048, 8), (Q5, 2353, 2304, 9), (Q5, 2371, 2304, 9), (Q5, 4735, 4096, 7), (Q5, 4743, 4096, 1),
    (Q3, 2353, 1792, 3), (Q3, 2353, 2048, 8), (Q3, 2371, 2304, 9), (Q3, 4735, 4096, 15), (Q3, 4743, 4096, 16),
    (Q3, 2353, 2048, 1), (Q3, 4743, 4096, 1), (Q5, 2353, 2048, 1), (Q6, 4743, 4096, 1), (Q5, 1031, 2816, 12), (Q5, 1031, 8192, 9)])      # one token; two octets, a CTA per SM
def test_both_sides(oracle, wt, N, K, b):
    from pipeinfer_b200 import load
    lib = load()
    lib.init(0)
    rng = np.random.default_rng(N + K + b)
    w, x = blocks(rng, wt, N, K), rng.standard_normal((b, K)).astype(np.float32)
    rows = np.unique(np.concatenate([np.arange(min(N, 34)), np.arange(max(0, N - 34), N), rng.integers(0, N, 64)]))
    h = lib.weight_upload(wt, w, K)
    got = lib.mul_mat(h, x, N, 0)
    again = lib.mul_mat(h, x, N, 0)
    lib.L.pib_weight_free(h)
    ref = oracle.mul_mat(wt, np.ascontiguousarray(w[rows]), x)
    assert np.array_equal(got, again) and np.isfinite(got).all()
    assert np.abs(got[:, rows] - ref).max() <= REL_TOL * max(1.0, np.abs(ref).max())
