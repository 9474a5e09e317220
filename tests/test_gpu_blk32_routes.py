"""Q4_0 / Q8_0 matmuls on both sides of each line at which pib_gemv changes between its ring kernels (eight or four warps per row tile) and the K split
(csrc/gemv_blk32.cu), with rows that fill no tile and widths that fill no record and leave warps fewer records than others, against the oracle."""
import numpy as np
import pytest

from oracle import oracle_py as op
from tests.test_gpu_kernels import REL_TOL, rand_blocks

pytestmark = pytest.mark.gpu
Q4, Q8 = op.TYPE_Q4_0, op.TYPE_Q8_0


@pytest.mark.parametrize("wt,N,K,b", [
    (Q4, 4725, 4096, 8), (Q4, 4739, 4096, 8), (Q4, 5675, 4160, 7), (Q4, 5683, 4160, 8),             # 296 / 297 and 355 / 356 tiles: eight warps, four, four, eight
    (Q4, 7543, 4160, 8), (Q4, 7555, 4160, 8), (Q8, 7543, 4160, 8), (Q8, 7555, 4160, 1),             # 472 / 473: eight warps, K split (of one)
    (Q4, 7555, 2048, 5), (Q4, 7555, 2080, 5), (Q4, 7543, 3552, 2),                                  # short rows: four warps, K split, four warps
    (Q4, 9471, 4160, 8), (Q4, 9480, 4160, 8), (Q4, 11827, 4544, 1), (Q4, 11841, 1056, 8),           # 592 / 593 and 740 / 741: K split, four warps, four warps, K split
    (Q4, 9471, 4160, 13), (Q4, 9481, 4160, 16), (Q8, 9471, 4160, 9), (Q8, 9481, 4160, 13),          # two token groups, 592 / 593: eight warps, K split
    (Q4, 2355, 18944, 13), (Q4, 2369, 18944, 13), (Q8, 3773, 18944, 9), (Q8, 3785, 18944, 16),      # long rows, 148 / 149 and 236 / 237: eight warps, K split, K split, eight warps
    (Q4, 1179, 14848, 8), (Q8, 1187, 14848, 8), (Q8, 944, 14848, 13), (Q4, 955, 14848, 13),         # few tiles: 74 / 75, two groups 59 / 60: K split, eight warps
    (Q4, 37, 4096, 1), (Q8, 37, 4160, 1), (Q8, 3, 3872, 16), (Q4, 1, 32, 1)])
def test_both_sides(oracle, wt, N, K, b):
    from pipeinfer_b200 import load
    lib = load()
    lib.init(0)
    rng = np.random.default_rng(N + K + b)
    w, x = rand_blocks(rng, wt, N, K), rng.standard_normal((b, K)).astype(np.float32)
    rows = np.unique(np.concatenate([np.arange(min(N, 34)), np.arange(max(0, N - 34), N), rng.integers(0, N, 64)]))
    h = lib.weight_upload(wt, w, K)
    got = lib.mul_mat(h, x, N, 0)
    again = lib.mul_mat(h, x, N, 0)
    lib.L.pib_weight_free(h)
    ref = oracle.mul_mat(wt, np.ascontiguousarray(w[rows]), x)
    assert np.array_equal(got, again) and np.isfinite(got).all()
    assert np.abs(got[:, rows] - ref).max() <= REL_TOL * max(1.0, np.abs(ref).max())
