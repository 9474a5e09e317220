"""Q4_0 / Q8_0 matmuls on both sides of the lines at which many row tiles go to the four-warp rings (csrc/gemv_blk32.cu), against the oracle; where one token group's route adds in the
same order, a token's sums are the same bits."""
import numpy as np
import pytest

from oracle import oracle_py as op
from tests.test_gpu_blk32_routes import Q4, Q8, test_both_sides as both_sides
from tests.test_gpu_kernels import rand_blocks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wt", [Q4, Q8])
@pytest.mark.parametrize("N,K,b", [(4731, 2048, 9), (4737, 2048, 16), (4739, 4096, 13), (7099, 4096, 9), (7105, 4096, 16), (7111, 1056, 11), (9466, 2048, 12), (9475, 2048, 9), (14208, 4096, 9),
                                   (14211, 4096, 10), (7099, 4352, 9), (18939, 4352, 9), (18945, 4352, 16), (18946, 96, 15), (4960, 1024, 13), (4961, 1056, 13), (18960, 7168, 10),
                                   (18961, 7200, 16)])      # 296 / 297, 444 / 445, 592 / 593, 888 / 889, 1184 / 1185 tiles; 4 / 5, 16 / 17, 28 / 29 records
def test_two_groups(oracle, wt, N, K, b):
    both_sides(oracle, wt, N, K, b)


@pytest.mark.parametrize("N,K,b", [(28416, 2048, 4), (28417, 2048, 4), (28417, 2048, 5), (28423, 8192, 8), (28417, 7936, 8), (28421, 160, 1), (28417, 1024, 3)])      # 1776 / 1777 tiles; 31 / 32 records
def test_one_group(oracle, N, K, b):
    both_sides(oracle, Q4, N, K, b)


def test_same_bits_at_any_number_of_tokens():
    from pipeinfer_b200 import load
    lib = load()
    lib.init(0)
    rng = np.random.default_rng(7)
    N, K = 28500, 1536
    w, x = rand_blocks(rng, Q4, N, K), rng.standard_normal((16, K)).astype(np.float32)
    h = lib.weight_upload(Q4, w, K)
    want = lib.mul_mat(h, x, N, 0)
    for b in (1, 4, 5, 8, 9):
        assert np.array_equal(lib.mul_mat(h, x[:b], N, 0), want[:b])
    lib.L.pib_weight_free(h)
