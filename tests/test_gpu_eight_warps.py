"""Q4_K matmuls of decode batches on both sides of the lines between four and eight warps per row tile where tiles are more than a round (csrc/gemv_mma.cu), against the oracle; a
token's sums are the same bits beside any other tokens up to eight, and up to sixteen on these shapes."""
import numpy as np
import pytest

from oracle import oracle_py as op
from tests.test_gpu_wide_routes import Q4, blocks, test_both_sides as both_sides

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,K", [(11840, 4096), (11841, 4096), (11841, 3840), (16571, 4096), (16577, 4096), (16577, 8192), (33145, 8192), (33153, 8192), (13000, 7936)])      # 740 / 741, 1036 / 1037, 2072 / 2073 tiles
@pytest.mark.parametrize("b", [1, 2, 3, 8, 13])
def test_lines(oracle, N, K, b):
    both_sides(oracle, Q4, N, K, b)


@pytest.mark.parametrize("N,K", [(12288, 4096), (11841, 8192)])
def test_same_bits_at_any_number_of_tokens(N, K):
    from pipeinfer_b200 import load
    lib = load()
    lib.init(0)
    rng = np.random.default_rng(N)
    w, x = blocks(rng, Q4, N, K), rng.standard_normal((16, K)).astype(np.float32)
    h = lib.weight_upload(Q4, w, K)
    want = lib.mul_mat(h, x, N, 0)
    for b in (1, 2, 3, 7, 8, 9, 15):
        assert np.array_equal(lib.mul_mat(h, x[:b], N, 0), want[:b])
    lib.L.pib_weight_free(h)
