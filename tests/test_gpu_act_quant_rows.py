"""RMSNorm + quantiser of wide rows in 32-element blocks (csrc/act_quant.cu) where the number of CTAs per row is held down: bit-exact against the oracle."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle_py as op

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wt", [op.TYPE_Q4_0, op.TYPE_Q8_0])
@pytest.mark.parametrize("b,K", [(16, 8192), (14, 8192), (13, 8224), (16, 14848), (16, 28672), (15, 4544), (1, 14848)])
def test_norm_and_blocks(oracle, wt, b, K):
    from pipeinfer_b200 import load
    lib = load()
    lib.init(0)
    rng = np.random.default_rng(b + K)
    x, w = (rng.standard_normal((b, K)) * 3).astype(np.float32), rng.uniform(0.5, 1.5, K).astype(np.float32)
    xn = np.empty_like(x)
    for t in range(b):
        oracle.L.po_rms_norm(x[t].ctypes.data_as(C.c_void_p), xn[t].ctypes.data_as(C.c_void_p), K, C.c_float(1e-5))
    assert np.array_equal(lib.quantize_act(wt, x, norm_w=w, eps=1e-5), oracle.quantize_act(wt, xn * w))
    assert np.array_equal(lib.quantize_act(wt, x), oracle.quantize_act(wt, x))
