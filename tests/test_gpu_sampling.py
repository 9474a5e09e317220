"""Top 8 and probabilities of a row (csrc/sampling.cu) against numpy where its slices and lists have edges: rows shorter than eight values, than a block, at the borders
of the register form, many rows (no cluster), equal values (the first index wins, across slices too), -inf everywhere but a few places, biases at slice borders."""
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
    f = getattr(L.L, next(n for n in names if "pib_sample_topkPf" in n))
    f.argtypes = [C.c_void_p, C.c_int, C.c_int, C.c_void_p, C.c_void_p, C.c_int] + [C.c_void_p] * 4
    return L, f


@pytest.mark.parametrize("rows,V,kind", [(1, 5, "plain"), (2, 8, "plain"), (3, 255, "ties"), (1, 4095, "plain"), (1, 4096, "ties"), (4, 4097, "plain"), (1, 8192, "inf"), (16, 32000, "ties"), (1, 32768, "plain"),
                                         (1, 32769, "plain"), (2, 65000, "inf"), (1, 151000, "ties"), (300, 1000, "ties"), (700, 9000, "plain")])
def test_topk(fn, rows, V, kind):
    L, f = fn
    rng = np.random.default_rng(rows + V)
    x = rng.standard_normal((rows, V)).astype(np.float32) * 3
    if kind == "ties":
        x = np.round(x)
    if kind == "inf":
        keep = rng.integers(0, V, (rows, 5))
        y = np.full_like(x, -np.inf)
        np.put_along_axis(y, keep, np.take_along_axis(x, keep, 1), 1)
        x = y
    ids = np.unique(np.concatenate([[0, V - 1], np.arange(1, 8) * V // 8, rng.integers(0, V, 4)])).astype(np.int32)
    val = rng.standard_normal(len(ids)).astype(np.float32)
    d, di, dv = L.to_device(x), L.to_device(ids), L.to_device(val)
    out = L.alloc(rows * 96)
    L.check(f(d, rows, V, di, dv, len(ids), out, None, None, None))
    raw = L.to_host(out, (rows, 24), np.int32)
    got_i, got_l, got_p = raw[:, :8], raw[:, 8:16].copy().view(np.float32), raw[:, 16:].copy().view(np.float32)
    x[:, ids] += val
    assert np.array_equal(L.to_host(d, x.shape, np.float32), x)
    n = min(8, V)
    for r in range(rows):
        order = np.argsort(-x[r], kind="stable")[:n]
        assert np.array_equal(got_i[r, :n], order) and np.array_equal(got_l[r, :n], x[r, order])
        z = np.exp((x[r] - x[r].max()).astype(np.float64))
        np.testing.assert_allclose(got_p[r, :n], (z / z.sum())[order], rtol=3e-6, atol=0)     # a float exponential's error (2 ulp) and one rounding
    for p in (d, di, dv, out):
        L.free(p)
