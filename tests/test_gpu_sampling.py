"""Top 8 and probabilities of a row (csrc/sampling.cu) against numpy where its slices and lists have edges: rows shorter than eight values, than a block, around the
lengths that are divided over 2, 4 or 8 blocks, many rows (no cluster), equal values (the first index wins, across slices too), zeros of both signs, -inf everywhere but a few
places, a row's best all in one thread's share (it keeps two and looks for the rest), values that are no numbers, biases at slice borders."""
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


def top8(L, f, x, ids, val):
    """ids, logits and probabilities of the top eight, and the rows afterwards"""
    rows, V = x.shape
    d, di, dv, out = L.to_device(x), L.to_device(ids), L.to_device(val), L.alloc(x.shape[0] * 96)
    L.check(f(d, rows, V, di, dv, len(ids), out, None, None, None))
    raw, after = L.to_host(out, (rows, 24), np.int32), L.to_host(d, x.shape, np.float32)
    for p in (d, di, dv, out):
        L.free(p)
    return raw[:, :8], raw[:, 8:16].copy().view(np.float32), raw[:, 16:].copy().view(np.float32), after


@pytest.mark.parametrize("rows,V,kind", [(1, 5, "plain"), (2, 8, "plain"), (3, 255, "ties"), (1, 4095, "plain"), (1, 4096, "ties"), (4, 4097, "plain"), (1, 8192, "inf"), (16, 32000, "ties"), (1, 32768, "plain"),
                                         (1, 32769, "plain"), (2, 65000, "inf"), (1, 151000, "ties"), (300, 1000, "ties"), (700, 9000, "plain"), (26, 32000, "ties"),
                                         (27, 32000, "plain"), (52, 20000, "plain"), (53, 20000, "ties"), (104, 9000, "plain"), (209, 5000, "plain"), (120, 49000, "ties"), (110, 97000, "plain")])
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
    got_i, got_l, got_p, after = top8(L, f, x, ids, val)
    x[:, ids] += val
    assert np.array_equal(after, x)
    n = min(8, V)
    for r in range(rows):
        order = np.argsort(-x[r], kind="stable")[:n]
        assert np.array_equal(got_i[r, :n], order) and np.array_equal(got_l[r, :n], x[r, order])
        z = np.exp((x[r] - x[r].max()).astype(np.float64))
        np.testing.assert_allclose(got_p[r, :n], (z / z.sum())[order], rtol=3e-6, atol=0)     # a float exponential's error (2 ulp) and one rounding


# a row of 40 000 is divided over 8 blocks of 256 threads, 700 rows are one block each
@pytest.mark.parametrize("rows,V,parts", [(1, 40000, 8), (700, 9000, 1)])
@pytest.mark.parametrize("order", ["falling", "rising", "equal"])
def test_best_of_one_thread(fn, rows, V, parts, order):
    """the eight largest values of a slice all lie in one thread's share: six of them come from its second and later walks"""
    L, f = fn
    rng = np.random.default_rng(V + parts)
    x = rng.uniform(-2, -1, (rows, V)).astype(np.float32)
    vals = {"falling": np.arange(16, 0, -1), "rising": np.arange(1, 17), "equal": np.full(16, 3)}[order]
    for r in range(rows):
        lo = V * int(rng.integers(parts)) // parts
        x[r, lo + int(rng.integers(256)) + 256 * np.arange(16)] = vals
    i, l, _, _ = top8(L, f, x, np.zeros(1, np.int32), np.zeros(1, np.float32))
    want = np.argsort(-x, axis=1, kind="stable")[:, :8]
    assert np.array_equal(i, want) and np.array_equal(l, np.take_along_axis(x, want, 1))


@pytest.mark.parametrize("rows,V", [(1, 300), (1, 40000), (700, 9000)])
def test_zeros_and_no_numbers(fn, rows, V):
    """-0 and +0 are equal, so the first of them wins; a value that is no number is never in front of one"""
    L, f = fn
    rng = np.random.default_rng(rows + V)
    bias = np.full(1, V - 1, np.int32), np.zeros(1, np.float32)
    x = np.where(rng.random((rows, V)) < 0.5, np.float32(0.0), np.float32(-0.0)).astype(np.float32)
    x[:, ::3] = -1
    i, l, p, _ = top8(L, f, x, *bias)
    assert np.array_equal(i, np.argsort(-x, axis=1, kind="stable")[:, :8]) and (l == 0).all()
    z = np.exp(x.astype(np.float64))
    np.testing.assert_allclose(p, np.broadcast_to(1 / z.sum(1, keepdims=True), p.shape), rtol=3e-6, atol=0)
    x = rng.standard_normal((rows, V)).astype(np.float32)
    x[:, rng.integers(0, V, V // 4)] = np.nan
    i, l, _, _ = top8(L, f, x, *bias)
    want = np.argsort(np.where(np.isnan(x), np.inf, -x), axis=1, kind="stable")[:, :8]
    assert np.array_equal(i, want) and np.array_equal(l, np.take_along_axis(x, want, 1))
