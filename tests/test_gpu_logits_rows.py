"""Which rows of logits cross to the host (llama_get_logits_ith): the rows that a batch marks in one copy, any other row by itself, and the same values either way."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
V = 2048


@pytest.fixture(scope="module")
def ctx():
    from pipeinfer_b200 import llama
    c = llama.Context(None, n_ctx=64, max_seq=8, synthetic=(2, 256, 4, 2, 512, V, 12, 2, 1, 0.8))
    c.L.llama_pib_io_bytes.argtypes = [C.c_void_p, C.POINTER(C.c_uint64), C.POINTER(C.c_uint64)]
    c.L.llama_get_logits.restype, c.L.llama_get_logits.argtypes = C.POINTER(C.c_float), [C.c_void_p]
    yield c
    c.close()


def read(ctx, n, marks, rows, whole=False):
    """decodes n tokens with the given rows marked (None: no marks), then reads rows one after the other: values, rows copied per read"""
    from pipeinfer_b200 import llama
    ctx.L.llama_kv_cache_clear(ctx.ctx)
    b, keep = llama.make_batch([5 + 7 * i for i in range(n)], list(range(n)), [[0]] * n, 0, 8)
    if marks is None:
        b.logits = None
    else:
        for i in range(n):
            b.logits[i] = 1 if i in marks else 0
    assert ctx.L.llama_decode(ctx.ctx, b) == 0
    sent, out, copied = C.c_uint64(), [], []

    def count():
        ctx.L.llama_pib_io_bytes(ctx.ctx, C.byref(C.c_uint64()), C.byref(sent))
        return sent.value

    before = count()
    for i in rows:
        p = ctx.L.llama_get_logits_ith(ctx.ctx, i)
        out.append(np.ctypeslib.as_array(p, shape=(V,)).copy())
        copied.append((count() - before) // (4 * V))
        before = count()
    if whole:
        out = np.ctypeslib.as_array(ctx.L.llama_get_logits(ctx.ctx), shape=(n, V)).copy()
        copied = (count() - before) // (4 * V)
    return np.array(out), copied


@pytest.mark.parametrize("n,marks,rows,copied", [
    (16, range(16), [3, 0, 15], [16, 0, 0]), (16, [15], [15, 15, 2, 3], [1, 0, 1, 1]), (13, [4, 6], [6, 4, 5, 12, 0], [3, 0, 0, 1, 1]), (5, [], [4, 1], [1, 1]), (1, [0], [0], [1]),
    (7, None, [2, 6], [7, 0])])
def test_rows_copied(ctx, n, marks, rows, copied):
    want, _ = read(ctx, n, range(n), range(n))
    got, c = read(ctx, n, marks, rows)
    assert np.array_equal(got, want[list(rows)]) and c == copied


@pytest.mark.parametrize("marks", [[2], [], range(9)])
def test_all_rows(ctx, marks):
    want, _ = read(ctx, 9, range(9), range(9))
    got, c = read(ctx, 9, marks, [], whole=True)
    assert np.array_equal(got, want) and c == 9
