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


def test_rows_that_cross_behind_the_kernels(ctx):
    """a program that read the last run's rows gets the next one's without a copy of their own: the same values, of decode batches and of prompts with marks far apart, also when it
    then reads other rows, all rows, or none"""
    want = {n: read(ctx, n, range(n), range(n))[0] for n in (1, 5, 16, 40)}
    for n, marks, rows in [(5, range(5), [0, 4]), (5, [1, 3], [3, 1, 2, 0]), (16, [15], [15]), (40, [3, 17, 39], [39, 3, 17, 20]), (40, range(16), [15, 0]), (40, range(17), [16, 2]), (1, [0], []), (1, [0], [0]),
                           (16, range(16), [7]), (40, [39], [39, 39])]:
        got, _ = read(ctx, n, marks, rows)
        assert not len(rows) or np.array_equal(got, want[n][list(rows)])
    for n, marks in [(16, range(16)), (16, [2]), (40, [39]), (5, [])]:
        read(ctx, n, marks, [marks[0]] if len(marks) else [0])
        assert np.array_equal(read(ctx, n, marks, [], whole=True)[0], want[n])


def test_bytes_of_rows_nobody_reads(ctx):
    sent = C.c_uint64()

    def count():
        ctx.L.llama_pib_io_bytes(ctx.ctx, C.byref(C.c_uint64()), C.byref(sent))
        return sent.value
    per = []
    for rows in ([0], [], [], []):                                   # read once, then never: one run's rows cross in vain
        before = count()
        read(ctx, 4, range(4), rows)
        per.append((count() - before) // (4 * V))
    assert per == [4, 0, 4, 0]


# rows that cross behind the kernels have memory of their run slot, of PIB_PINS slots
PINS = 4


def fresh():
    from pipeinfer_b200 import llama
    return llama.Context(None, n_ctx=256, max_seq=16, synthetic=(2, 256, 4, 2, 512, V, 12, 2, 1, 0.8))


def row(ctx, i):
    return np.ctypeslib.as_array(ctx.L.llama_get_logits_ith(ctx.ctx, i), shape=(V,)).copy()


def check_rows(ctx, n):
    """the finished run's rows are its own: they hold what its sampling kernel found"""
    for i in reversed(range(n)):
        r, top = row(ctx, i), ctx.top8(i)
        assert [float(r[t[0]]) for t in top] == [t[1] for t in top] and r.max() == top[0][1]


def test_nothing_is_allocated_while_a_decode_is_started():
    """rows of a run with more marked rows than were ever read do not cross behind its kernels: only reading makes the memory larger, of the run read and of the next one"""
    ctx, sent, per = fresh(), C.c_uint64(), []
    ctx.L.llama_pib_io_bytes.argtypes = [C.c_void_p, C.POINTER(C.c_uint64), C.POINTER(C.c_uint64)]
    try:
        for n, rows in [(1, [0]), (16, []), (1, []), (16, [0]), (16, []), (16, [])]:
            ctx.L.llama_pib_io_bytes(ctx.ctx, C.byref(C.c_uint64()), C.byref(sent))
            before = sent.value
            read(ctx, n, range(n), rows)
            ctx.L.llama_pib_io_bytes(ctx.ctx, C.byref(C.c_uint64()), C.byref(sent))
            per.append((sent.value - before) // (4 * V))             # rows nobody read count when the next run is finished
        assert per == [1, 0, 0, 16, 0, 16]
    finally:
        ctx.close()


def test_rows_with_runs_in_flight():
    """more of them than there are places, with growing numbers of rows, each read after it is finished while others run"""
    ctx = fresh()
    try:
        ctx.L.llama_kv_cache_clear(ctx.ctx)
        h, b, keep = ctx.start([3], [0], [[15]])
        assert ctx.finish(h, b) == 1
        row(ctx, 0)
        runs = []
        for k in range(24):
            n = 1 + (5 * k) % 9
            ctx.seq_rm(k % 12, 0, 64)
            runs.append((n, ctx.start([(31 * k + 7 * i) % V for i in range(n)], list(range(n)), [[k % 12]] * n)))
            if len(runs) > PINS + 2:
                n0, (h, b, keep) = runs.pop(0)
                assert ctx.finish(h, b) == 1
                check_rows(ctx, n0)
        for n0, (h, b, keep) in runs:
            assert ctx.finish(h, b) == 1
            check_rows(ctx, n0)
    finally:
        ctx.close()


def test_rows_behind_a_cancelled_run():
    """runs behind a cancelled one, and the run that gets its slot, have their own rows: those of the same tokens without a cancellation"""
    ctx = fresh()
    try:
        def go(cancel):
            ctx.L.llama_kv_cache_clear(ctx.ctx)
            out, runs = [], []
            for k in range(3):
                runs.append(ctx.start([40 + 10 * k + i for i in range(4)], list(range(4)), [[k]] * 4, batch_id=100 + k))
                if k == 1 and cancel:
                    ctx.L.llama_cancel_run(ctx.ctx, (C.c_int32 * 1)(101), 1)
            for k, (h, b, keep) in enumerate(runs):
                assert ctx.finish(h, b) == 1
                if k != 1:
                    check_rows(ctx, 4)
                    out.append(np.stack([row(ctx, i) for i in range(4)]))
            for k in range(4):                                       # the slots again
                h, b, keep = ctx.start([70 + k], [0], [[4 + k]], batch_id=110 + k)
                assert ctx.finish(h, b) == 1
                check_rows(ctx, 1)
                out.append(row(ctx, 0)[None])
            return np.concatenate(out)
        want = go(False)
        for _ in range(3):
            assert np.array_equal(go(True), want)
    finally:
        ctx.close()
