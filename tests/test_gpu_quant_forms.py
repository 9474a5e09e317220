"""The activation quantiser's forms (csrc/act_quant.cu) at the edges of how rows are divided (a warp per 256 values, 32 warps per row, blocks of 8 that share a normed row), with operands
on any address, bit for bit against the oracle's quantiser; the planes of the lean form and the gated matmul (csrc/gemv_mma.cu) against the general ones, bit for bit."""
import ctypes as C
import ctypes.util
import subprocess

import numpy as np
import pytest

from oracle import oracle_py as op
from tests.test_gpu_gemm import rand_q4k

pytestmark = pytest.mark.gpu
Q4_0, Q8_0, Q4_K = op.TYPE_Q4_0, op.TYPE_Q8_0, op.TYPE_Q4_K
V, I, F, L64 = C.c_void_p, C.c_int, C.c_float, C.c_int64
ARGS = {"pib_quantize_act_c": [I, V, I, L64, V, V, V, V, C.c_bool], "pib_silu_mul_quantize_act": [I, V, V, L64, I, L64, V, V, V, V, C.c_bool], "pib_gelu_quantize_act": [I, V, I, L64, V, V, V],
        "pib_add_rmsnorm_quantize_act": [I, V, V, V, V, F, I, L64, V, V, V, V, C.c_bool], "pib_add_layernorm_quantize_act": [I, V, V, V, V, V, V, F, I, L64, V, V, V],
        "pib_gemv_gated": [V, V, I, V, V, V], "pib_gemv_gated_ok": [V, I]}


@pytest.fixture(scope="module")
def lib():
    from pipeinfer_b200 import lib as pib
    L = pib.load()
    L.init(0)
    names = subprocess.run(["nm", "-D", "--defined-only", pib.SO_PATH], capture_output=True, text=True, check=True).stdout.split()
    L.f = {}
    for n, args in ARGS.items():
        L.f[n] = getattr(L.L, next(s for s in names if s.startswith("_Z%d%s" % (len(n), n))))
        L.f[n].argtypes = args
    L.f["pib_gemv_gated_ok"].restype = C.c_bool
    return L


@pytest.fixture(scope="module")
def tables():
    m = C.CDLL(ctypes.util.find_library("m"))
    for f in (m.expf, m.tanhf):
        f.restype, f.argtypes = C.c_float, [C.c_float]
    x = np.arange(65536, dtype=np.uint16).view(np.float16).astype(np.float32)
    with np.errstate(all="ignore"):
        silu = x / (np.float32(1) + np.array([m.expf(-v) for v in x.tolist()], np.float32))
        inner = np.float32(0.79788456080286535587989211986876) * x * (np.float32(1) + np.float32(0.044715) * x * x)
        gelu = np.float32(0.5) * x * (np.float32(1) + np.array([m.tanhf(v) for v in inner.tolist()], np.float32))
        return silu.astype(np.float16), gelu.astype(np.float16)


def look(table, x):
    return table[x.astype(np.float16).view(np.uint16)].astype(np.float32)


class Buffers:
    """device copies that start `off` floats behind an allocation's address"""
    def __init__(self, lib, off):
        self.lib, self.off, self.all = lib, off, []

    def put(self, a):
        d = self.lib.to_device(np.concatenate([np.zeros(self.off, np.float32), np.asarray(a, np.float32).ravel()]))
        self.all.append(d)
        return d + 4 * self.off

    def blocks(self, wt, b, K, act):
        be, bb = {Q4_K: (256, 292)}.get(wt, (32, 34))
        out = np.zeros((b, K // be * bb), np.uint8)
        self.lib.check(self.lib.L.pib_act_to_blocks(wt, act, b, K, out.ctypes.data))
        return out

    def act(self, wt, b, K):
        self.all.append(self.lib.alloc(self.lib.L.pib_act_bytes(wt, K, b)))
        return self.all[-1]

    def free(self):
        for d in self.all:
            self.lib.free(d)


@pytest.mark.parametrize("wt,K", [(Q4_K, 256), (Q4_K, 2048), (Q4_K, 2304), (Q4_K, 8192), (Q4_K, 8448), (Q4_K, 14848), (Q4_0, 32), (Q4_0, 2720), (Q8_0, 4096), (Q4_0, 8224), (Q8_0, 14848)])
@pytest.mark.parametrize("b,off", [(1, 0), (3, 1), (16, 0), (17, 0)])
def test_forms(lib, oracle, tables, wt, K, b, off):
    rng = np.random.default_rng(K + b)
    B = Buffers(lib, off)
    x, y, z = (rng.standard_normal((b, K)).astype(np.float32) * 2 for _ in range(3))
    w, bias = rng.uniform(0.5, 1.5, K).astype(np.float32), rng.standard_normal(K).astype(np.float32)
    if K > 32:
        x[0, 32:64] = 0                                             # a block of zeros
    dx, dy, dz, dw, db, ds = B.put(x), B.put(y), B.put(z), B.put(w), B.put(bias), B.put(np.zeros((b, K)))
    act = B.act(wt, b, K)
    f, ok = lib.f, lib.check

    def same(v):
        assert np.array_equal(B.blocks(wt, b, K, act), oracle.quantize_act(wt, np.ascontiguousarray(v, np.float32)))

    def sums():
        return lib.to_host(ds, (b, K), np.float32)
    ok(f["pib_quantize_act_c"](wt, dx, b, K, act, None, None, None, False))
    same(x)
    for add in (False, True):
        v = x + y if add else x
        n = np.empty_like(v)
        for t in range(b):
            oracle.L.po_rms_norm(v[t].ctypes.data_as(V), n[t].ctypes.data_as(V), K, F(1e-5))
        ok(f["pib_add_rmsnorm_quantize_act"](wt, dx, dy if add else None, ds if add else None, dw, 1e-5, b, K, act, None, None, None, False))
        same(n * w)
        assert not add or np.array_equal(sums(), v)
    v = (x + y) + z
    mean = (v.astype(np.float64).sum(1) / K).astype(np.float32)[:, None]
    var = (((v - mean) ** 2).astype(np.float64).sum(1) / K).astype(np.float32)[:, None]
    ok(f["pib_add_layernorm_quantize_act"](wt, dx, dy, dz, ds, dw, db, 1e-5, b, K, act, None, None))
    same((v - mean) * (np.float32(1) / np.sqrt(var + np.float32(1e-5))) * w + bias)
    assert np.array_equal(sums(), v)
    ok(f["pib_gelu_quantize_act"](wt, dx, b, K, act, None, None))
    same(look(tables[1], x))
    gu = B.put(np.concatenate([x, y], 1))
    ok(f["pib_silu_mul_quantize_act"](wt, gu, gu + 4 * K, 2 * K, b, K, act, None, None, None, False))
    same(look(tables[0], x) * y)
    B.free()


@pytest.mark.parametrize("wt", [Q4_0, Q8_0, Q4_K])
def test_tiny_maxima(lib, oracle, wt):
    """blocks whose largest value is so small that the factor overflows, around that border and at the smallest numbers: the reference's bytes"""
    K, edge = 256 * 12, np.float32(2.0 ** -121 if wt == Q4_K else 127.0 / float(np.finfo(np.float32).max))
    tops = [0.0, edge, np.nextafter(edge, np.float32(1)), np.nextafter(edge, np.float32(0)), 1e-38, 1e-45, 3e-37, 4e-37, 1e-36, 1e-40, -1e-38, -edge]
    x = np.random.default_rng(1).uniform(-1, 1, (12, 256)).astype(np.float32)
    x[:, ::7] = 0
    x /= np.abs(x).max(1, keepdims=True)
    x = (x.astype(np.float64) * np.array(tops, np.float64)[:, None]).astype(np.float32)
    x[:, 3] = tops
    x = x.reshape(1, K)
    with np.errstate(all="ignore"):
        assert np.array_equal(lib.quantize_act(wt, x), oracle.quantize_act(wt, x))


@pytest.mark.parametrize("wt", [Q4_0, Q8_0, Q4_K])
@pytest.mark.parametrize("b", [1, 5, 8, 9, 16])
def test_lean_planes(lib, wt, b):
    """a matmul behind the lean form reads the same planes as behind the general one"""
    N, K = 48, 2304
    rng = np.random.default_rng(b)
    B = Buffers(lib, 0)
    if wt == Q4_K:
        wts = rand_q4k(rng, N, K)
    else:
        wts = rng.integers(0, 256, (N, K // 32, 18 if wt == Q4_0 else 34), dtype=np.uint8)
        wts[:, :, 0:2] = (rng.uniform(0.5, 1.5, (N, K // 32)) * 0.01).astype(np.float16).view(np.uint8).reshape(N, -1, 2)
        wts = wts.reshape(N, -1)
    w = lib.weight_upload(wt, wts, K)
    x = B.put(rng.standard_normal((b, K)))
    out = []
    for lean in (False, True):
        act = B.act(wt, b, K)
        lib.check(lib.L.pib_memcpy_h2d(act, np.full(lib.L.pib_act_bytes(wt, K, b), 0x5a, np.uint8).ctypes.data, lib.L.pib_act_bytes(wt, K, b), None))
        lib.check(lib.f["pib_quantize_act_c"](wt, x, b, K, act, None, None, None, lean))
        y = B.put(np.zeros((b, N)))
        lib.check(lib.L.pib_gemv(w, act, b, y, 0, None))
        out.append(lib.to_host(y, (b, N), np.float32))
    lib.L.pib_weight_free(w)
    B.free()
    assert np.array_equal(*out) and np.abs(out[0]).sum() > 0


@pytest.mark.parametrize("N,K", [(32, 256), (96, 1024), (7584, 2048), (9504, 4096)])
@pytest.mark.parametrize("b", [1, 3, 8, 9, 16])
def test_gated_matmul(lib, tables, N, K, b):
    rng = np.random.default_rng(N + b)
    B = Buffers(lib, 0)
    w = lib.weight_upload(Q4_K, rand_q4k(rng, N, K), K)
    x, act = B.put(rng.standard_normal((b, K)) * 0.3), B.act(Q4_K, b, K)
    y, h = B.put(np.zeros((b, N))), B.put(np.full((b, N // 2), np.nan))
    lib.check(lib.L.pib_quantize_act(Q4_K, x, b, K, act, None))
    lib.check(lib.L.pib_gemv(w, act, b, y, 0, None))
    assert lib.f["pib_gemv_gated_ok"](w, b)
    lib.check(lib.f["pib_gemv_gated"](w, act, b, h, None, None))
    gu, got = lib.to_host(y, (b, N), np.float32), lib.to_host(h, (b, N // 2), np.float32)
    lib.L.pib_weight_free(w)
    B.free()
    assert np.array_equal(got, look(tables[0], gu[:, :N // 2]) * gu[:, N // 2:])


@pytest.mark.parametrize("b,K", [(300, 4096), (4800, 256), (151, 8448), (290, 4352)])        # from a super-block per warp of the machine on (32 x 148): the table in shared memory
def test_gated_rows_of_prompts(lib, b, K):
    """the fp16 rows of a long prompt's gated product are those of its parts, which are too short for that route"""
    rng = np.random.default_rng(b)
    B = Buffers(lib, 0)
    g = rng.standard_normal((b, 2 * K)).astype(np.float32) * 3
    g[0, :256], g[1, 5] = 0, 40000.0
    gu, out, part = B.put(g), B.put(np.zeros((b, K // 2))), B.put(np.zeros((b, K // 2)))
    f = lib.f["pib_silu_mul_quantize_act"]
    lib.check(f(Q4_K, gu, gu + 4 * K, 2 * K, b, K, None, None, None, out, False))
    for r in range(0, b, 40):
        n = min(40, b - r)
        lib.check(f(Q4_K, gu + 8 * K * r, gu + 8 * K * r + 4 * K, 2 * K, n, K, None, None, None, part + 2 * K * r, False))
    got, want = lib.to_host(out, (b, K), np.float16), lib.to_host(part, (b, K), np.float16)
    B.free()
    assert np.array_equal(got.view(np.uint16), want.view(np.uint16)) and np.abs(want.astype(np.float32)).sum() > 0
