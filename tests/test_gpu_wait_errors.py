"""A tensor-core kernel whose bounded wait runs out leaves a word in its stream.  The word is written here in the kernel's place: the call that asks reports it once, a run
that launched such kernels fails, and neither a run without them nor a later one inherits it."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from oracle import oracle_py as op
from tests import gusedra_oracle as O
from tests.gusedra_configs import CONFIGS
from tests.test_gpu_gemm import rand_q4k

pytestmark = pytest.mark.gpu


def test_gemm_check():
    from pipeinfer_b200 import lib as pib
    lib = pib.load()
    lib.init(0)
    L, N, K, b = lib.L, 256, 512, 40
    L.pib_gemm.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_void_p, C.c_void_p, C.c_void_p]
    L.pib_gemm_check.argtypes = [C.c_void_p]
    L.pib_gemm_scratch_bytes.restype, L.pib_gemm_scratch_bytes.argtypes = C.c_size_t, [C.c_int64, C.c_int]
    names = subprocess.run(["nm", "-D", "--defined-only", pib.SO_PATH], capture_output=True, text=True, check=True).stdout.split()
    word = getattr(L, next(n for n in names if "pib_tc_error_word" in n))
    word.restype, word.argtypes = C.c_void_p, [C.c_void_p]
    rng = np.random.default_rng(1)
    w = lib.weight_upload(op.TYPE_Q4_K, rand_q4k(rng, N, K), K)
    act, scr, y = (lib.alloc(n) for n in (L.pib_act_bytes(op.TYPE_Q4_K, K, b), L.pib_gemm_scratch_bytes(K, b), b * N * 4))
    x = lib.to_device(rng.standard_normal((b, K)).astype(np.float32))
    L.pib_quantize_act_rows.argtypes = L.pib_quantize_act.argtypes
    lib.check(L.pib_quantize_act_rows(op.TYPE_Q4_K, x, b, K, act, None))
    lib.check(L.pib_gemm(w, act, b, y, scr, None))
    lib.check(L.pib_gemm_check(None))
    seven = np.array([7], np.int32)
    lib.check(L.pib_memcpy_h2d(word(None), seven.ctypes.data, 4, None))
    lib.check(L.pib_gemm(w, act, b, y, scr, None))
    assert L.pib_gemm_check(None) == -1 and b"block 6" in L.pib_last_error()
    lib.check(L.pib_gemm_check(None))
    L.pib_weight_free(w)
    for p in (x, act, scr, y):
        lib.free(p)


def decode(ctx, n, bid):
    from pipeinfer_b200 import llama
    ctx.L.llama_kv_cache_seq_rm(ctx.ctx, 0, 0, -1)
    b, keep = llama.make_batch([3 + i % 90 for i in range(n)], list(range(n)), [[0]] * n, bid, ctx.max_seq)
    return ctx.L.llama_decode(ctx.ctx, b)


def test_prompt_run():
    from pipeinfer_b200 import llama
    ctx = llama.Context(None, n_ctx=768, max_seq=2, synthetic=(2, 512, 8, 8, 1024, 256, op.TYPE_Q4_K, 1, 1, 1.0))
    L = ctx.L
    L.llama_pib_debug_tc_error.argtypes = [C.c_void_p, C.c_int]
    assert decode(ctx, 40, 0) == 0
    assert L.llama_pib_debug_tc_error(ctx.ctx, 3) == 0
    assert decode(ctx, 1, 1) == 0                     # launches none of these kernels
    assert decode(ctx, 600, 2) != 0                   # three passes: the first one's word reaches the run
    assert decode(ctx, 600, 3) == 0 and decode(ctx, 1, 4) == 0
    ctx.close()


def test_layer_list_run(tmp_path):
    from pipeinfer_b200 import llama
    cfg = CONFIGS["mixed_small"]()
    O.write_model(str(tmp_path), cfg, O.random_weights(cfg, 3))
    ctx = llama.Context(model_dir=str(tmp_path), n_ctx=128, max_seq=2)
    L = ctx.L
    L.llama_pib_debug_tc_error.argtypes = [C.c_void_p, C.c_int]
    assert decode(ctx, 20, 0) == 0
    assert L.llama_pib_debug_tc_error(ctx.ctx, 3) == 0
    assert decode(ctx, 20, 1) != 0 and decode(ctx, 20, 2) == 0
    ctx.close()
