"""Attention of decode steps in layer-list models (csrc/mixer_kernels.cu): a batch of one token per sequence fetches rows in front of the launch it waits for, a batch in which some
sequence has two does not.  The same tokens both ways, behind prompts shorter than a block's warps, around a trip of keys, and longer than a window."""
import json

import numpy as np
import pytest

from tests.gusedra_configs import CONFIGS

pytestmark = pytest.mark.gpu


def run(cfg, prompts, steps, two, alone=False):
    from pipeinfer_b200 import llama
    ctx = llama.Context(config=json.dumps(cfg), n_ctx=1024, max_seq=8, float32=True, seed=5, state_slots=8)
    L, S, out = ctx.L, len(prompts), []

    def decode(toks, pos, seqs):
        b, keep = llama.make_batch(toks, pos, [[s] for s in seqs], 1, ctx.max_seq)
        assert L.llama_decode(ctx.ctx, b) == 0
        return np.stack([np.ctypeslib.as_array(L.llama_get_logits_ith(ctx.ctx, i), shape=(ctx.n_vocab,)).copy() for i in range(len(toks))])
    for s, p in enumerate(prompts):
        decode(p, list(range(len(p))), [s] * len(p))
    for k, row in enumerate(steps):
        toks, pos, seqs = list(row), [len(p) + k for p in prompts], list(range(S))
        if two:                                                      # another sequence's two tokens behind them
            toks, pos, seqs = toks + [3, 4], pos + [2 * k, 2 * k + 1], seqs + [S, S]
        if alone:                                                    # two other sequences' one token each: as many rows, every one a sequence of its own
            toks, pos, seqs = toks + [3, 4], pos + [k, k], seqs + [S, S + 1]
        out.append(decode(toks, pos, seqs)[:S])
    ctx.close()
    return np.stack(out)


@pytest.mark.parametrize("name", ["slope_only", "bucket_only", "shared_cells", "far_keys", "wide_heads", "big_heads"])
def test_steps_both_ways(name):
    cfg = CONFIGS[name]()
    rng = np.random.default_rng(3)
    prompts = [rng.integers(0, cfg["vocab"], n).tolist() for n in (1, 14, 63, 64, 300)]
    steps = rng.integers(0, cfg["vocab"], (4, len(prompts))).tolist()
    a, b = run(cfg, prompts, steps, False), run(cfg, prompts, steps, True)
    # fp32 throughout; matmuls of 5 and of 7 rows add in the same order, so what differs is at most the rounding of a fused multiply-add per score
    assert np.abs(a - b).max() <= 1e-4 * np.abs(b).max()


@pytest.mark.parametrize("name", ["slope_only", "bucket_only", "shared_cells", "far_keys", "wide_heads", "big_heads", "mixed_small"])
def test_same_bits_beside_other_sequences(name):
    """as many rows in a batch, so that the same blocks share a head's keys: the two forms of the kernel round alike"""
    cfg = CONFIGS[name]()
    rng = np.random.default_rng(4)
    prompts = [rng.integers(0, cfg["vocab"], n).tolist() for n in (2, 15, 64, 65, 301)]
    steps = rng.integers(0, cfg["vocab"], (6, len(prompts))).tolist()
    assert np.array_equal(run(cfg, prompts, steps, False, alone=True), run(cfg, prompts, steps, True))
