"""Switches of the environment that a program sets after the library is loaded, or that one of several kernels of a step could pass by (children: each is read once per process)."""
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def child(code, **env):
    r = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, **env), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    return r.stdout


@pytest.mark.gpu
def test_dumps_of_a_program_that_asks_for_them_before_its_first_decode(tmp_path):
    child("import os\nfrom pipeinfer_b200 import llama, load\nload()\n"
          "c = llama.Context(None, n_ctx=64, max_seq=2, synthetic=(2, 256, 4, 2, 512, 512, 12, 2, 1, 0.8))\n"
          f"os.environ['PIB_DUMP_DIR'] = {str(tmp_path)!r}\n"
          "assert c.decode([1, 2, 3], [0, 1, 2], [[0]] * 3)[0] == 0\nc.close()\n", PIB_GRAPHS="0")
    for il in range(2):
        gate, up = (np.fromfile(tmp_path / f"{n}.{il}.bin", np.float32) for n in ("gate", "up"))
        assert gate.shape == up.shape == (3 * 512,) and np.isfinite(gate).all() and gate.any() and up.any()


@pytest.mark.gpu
def test_k_shares_of_every_matmul(tmp_path):
    """PIB_RING_SPLIT reaches the gate and up matmul of a decode batch also where its product would be formed behind it (with dumps it is not: the same bits with and without)"""
    out = []
    for k, env in enumerate([{}, {"PIB_DUMP_DIR": str(tmp_path)}]):
        path = tmp_path / f"logits{k}.npy"
        child("import numpy as np\nfrom pipeinfer_b200 import llama\n"
              "c = llama.Context(None, n_ctx=64, max_seq=2, synthetic=(4, 2048, 32, 4, 5632, 512, 12, 2, 0, 0.0))\n"
              f"np.save({str(path)!r}, c.decode([1, 2, 3], [0, 1, 2], [[0]] * 3)[1])\nc.close()\n", PIB_GRAPHS="0", PIB_RING_SPLIT="2", **env)
        out.append(np.load(path))
    assert np.array_equal(out[0], out[1])
