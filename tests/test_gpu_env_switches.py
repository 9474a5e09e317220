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
