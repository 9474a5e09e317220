"""CPU: the sizes of a context's prompt buffers (csrc/prompt_plan.cuh) over prompts of growing length and where memory refuses: at most two allocations, none asked for again
after a refusal, none given up before the larger one is there."""
import os
import subprocess

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "prompt_plan.cuh"
int main(int argc, char ** argv) {      // n_ctx, stages, tokens memory holds, then prompts: a line per prompt with the capacity behind it and the sizes asked for
    pib_prompt_plan p;
    for (int i = 4; i < argc; i++) {
        printf("%s:", argv[i]);
        const bool ok = p.grow(atoi(argv[i]), atoi(argv[1]), atoi(argv[2]), [&](int n) { printf(" ask %d", n); return n <= atoi(argv[3]); });
        printf(" %s %d\n", ok ? "cap" : "none", p.cap);
    }
}
"""


def plan(tmp_path, *args):
    exe = tmp_path / "plan"
    if not exe.exists():
        (tmp_path / "plan.cpp").write_text(PROGRAM)
        subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "pipeinfer_b200", "csrc"), "-o", str(exe), str(tmp_path / "plan.cpp")], check=True)
    return subprocess.run([str(exe)] + [str(a) for a in args], check=True, capture_output=True, text=True).stdout.split("\n")[:-1]


def test_sizes(tmp_path):
    assert plan(tmp_path, 4096, 1, 1 << 20, 40, 256, 300, 600, 900, 1024, 3000, 40) == [
        "40: ask 256 cap 256", "256: cap 256", "300: ask 1024 cap 1024", "600: cap 1024", "900: cap 1024", "1024: cap 1024", "3000: cap 1024", "40: cap 1024"]
    assert plan(tmp_path, 500, 1, 1 << 20, 300, 500) == ["300: ask 512 cap 512", "500: cap 512"]                    # no longer than the context
    assert plan(tmp_path, 4096, 4, 1 << 20, 40, 3000) == ["40: ask 256 cap 256", "3000: cap 256"]                   # stages overlap passes of 256
    assert plan(tmp_path, 4096, 1, 600, 300, 900, 2000, 100) == ["300: ask 1024 ask 768 ask 512 cap 512", "900: cap 512", "2000: cap 512", "100: cap 512"]
    assert plan(tmp_path, 4096, 1, 300, 40, 300, 900, 40) == ["40: ask 256 cap 256", "300: ask 1024 ask 768 ask 512 cap 256", "900: cap 256", "40: cap 256"]
    assert plan(tmp_path, 4096, 1, 0, 300, 40) == ["300: ask 1024 ask 768 ask 512 ask 256 none 0", "40: ask 256 none 0"]
