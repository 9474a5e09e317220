"""CPU: the record of kernel attributes (csrc/per_device.cuh) against a made-up device number: set once per device and size, on a second device of the process too, and again after an
error."""
import os
import subprocess

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
PROGRAM = r"""
#include <cstdio>
#include "per_device.cuh"
static int device = 0;
extern "C" cudaError_t cudaGetDevice(int * d) { *d = device; return cudaSuccess; }
static pib_per_device flag, sized;
static void ask(int dev, size_t size, cudaError_t answer) {
    device = dev;
    int called = 0;
    const cudaError_t r = size ? sized.once(size, [&] { called++; return answer; }) : flag.once([&] { called++; return answer; });
    printf("%d%s ", called, r == cudaSuccess ? "" : "!");
}
int main() {
    const cudaError_t bad = cudaErrorInvalidValue;
    ask(0, 0, cudaSuccess); ask(0, 0, cudaSuccess); ask(1, 0, cudaSuccess); ask(1, 0, cudaSuccess); ask(0, 0, cudaSuccess);
    ask(2, 0, bad); ask(2, 0, cudaSuccess); ask(2, 0, cudaSuccess); ask(63, 0, cudaSuccess); ask(63, 0, cudaSuccess); ask(64, 0, cudaSuccess); ask(64, 0, cudaSuccess);
    printf("\n");
    ask(0, 100, cudaSuccess); ask(0, 90, cudaSuccess); ask(0, 200, cudaSuccess); ask(0, 100, cudaSuccess); ask(3, 100, cudaSuccess); ask(3, 200, bad); ask(3, 200, cudaSuccess); ask(3, 150, cudaSuccess);
}
"""


def test_set_once_per_device_and_size(tmp_path):
    (tmp_path / "t.cpp").write_text(PROGRAM)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(cuda, "include"), "-I", os.path.join(ROOT, "pipeinfer_b200", "csrc"), "-o", str(tmp_path / "t"), str(tmp_path / "t.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "t")], check=True, capture_output=True, text=True).stdout.split("\n")
    assert out[0].split() == ["1", "0", "1", "0", "0", "1!", "1", "0", "1", "0", "1", "1"]
    assert out[1].split() == ["1", "0", "1", "0", "1", "1!", "1", "0"]


def test_launches_keep_no_flag_of_the_process():
    """the attribute of a kernel is never recorded for the whole process"""
    src = os.path.join(ROOT, "pipeinfer_b200", "csrc")
    for f in sorted(os.listdir(src)):
        if f.endswith((".cu", ".cuh")):
            assert "bool configured" not in open(os.path.join(src, f)).read(), f
