"""Host code of the launchers, compiled for the CPU."""
import os
import pathlib
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "pssa_b200" / "csrc"
CUDA = pathlib.Path(os.environ.get("CUDA_HOME", "/usr/local/cuda"))


def run_cpp(tmp_path, body):
    """Compiles and runs a program that returns the number of failed checks."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text('#include <cstdio>\n#include "context.hpp"\nusing namespace pssa;\nint bad = 0;\n'
                   '#define CHECK(x) do { if (!(x)) { ++bad; std::printf("line %d: %s\\n", __LINE__, #x); } } while (0)\n'
                   f"int main() {{\n{body}\nreturn bad;\n}}\n")
    build = subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-I", str(CUDA / "include"), str(src), "-o", str(exe)],
                           capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    ran = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert ran.returncode == 0, ran.stdout


@pytest.mark.skipif(not (CUDA / "include" / "cuda_runtime.h").exists(), reason="no CUDA headers")
def test_resident_ctas_follow_the_shared_memory_whatever_came_first(tmp_path):
    """One kernel, launches of several widths: each is judged by its own CTAs to an SM, in any order and on each device; an
    unchanged width is not asked for twice, and an error is not kept."""
    run_cpp(tmp_path, """
    PerDeviceCount c;
    int asked = 0, n = 0;
    auto fits = [](size_t smem) { return (int)(233472 / (smem + 1024)); };
    auto get = [&](int dev, size_t smem) {
        CHECK(c.get(dev, smem, &n, [&](int* k) { ++asked; *k = fits(smem); return cudaSuccess; }) == cudaSuccess);
        return n;
    };
    for (size_t smem : {6144, 65536, 24576, 65536, 6144, 0, 232448, 0})
        for (int dev : {0, 3, 63, 64, -1}) CHECK(get(dev, smem) == fits(smem));
    asked = 0;
    for (int i = 0; i < 5; ++i) CHECK(get(7, 40960) == fits(40960));
    CHECK(asked == 1);
    CHECK(c.get(8, 1024, &n, [&](int*) { return cudaErrorInvalidValue; }) == cudaErrorInvalidValue);
    CHECK(get(8, 1024) == fits(1024));""")
