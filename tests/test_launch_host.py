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
    src.write_text('#include <cstdio>\n#include "context.hpp"\n#include "model.hpp"\nusing namespace pssa;\nint bad = 0;\n'
                   '#define CHECK(x) do { if (!(x)) { ++bad; std::printf("line %d: %s\\n", __LINE__, #x); } } while (0)\n'
                   f"int main() {{\n{body}\nreturn bad;\n}}\n")
    build = subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), "-I", str(CUDA / "include"), str(src), "-o", str(exe)],
                           capture_output=True, text=True)
    assert build.returncode == 0, build.stderr
    ran = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert ran.returncode == 0, ran.stdout


pytestmark = pytest.mark.skipif(not (CUDA / "include" / "cuda_runtime.h").exists(), reason="no CUDA headers")


def test_a_host_call_sends_what_its_own_lanes_need(tmp_path):
    """The tables of a call lie apart, on 16 bytes, inside what the workspace holds for a call of that size, and take no more
    words than they have but for the rounding, however many lanes a workspace has room for."""
    run_cpp(tmp_path, """
    size_t at[kHostTables];
    for (size_t lanes : {1, 2, 3, 4, 5, 37, 16384})
        for (size_t rows : {1, 4, 63, 200, 65536})
            for (int given = 0; given < 64; ++given) {  // which of the lane tables a call fills
                size_t n[kHostTables], sum = rows;
                for (size_t i = 0; i + 1 < kHostTables; ++i) sum += n[i] = given >> i & 1 ? lanes : 0;
                n[kHostTables - 1] = rows;
                const size_t words = lay_host_tables(n, at);
                CHECK(words >= sum && words < sum + 4 * kHostTables && words <= host_tables_words(rows, lanes));
                for (size_t i = 0; i < kHostTables; ++i) CHECK(at[i] % 4 == 0 && at[i] + n[i] <= (i + 1 < kHostTables ? at[i + 1] : words));
            }""")


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
