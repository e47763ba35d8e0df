"""The passes over host rows (chromofold_b200/csrc/host_rows.cpp), in the form of this machine's processor and in the one that any
processor compiles: copies are exact, and a row with NaN or Inf is told from every finite one."""
import os
import shutil
import subprocess

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chromofold_b200", "csrc")

PROGRAM = r"""
#include "host_rows.h"
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <vector>
int main() {
    for (size_t n : {1u, 3u, 31u, 32u, 33u, 64u, 127u, 1000u})
        for (size_t at = 0; at < n; at += 1 + n / 40)
            for (float odd : {0.0f, -3e38f, std::numeric_limits<float>::infinity(), -std::numeric_limits<float>::infinity(), std::nanf(""), -std::nanf("")}) {
                std::vector<float> a(n + 1), b(n + 1, 7.0f);
                for (size_t i = 0; i < n; ++i) a[i] = (i % 2 ? -1.0f : 1.0f) * static_cast<float>(i);
                a[at] = odd;
                const bool finite = std::isfinite(odd);
                if ((chromofold_max_magnitude(a.data(), n) < 0x7f800000u) != finite) return 1;
                if ((chromofold_copy_max_magnitude(b.data(), a.data(), n) < 0x7f800000u) != finite) return 2;
                if (memcmp(a.data(), b.data(), n * sizeof(float)) != 0 || b[n] != 7.0f) return 3;
            }
    std::puts("ok");
    return 0;
}
"""


@pytest.mark.parametrize("flags", [[], ["-U__x86_64__", "-U__i386__", "-D__builtin_cpu_supports=no_such_builtin"]], ids=["own", "any"])
def test_rows_are_copied_and_told_apart(tmp_path, flags):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src = tmp_path / "rows.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "rows"
    unit = tmp_path / "unit.o"
    subprocess.run([gxx, "-std=c++17", "-O3", *flags, "-c", os.path.join(SRC, "host_rows.cpp"), "-o", str(unit)], check=True, capture_output=True)
    subprocess.run([gxx, "-std=c++17", "-O1", "-I", SRC, str(src), str(unit), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == "ok\n"
