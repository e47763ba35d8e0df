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


ELSEWHERE = """
#include <stddef.h>
#include <stdint.h>
#include <string.h>
#undef __x86_64__
#undef __i386__
#define __builtin_cpu_supports no_such_builtin
"""


@pytest.mark.parametrize("before", ["", ELSEWHERE], ids=["own", "any"])
def test_rows_are_copied_and_told_apart(tmp_path, before):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    unit, src, exe = tmp_path / "unit.cpp", tmp_path / "rows.cpp", tmp_path / "rows"
    unit.write_text(before + '#include "host_rows.cpp"\n')
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O2", "-I", SRC, str(unit), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True).stdout == "ok\n"
