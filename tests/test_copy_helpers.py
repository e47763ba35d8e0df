"""Checked copies of host rows shared by several threads (chromofold_b200/csrc/copy_helpers.h): every size around the pieces' edges, one
copy after the other and after pauses in which the helpers fall asleep; a value that is not finite is found wherever it lies. Without
memory for the helpers, and in a process that was forked and has none, the caller copies alone."""
import os
import shutil
import subprocess

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chromofold_b200", "csrc")

PROGRAM = r"""
#include "copy_helpers.h"
#include <cstdio>
#include <cstring>
#include <limits>
using cfb::CopyHelpers;
int main() {
    const size_t piece = CopyHelpers::kPieceFloats, least = CopyHelpers::kLeastFloats;
    for (int object = 0; object < 3; ++object) {
        CopyHelpers helpers;   // one of them ends without a copy, and one that is asleep
        for (int turn = 0; object < 2 && turn < 60; ++turn)
            for (size_t n : {size_t{1}, least - 1, least, least + 1, 5 * piece - 1, 5 * piece, 5 * piece + 1, 33 * piece + 7}) {
                std::vector<float> a(n + 1), b(n + 1, 7.0f);
                for (size_t i = 0; i < n; ++i) a[i] = static_cast<float>((i * 31 + turn) % 1000) - 500.0f;
                const bool finite = turn % 3 != 0;
                if (!finite) a[(n * static_cast<size_t>(turn)) / 60] = -std::numeric_limits<float>::infinity();
                if ((helpers.copy(b.data(), a.data(), n) < 0x7f800000u) != finite) return 1;
                if (std::memcmp(a.data(), b.data(), n * sizeof(float)) != 0 || b[n] != 7.0f) return 2;
                if (turn % 20 == 7) std::this_thread::sleep_for(2 * CopyHelpers::kAwake);
            }
        if (object == 1) std::this_thread::sleep_for(20 * CopyHelpers::kAwake);
    }
    std::puts("ok");
    return 0;
}
"""


NO_MEMORY = r"""
#include "copy_helpers.h"
#include <cstdio>
#include <algorithm>
#include <cstdlib>
#include <new>
using cfb::CopyHelpers;
static int allocations = -1;   // that still succeed, -1: all
void *operator new(std::size_t n) {
    if (allocations == 0) throw std::bad_alloc();
    if (allocations > 0) --allocations;
    return std::malloc(n);
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }
int main() {
    const size_t n = CopyHelpers::kLeastFloats + 5;
    std::vector<float> a(n, 1.0f), b(n);
    for (int left = 0; left < 12; ++left) {
        std::fill(b.begin(), b.end(), 0.0f);
        CopyHelpers helpers;
        for (int turn = 0; turn < 3; ++turn) {
            allocations = left;
            const uint32_t top = helpers.copy(b.data(), a.data(), n);
            allocations = -1;
            if (top != 0x3f800000u || a != b) return 1;
        }
    }
    std::puts("ok");
    return 0;
}
"""


FORKED = r"""
#include "copy_helpers.h"
#include <algorithm>
#include <cstdio>
#include <sys/wait.h>
#include <unistd.h>
using cfb::CopyHelpers;
int main() {
    const size_t n = 40 * CopyHelpers::kPieceFloats;
    std::vector<float> a(n, 1.0f), b(n);
    for (int turn = 0; turn < 20; ++turn) {
        CopyHelpers *helpers = new CopyHelpers;
        if (turn % 5) helpers->copy(b.data(), a.data(), n);
        if (turn % 2) std::this_thread::sleep_for(20 * CopyHelpers::kAwake);   // they are asleep, or awake
        const pid_t child = fork();
        if (child == 0) {
            alarm(10);
            std::fill(b.begin(), b.end(), 0.0f);
            const uint32_t top = helpers->copy(b.data(), a.data(), n);
            const bool right = top == 0x3f800000u && a == b;
            delete helpers;
            _exit(right ? 0 : 1);
        }
        int status = 0;
        if (waitpid(child, &status, 0) != child || status != 0) return 1;
        std::fill(b.begin(), b.end(), 0.0f);   // and in the one that has them all goes on
        if (helpers->copy(b.data(), a.data(), n) != 0x3f800000u || a != b) return 2;
        delete helpers;
    }
    std::puts("ok");
    return 0;
}
"""


AWAKE = r"""
#include "copy_helpers.h"
#include <algorithm>
#include <cstdio>
using cfb::CopyHelpers;
int main() {
    const size_t n = 24u << 20;   // a copy of several milliseconds
    std::vector<float> a(n, 1.0f), b(n);
    CopyHelpers helpers;
    std::vector<uint32_t> asleep(41);
    for (uint32_t &count : asleep) {
        helpers.copy(b.data(), a.data(), n);
        const auto until = std::chrono::steady_clock::now() + CopyHelpers::kAwake / 2;
        while (std::chrono::steady_clock::now() < until) {}
        count = helpers.asleep();
        std::this_thread::sleep_for(20 * CopyHelpers::kAwake);
    }
    std::sort(asleep.begin(), asleep.end());
    if (asleep[20] > 1) return 1;   // the odd one may be kept from running
    std::puts("ok");
    return 0;
}
"""


SMALL = r"""
#include "copy_helpers.h"
#include <cstdio>
#include <filesystem>
#include <iterator>
using cfb::CopyHelpers;
static long threads() { return std::distance(std::filesystem::directory_iterator("/proc/self/task"), std::filesystem::directory_iterator()); }
int main() {
    CopyHelpers helpers;
    std::vector<float> a(256 * 128, 1.0f), b(256 * 128);
    helpers.copy(b.data(), a.data(), 160 * 128);
    if (threads() != 1) return 1;
    helpers.copy(b.data(), a.data(), 256 * 128);
    if (threads() == 1) return 2;
    std::puts("ok");
    return 0;
}
"""


def _run(tmp_path, program):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src, exe = tmp_path / "copies.cpp", tmp_path / "copies"
    src.write_text(program)
    subprocess.run([gxx, "-std=c++17", "-O2", "-pthread", "-I", SRC, os.path.join(SRC, "host_rows.cpp"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.stdout == "ok\n", out.returncode


def test_shared_copies_are_exact(tmp_path):
    _run(tmp_path, PROGRAM)


def test_a_caller_without_memory_for_helpers_copies_alone(tmp_path):
    _run(tmp_path, NO_MEMORY)


def test_a_forked_process_copies_alone_and_ends(tmp_path):
    _run(tmp_path, FORKED)


@pytest.mark.skipif((os.cpu_count() or 1) < 4, reason="needs a processor for each helper")
def test_helpers_look_for_the_next_copy_after_a_long_one(tmp_path):
    _run(tmp_path, AWAKE)


@pytest.mark.skipif((os.cpu_count() or 1) < 2 or not os.path.isdir("/proc/self/task"), reason="counts threads")
def test_small_copies_start_no_helpers(tmp_path):
    """160 rows of 128 channels are copied faster by the caller alone, 256 with helpers."""
    _run(tmp_path, SMALL)
