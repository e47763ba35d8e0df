"""The barriers on which the softmax warps of the shared-prefix kernel tell the issuing thread of a pair's CTA that a round's weights are
stored (weights_barrier, chromofold_b200/csrc/cf_device_common.cuh), checked on the host over every order of events that the
roles' other waits allow: the issuer must see a round's arrival exactly when it has happened."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "cf_device_common.cuh"
#include <cstdio>
#include <set>
#include <tuple>
#include <vector>
using namespace cfb;
int main() {
    // (scores issued, outputs issued, rounds whose weights are stored): issuer_role sends scores at most two rounds ahead of its
    // outputs, softmax_role stores the weights of a round whose scores are there, and then arrives
    const uint32_t rounds = 12;
    std::set<std::tuple<uint32_t, uint32_t, uint32_t>> seen;
    std::vector<std::tuple<uint32_t, uint32_t, uint32_t>> todo = {{0, 0, 0}};
    while (!todo.empty()) {
        const auto [s, o, stored] = todo.back();
        todo.pop_back();
        if (!seen.insert({s, o, stored}).second) continue;
        if (o < s) {
            const RoundBarrier b = weights_barrier(o);
            if (b.index >= kWeightBarriers) return 1;
            uint32_t completed = 0;   // phases of the barrier that round o goes by
            for (uint32_t r = 0; r < stored; ++r) completed += weights_barrier(r).index == b.index;
            const bool visible = (completed & 1u) != b.parity;   // mbarrier.test_wait.parity
            if (visible != (stored > o)) return 2;
            if (visible) todo.push_back({s, o + 1, stored});
        }
        if (s < rounds && s < o + 2) todo.push_back({s + 1, o, stored});
        if (stored < s) todo.push_back({s, o, stored + 1});
    }
    std::printf("%d\n", static_cast<int>(seen.count({rounds, rounds, rounds})));
    return 0;
}
"""


def test_the_issuer_sees_a_rounds_weights_exactly_when_they_are_stored(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "weights.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "weights"
    subprocess.run([nvcc, "-std=c++17", "-Wno-deprecated-gpu-targets", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "chromofold_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0, f"check {out.returncode} failed"
    assert int(out.stdout) == 1
