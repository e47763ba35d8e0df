"""How the decoder warps of a pair of CTAs hand pages to each other in the shared-prefix kernel (pair_slot, pair_round,
pair_rounds_arrived, chromofold_b200/csrc/cf_device_common.cuh), played on the host in random order with mbarriers as the PTX manual describes them: each
round's barrier takes eight arrivals and the bytes of the other CTA's pages. Warps may leave at any slot and issuing threads at any
round, as they do when a wait runs out. A warp arrives for a round only when the tiles of the one two before are free in both CTAs, so
no arrival may meet a barrier that has had its eight; a warp whose record never came sends pages all the same. And what a pair
waits for before it leaves early (pair_rounds_arrived) tells when the pages that were sent have landed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "cf_device_common.cuh"
#include <algorithm>
#include <random>
#include <vector>
using namespace cfb;
constexpr uint32_t kWarps = 11, kBytes = 8192;
struct Barrier {   // of one parity of rounds in one CTA
    uint32_t phase = 0, pending = 8;
    uint64_t bytes = 0;
    bool overrun = false;
    void settle() { if (pending == 0 && bytes == 0) ++phase, pending = 8; }
    void arrive(uint64_t expect) {
        bytes += expect;
        if (pending == 0) overrun = true; else --pending;
        settle();
    }
    void land() { bytes -= kBytes; settle(); }
    bool done(uint32_t round) const { return phase > round >> 1; }
};
struct Copy { uint32_t to, parity; };
int main() {
    std::mt19937 rng(1);
    auto below = [&](uint32_t n) { return static_cast<uint32_t>(rng() % n); };
    for (uint32_t rank = 0; rank < 2; ++rank)   // the two CTAs' slots are those of the pair's sequence, each once
        for (uint32_t m = 0; m < 1000; ++m)
            if (pair_slot(m, rank) / 8 != pair_round(m) || pair_slot(m, rank) % 8 != 4 * rank + m % 4) return 1;
    int left_early = 0;
    for (int game = 0; game < 8000; ++game) {
        const uint32_t rounds = 1 + below(12);   // with the one that tells to stop
        const bool trouble = game % 4 != 0;
        Barrier full[2][2];
        uint32_t next[2][kWarps], taken[2] = {0, 0};   // next slot of a warp; rounds an issuer has taken, and so freed
        bool left[2][kWarps] = {}, over[2] = {}, gave_up[2] = {};
        std::vector<Copy> flying;
        for (auto &cta : next) for (uint32_t w = 0; w < kWarps; ++w) cta[w] = w;
        auto land = [&](uint32_t i) {
            full[flying[i].to][flying[i].parity].land();
            flying[i] = flying.back();
            flying.pop_back();
        };
        for (;;) {
            const uint32_t c = below(2), w = below(kWarps + 2);
            if (w == kWarps + 1) {
                if (!flying.empty()) land(below(static_cast<uint32_t>(flying.size())));
            } else if (w == kWarps) {
                if (over[c]) continue;
                if (full[c][taken[c] & 1].done(taken[c])) over[c] = ++taken[c] == rounds;
                else if (trouble && below(300) == 0) over[c] = gave_up[c] = true;
            } else if (!left[c][w]) {
                const uint32_t round = pair_round(next[c][w]);
                if (round >= rounds) {
                    left[c][w] = true;
                } else if (round < 2 || (taken[0] > round - 2 && taken[1] > round - 2)) {
                    full[c][round & 1].arrive(0);
                    const bool stop = round + 1 == rounds;   // no pages in it
                    full[c ^ 1][round & 1].arrive(stop ? 0 : kBytes);
                    if (!stop) flying.push_back({c ^ 1, round & 1});
                    next[c][w] += kWarps;
                } else if (trouble && below(200) == 0) {
                    left[c][w] = true;
                }
            }
            bool end = over[0] && over[1];
            for (auto &cta : left) for (bool l : cta) end = end && l;
            if (end) break;
        }
        for (auto &cta : full) for (const Barrier &b : cta) if (b.overrun) return 2;
        if (!gave_up[0] && !gave_up[1] && !flying.empty()) return 3;   // issuers that took every round have seen every page land
        if (!gave_up[0] && !gave_up[1]) continue;
        // Before they leave, the warps make up arrivals up to the last round that any has arrived for; then the barriers of the last
        // two rounds must tell exactly when the last page has landed.
        uint32_t arrived = 0;
        for (auto &cta : next) for (uint32_t m : cta) arrived = std::max(arrived, pair_rounds_arrived(m, kWarps));
        std::vector<uint32_t> missing[2];
        for (uint32_t c = 0; c < 2; ++c)
            for (uint32_t m : next[c]) for (; pair_round(m) < arrived; m += kWarps) missing[c].push_back(pair_round(m));
        for (;;) {
            for (uint32_t c = 0; c < 2; ++c) {
                bool told = missing[0].empty() && missing[1].empty(), there = true;
                for (uint32_t r = arrived < 2 ? 0 : arrived - 2; r < arrived; ++r) {
                    told = told && full[c][r & 1].done(r);
                    if (full[c][r & 1].phase > (r >> 1) + 1) return 4;   // the parity would be that of a phase to come
                }
                for (const Copy &f : flying) there = there && f.to != c;
                if (missing[0].empty() && missing[1].empty() && told != there) return 5;
            }
            if (flying.empty() && missing[0].empty() && missing[1].empty()) break;
            const uint32_t c = below(2);
            if (!missing[c].empty() && below(2)) {
                const uint32_t i = below(static_cast<uint32_t>(missing[c].size()));
                for (auto &cta : full) cta[missing[c][i] & 1].arrive(0);
                missing[c].erase(missing[c].begin() + i);
            } else if (!flying.empty()) {
                land(below(static_cast<uint32_t>(flying.size())));
            }
        }
        for (auto &cta : full) for (const Barrier &b : cta) if (b.overrun) return 6;
        ++left_early;
    }
    return left_early > 2000 ? 0 : 7;
}
"""


def test_no_arrival_meets_a_full_round_and_no_page_lands_after_the_end(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    src = tmp_path / "pair.cu"
    src.write_text(PROGRAM)
    exe = tmp_path / "pair"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Wno-deprecated-gpu-targets", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "chromofold_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, f"check {out.returncode} failed"
