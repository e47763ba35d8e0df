"""SlotRing (chromofold_b200/csrc/slot_ring.h) on the host: whatever threads do in between, a call that waits for its slot's event
finds it recorded after the slot's last launch."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "slot_ring.h"
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>
int main() {
    cfb::SlotRing<4> ring;
    std::atomic<int> launched[4] = {}, recorded[4] = {}, bad{0}, calls{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 12; ++t)
        threads.emplace_back([&] {
            for (int i = 0; i < 200; ++i)
                ring.take([&](uint32_t slot) {
                    if (launched[slot] != recorded[slot]) ++bad;   // the event waited for is an older use's
                    std::this_thread::yield();
                    ++launched[slot];
                    std::this_thread::sleep_for(std::chrono::microseconds(i % 5));
                    ++recorded[slot];
                    return ++calls;
                });
        });
    for (auto &t : threads) t.join();
    for (int s = 0; s < 4; ++s) bad += launched[s] != 600;   // and the slots are taken in turn
    std::printf("%d %d\n", bad.load(), calls.load());
    return 0;
}
"""


def test_a_slot_is_chosen_launched_into_and_marked_in_one_step(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not found")
    src = tmp_path / "ring.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "ring"
    subprocess.run([gxx, "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "chromofold_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split() == ["0", "2400"]
