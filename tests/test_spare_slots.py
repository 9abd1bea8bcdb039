"""The slots that keep destroyed batches' buffers, by themselves, in a program built from spare_slots.h: one per owner,
whoever puts and takes at the same time, and none lost."""
import os
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "gatk_gb300", "csrc")

MAIN = r"""
#include <atomic>
#include <thread>

#include "spare_slots.h"

int main() {
    ghmm::SpareSlots<int> slots;
    std::atomic<int> live{0};
    auto drop = [&](int *p) {
        if (p) --live;
        delete p;
    };
    auto make = [&] {
        ++live;
        return new int(0);
    };
    const int rounds = 2000;
    int twice = 0;
    for (int round = 0; round < rounds; round++) {
        auto user = [&](uint64_t owner) {
            for (int i = 0; i < 4; i++) drop(slots.put(owner, 0, make()));
        };
        std::thread a(user, 1), b(user, 1), c(user, 2);
        a.join();
        b.join();
        c.join();
        drop(slots.take(1));
        if (int *second = slots.take(1)) {
            twice++;
            drop(second);
        }
        if (round % 2) drop(slots.take(2));
        if (live.load() != (round % 2 ? 0 : 1)) return 2;
    }
    slots.put(3, 0, make());
    slots.put(4, 1, make());
    const auto all = slots.take_all();
    if (all.size() != 2 || all[0].device != 0 || all[1].device != 1 || slots.take(3) || slots.take(4)) return 3;
    for (const auto &s : all) drop(s.kept);
    return twice || live.load() ? 1 : 0;
}
"""


def test_one_per_owner_and_none_lost(tmp_path):
    src, exe = tmp_path / "prog.cpp", tmp_path / "prog"
    src.write_text(MAIN)
    subprocess.run([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-pthread", "-I", CSRC, str(src), "-o", str(exe)],
                   check=True, capture_output=True)
    assert subprocess.run([str(exe)], timeout=120).returncode == 0
