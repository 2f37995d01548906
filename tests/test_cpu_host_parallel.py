"""Loops over host threads (csrc/host_parallel.h, built here by itself): every
index once, and an exception in any of the threads reaches the caller (planning a
batch's LPs allocates; an exception that left its thread would end the process
instead of returning a status)."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "coolpdlp.jl_gb300", "csrc")
MAIN = r"""
#include <atomic>
#include <new>
#include "host_parallel.h"
int main() {
    for (int64_t count : {0, 1, 63, 64, 65, 129, 5000}) {
        std::vector<std::atomic<int>> seen((size_t)count);
        cpdlp::parallel_for(count, [&](int64_t k) { seen[(size_t)k]++; });
        for (auto& s : seen)
            if (s != 1) return 1;
    }
    for (int64_t bad : {0, 40, 2500, 4999}) {
        std::atomic<int> ran{0};
        bool caught = false;
        try {
            cpdlp::parallel_for(5000, [&](int64_t k) {
                if (k == bad) throw std::bad_alloc();
                ran++;
            });
        } catch (const std::bad_alloc&) {
            caught = true;
        }
        if (!caught || ran >= 5000) return 2;
    }
}
"""


def test_exceptions_reach_the_caller(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.check_call(["g++", "-std=c++17", "-pthread", "-I", CSRC, str(tmp_path / "main.cpp"), "-o", exe])
    assert subprocess.run([exe]).returncode == 0
