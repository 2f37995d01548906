"""The flag that kernels set when they give up a wait (csrc/wait_flag.h, built
here by itself), with host code in the kernels' place: a report lasts until the
host has looked, however many kernels are queued in between."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "coolpdlp.jl_gb300", "csrc")
MAIN = r"""
#include "wait_flag.h"
int main() {
    double memory = 7.0;  // as allocated: not cleared
    cpdlp::WaitFlag f;
    if (f.take()) return 1;                     // nothing queued
    double* first = f.arm(&memory);
    if (f.take()) return 2;                     // ran, nothing to report
    first = f.arm(&memory);
    *first = 1.0;                               // the first of three gives up
    f.arm(&memory);
    f.arm(&memory);
    if (!f.take()) return 3;
    f.arm(&memory);
    return f.take() ? 4 : 0;                    // told once
}
"""


def test_a_later_kernel_does_not_erase_a_report(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.check_call(["g++", "-std=c++17", "-I", CSRC, str(tmp_path / "main.cpp"), "-o", exe])
    assert subprocess.run([exe]).returncode == 0
