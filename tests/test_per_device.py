"""Kernel attributes belong to a device: what a call site has set is kept per device
(csrc/qg_perdev.h).  Host-only: the bookkeeping is compiled on its own."""
import re
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "query_on_opencl_fpga_gb300" / "csrc"

PROGRAM = r"""
#include "qg_perdev.h"
#include <stdio.h>
#include <thread>
static qg_per_device a, b[2];
int main() {
    if (a.covers(0, 1) || !a.covers(0, 0)) return 1;            // nothing set yet
    a.set(0, 100);
    if (!a.covers(0, 100) || a.covers(0, 101)) return 2;         // the value set, no more
    if (a.covers(1, 1) || b[0].covers(0, 1)) return 3;           // neither another device nor another site
    a.set(0, 50);
    if (!a.covers(0, 100)) return 4;                             // never less
    a.set(63, 7);
    if (!a.covers(63, 7) || a.covers(62, 1)) return 5;
    a.set(64, 9);                                                // beyond the table: set each time
    a.set(-1, 9);
    if (a.covers(64, 1) || a.covers(-1, 1) || a.covers(63, 8)) return 6;
    std::thread t[4];
    for (int i = 0; i < 4; i++) t[i] = std::thread([i] { for (int k = 0; k < 10000; k++) b[1].set(5, 4 * k + i); });
    for (auto &x : t) x.join();
    return b[1].covers(5, 39999) && !b[1].covers(5, 40000) ? 0 : 7;
}
"""


def test_values_are_kept_per_site_and_device(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", f"-I{CSRC}", str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0


def test_kernel_attributes_go_through_it():
    # one call in the helper, and one that is made each time a batch is created
    calls = {f.name: len(re.findall(r"cudaFuncSetAttribute\(", f.read_text())) for f in CSRC.iterdir() if f.is_file()}
    assert {k: v for k, v in calls.items() if v} == {"qg_internal.cuh": 1, "qg_bpersist.cu": 1}
