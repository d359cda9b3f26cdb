"""The library's shared host-side bookkeeping (csrc/lbm_shared.h), compiled by
itself: set-up calls that hold for one device are made for each device, and
launches counted by one thread survive another thread's graph capture."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mpi-multi-process-version_b200", "csrc")

PROGRAM = r"""
#include "lbm_shared.h"
#include <stdio.h>
#include <thread>
enum Err { kOk = 0, kBad = 1 };
int main()
{
    lbm::OncePerDevice once;
    int calls = 0;
    auto ok = [&] { ++calls; return kOk; };
    auto bad = [&] { ++calls; return kBad; };
    if (once.run(0, bad) != kBad || once.run(0, ok) != kOk || calls != 2) return 1;       // a failure is tried again
    if (once.run(0, bad) != kOk || calls != 2) return 2;                                  // done on device 0
    if (once.run(1, ok) != kOk || calls != 3 || once.run(1, bad) != kOk || calls != 3) return 3;  // device 1: its own
    if (once.run(70, ok) != kOk || once.run(70, ok) != kOk || calls != 5) return 4;       // beyond the mask: every time
    lbm::LaunchCount n;
    n += 2;
    const int64_t mark = n.mark();
    ++n;
    std::thread other([&] { for (int k = 0; k < 1000; ++k) ++n; const int64_t m = n.mark(); n += 5; if (n.take(m) != 5) ++n; });
    n += 3;
    other.join();
    if (n.take(mark) != 4) return 5;          // this thread's own
    if (n.total() != 1002) return 6;          // the other thread's stay
    if (n.mark() != mark) return 7;
    puts("ok");
    return 0;
}
"""


def test_shared_bookkeeping(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok"


@pytest.mark.parametrize("name", ["lbm_kernels.cu", "unet_kernels.cu"])
def test_function_attributes_are_not_set_once_a_process(name):
    # a flag of the process would leave every device but the first without its kernels' shared memory
    text = open(os.path.join(CSRC, name)).read()
    assert "static bool done" not in text
