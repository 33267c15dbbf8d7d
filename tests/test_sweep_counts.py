"""Sweeps of a cadence are counted on the host and reach the device's sweep
counter later.  When a launch fails part way, the sweeps already launched must
still be counted (a caller that goes on would otherwise draw their stream
words again), and those of a failed capture, which never ran, must not.  The
counting is compiled for the host with stand-ins for its two launches."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SOURCE = r"""
#include "ym_internal.hpp"
#include <cstdio>

static long counted = 0;   // what the device's counter has received
namespace ym {
cudaError_t launch_counted_sweeps(ym_ensemble *e) {
    counted += e->sweep_slot;
    e->sweep_slot = 0;
    return cudaSuccess;
}
cudaError_t launch_advance_sweep(ym_ensemble *e) {
    ++e->sweep_slot;
    return launch_counted_sweeps(e);
}
}

// n sweeps, then a launch that fails
template <class Scope>
static cudaError_t cadence(ym_ensemble *e, int n) {
    const Scope scope(e);
    for (int k = 0; k < n; ++k)
        if (cudaError_t err = ym::count_sweep(e)) return err;
    return cudaErrorLaunchFailure;
}

int main() {
    for (int n : {0, 1, 31, 32, 33, 70}) {
        ym_ensemble e;
        counted = 0;
        cadence<ym::SCOPE>(&e, n);
        std::printf("%d %ld %d\n", n, counted, e.sweep_slot);
    }
}
"""


def _run(tmp_path, scope):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src = tmp_path / "counts.cu"
    src.write_text(SOURCE)
    exe = str(tmp_path / "counts")
    subprocess.run([nvcc, "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", f"-DSCOPE={scope}",
                    "-I", os.path.join(ROOT, "yang-mills_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    str(src), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    return [tuple(int(v) for v in line.split()) for line in out.splitlines()]


def test_launched_sweeps_are_counted_after_a_failed_launch(tmp_path):
    for n, counted, left in _run(tmp_path, "SweepSlotScope"):
        assert (counted, left) == (n, 0)


def test_sweeps_of_a_failed_capture_are_not(tmp_path):
    # a cadence of 32 sweeps or more advances the counter inside the capture
    for n, counted, left in _run(tmp_path, "CapturedSweeps"):
        assert (counted, left) == (n // 32 * 32, 0)
