"""CPU tests of code of the kernels and of their host side in orders of events that a GPU
run cannot be made to take (tests/emulation): lanes of a warp that advance one at a
time, a preview beside the kernel that adds up the tally's copies.  The code is compiled
for the host from the library's own headers."""
from __future__ import annotations

import subprocess
from pathlib import Path

REPO = Path(__file__).resolve().parents[1]


def _run(name, tmp_path):
    exe = tmp_path / name
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-pthread", "-Wno-unknown-pragmas", f"-I{REPO / 'dxmclib_gb300' / 'csrc'}", f"-I{REPO / 'tests' / 'emulation'}",
                        str(REPO / "tests" / "emulation" / f"{name}.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_work_units_are_taken_whatever_the_order_of_the_lanes(tmp_path):
    _run("work_split_check", tmp_path)


def test_shell_sums_are_in_the_precision_of_the_kernel(tmp_path):
    """Kernels in double sum the shells' weights in double, below and above the
    material's highest binding energy; kernels in single precision take the LUT's sums."""
    _run("shells_check", tmp_path)


def test_preview_counts_no_copy_twice(tmp_path):
    _run("preview_check", tmp_path)


def test_team_of_threads_where_memory_runs_out(tmp_path):
    """Fewer threads do the same work; the C ABI never ends the process for want of memory."""
    _run("worker_team_check", tmp_path)
