"""The plan of the pipelined triangular solves, checked on the CPU.

A solve's blocks wait on one another's progress and read x from a
shared-memory ring that is overwritten as they go.  ilu_pipe_check.cu
compiles the host-side planner of tnl_b200/csrc/ilu_pipe.cuh (no GPU
needed) and runs the plans of grids, bands and random triangles step by
step: no deadlock, every ring slot read holds the row meant, no external
value is read before its row is finished.
"""
import subprocess
from pathlib import Path

import pytest

from test_band_plan import CSRC, _nvcc

HERE = Path(__file__).resolve().parent


def test_ilu_pipe_plan_runs_to_its_end(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("no nvcc")
    exe = tmp_path / "ilu_pipe_check"
    p = subprocess.run([nvcc, "-std=c++17", "-O2", "-Wno-deprecated-gpu-targets", "--expt-relaxed-constexpr",
                        "-gencode", "arch=compute_100a,code=sm_100a", f"-I{CSRC}", str(HERE / "ilu_pipe_check.cu"),
                        "-o", str(exe)], capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.startswith("ok "), r.stdout + r.stderr
    assert int(r.stdout.split()[1]) > 1_000_000
