"""Which systems the resident solver kernels take, checked on the CPU
(persist_rule_check.cu)."""
import subprocess
from pathlib import Path

import pytest

from test_band_plan import CSRC, _nvcc

HERE = Path(__file__).resolve().parent


def test_resident_solvers_end_where_launches_are_faster(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("no nvcc")
    exe = tmp_path / "persist_rule_check"
    p = subprocess.run([nvcc, "-std=c++17", "-O1", "-Wno-deprecated-gpu-targets", "--expt-relaxed-constexpr",
                        "-gencode", "arch=compute_100a,code=sm_100a", f"-I{CSRC}", f"-I{CSRC.parents[1] / 'include'}",
                        str(HERE / "persist_rule_check.cu"), "-o", str(exe)], capture_output=True, text=True,
                       timeout=600)
    assert p.returncode == 0, p.stderr[-2000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
