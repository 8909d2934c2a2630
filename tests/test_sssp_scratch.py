"""Slot counts of the batched search's scratch (csrc/sssp_scratch.h)."""
import subprocess

from conftest import ROOT


def test_slots_after_failed_growth(tmp_path):
    """A scratch buffer that failed to grow is empty: the slots it held before
    are not counted any more (the kernels would store through a null base)."""
    exe = tmp_path / "sssp_scratch_check"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "fastapsp_gb300" / "csrc"),
                        str(ROOT / "tests" / "sssp_scratch_check.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr
