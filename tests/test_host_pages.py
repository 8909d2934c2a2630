"""Pages of host result arrays (csrc/host_pages.h)."""
import subprocess

from conftest import ROOT


def test_pages_are_brought_in_and_given_up(tmp_path):
    """A waited-for array has its pages and contents; one whose solve failed keeps
    most of its pages absent."""
    exe = tmp_path / "host_pages_check"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(ROOT / "fastapsp_gb300" / "csrc"),
                        str(ROOT / "tests" / "host_pages_check.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "OK" in r.stdout, r.stdout + r.stderr
