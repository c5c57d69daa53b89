"""The division of a strip-form launch between its warps (mcv_sw_b200/csrc/mcv_cut.h)
on the host: tests/native/cut_test.cpp walks the cut as the kernels do, for one grid
and several, and requires every cell in exactly one strip and every way of cutting
seen -- equal segments, segments of two lengths, several strips to a warp, runs that
end inside a column, runs from one grid's columns into the next's."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_cell_in_one_strip(tmp_path):
    exe = tmp_path / "cut_test"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror",
                    "-I", os.path.join(ROOT, "mcv_sw_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "cut_test.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
