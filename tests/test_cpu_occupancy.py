"""The kept occupancy answers (compute_rasterizer_gb300/csrc/cr_occupancy.h): a
failed driver query does not stay, and devices do not share an answer."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_failed_answer_is_not_kept(tmp_path):
    exe = tmp_path / "occupancy_check"
    cmd = ["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror",
           str(ROOT / "tests" / "cpp" / "occupancy_check.cpp"), "-o", str(exe)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout
