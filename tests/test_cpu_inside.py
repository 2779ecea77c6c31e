"""The cull's inside proof (compute_rasterizer_gb300/csrc/cr_inside.h) never holds
for a box with a point that projects outside the view, transforms with infinite or
NaN entries included (tests/cpp/inside_check.cpp)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_inside_proof_is_sound(tmp_path):
    exe = tmp_path / "inside_check"
    cmd = ["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-Wno-unknown-pragmas",
           "-ffp-contract=off", "-fno-fast-math", str(ROOT / "tests" / "cpp" / "inside_check.cpp"),
           "-o", str(exe)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe), "400000"], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    proofs, special, _ = (int(x) for x in res.stdout.split())
    assert proofs > 10_000 and special > 90_000
