"""The GPU builders' quick form of the integer quantisation
(compute_rasterizer_gb300/csrc/cr_quant.h, quant_quick) agrees with quant_fast
wherever it decides, over the setups tests/cpp/quant_quick_check.cpp draws; and
it decides nearly every uniform point of those whose cells are not exact."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_quick_form_matches(tmp_path):
    exe = tmp_path / "quant_quick_check"
    cmd = ["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-ffp-contract=off",
           "-fno-fast-math", str(ROOT / "tests" / "cpp" / "quant_quick_check.cpp"), "-o", str(exe)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe), "100000"], capture_output=True, text=True, timeout=300)
    assert res.returncode == 0, res.stdout + res.stderr
    checked, uniform, decided = (int(x) for x in res.stdout.split())
    assert checked > 10**7
    # a fifth of the setups have power-of-two scales, which may leave every point
    # on a cell boundary, and georeferenced offsets widen the margin of small boxes
    assert decided > uniform // 2
