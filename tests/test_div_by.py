"""Division by a fixed divisor (mk::div_by) equals the division, bit for bit."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_div_by_equals_division(tmp_path):
    exe = tmp_path / "div_by_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'monkeygl_b200' / 'csrc'}",
                    str(ROOT / "tests" / "native" / "div_by_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
