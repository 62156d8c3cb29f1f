"""A run of equal float additions of the ray schedule in one step
(mk::add_steps) equals the additions one by one, bit for bit."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_add_steps_equals_single_additions(tmp_path):
    exe = tmp_path / "add_steps_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'monkeygl_b200' / 'csrc'}",
                    str(ROOT / "tests" / "native" / "add_steps_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout
