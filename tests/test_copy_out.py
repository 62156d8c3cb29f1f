"""The shared copy of a finished image (mk::copy_out): sizes around its limits
and pieces, concurrent callers, a forked child."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_copy_out_copies_every_byte(tmp_path):
    exe = tmp_path / "copy_out_check"
    csrc = ROOT / "monkeygl_b200" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", f"-I{csrc}", "-I/usr/local/cuda/include",
                    str(ROOT / "tests" / "native" / "copy_out_check.cpp"), str(csrc / "host_copy.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
