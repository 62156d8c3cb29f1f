"""The shared copy of a finished image in children forked while other threads use
it (mk::copy_out): every child ends, with its bytes."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_children_forked_while_others_copy(tmp_path):
    exe = tmp_path / "copy_fork_check"
    csrc = ROOT / "monkeygl_b200" / "csrc"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", f"-I{csrc}", "-I/usr/local/cuda/include",
                    str(ROOT / "tests" / "native" / "copy_fork_check.cpp"), str(csrc / "host_copy.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
