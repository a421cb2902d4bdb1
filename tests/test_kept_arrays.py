"""The arrays kept between differentiable sessions (sphere_b200/csrc/kept.h), on the
host: taken back by their owner, freed once for whoever runs out of memory, never
past their limit, from several threads."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent
HERE = Path(__file__).resolve().parent


def test_kept_arrays_come_back_or_are_given_back(tmp_path):
    exe = tmp_path / "kept_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", str(ROOT / "sphere_b200" / "csrc"),
                    str(HERE / "kept_check.cpp"), "-o", str(exe)], check=True)
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0 and res.stdout == "", res.stdout + res.stderr
