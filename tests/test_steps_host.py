"""The index steps of the kernels that read several strides ahead, compiled for the host: ranges that end at
INT_MAX are walked whole, with no signed overflow (CPU test)."""
import os
import subprocess

from conftest import PKG_DIR, ROOT


def test_steps_up_to_int_max(tmp_path):
    exe = str(tmp_path / "steps_check")
    src = os.path.join(ROOT, "tests", "native", "steps_check.cpp")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-x", "c++", "-fsanitize=signed-integer-overflow",
                           "-fsanitize-undefined-trap-on-error", "-I", os.path.join(PKG_DIR, "csrc"), src, "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.startswith("ok")
