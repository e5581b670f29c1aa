"""The page-locked block that a call's new rows pass through: no place is given out again before a wait that covers its kernel."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_place_is_reused_before_a_wait_that_covers_it(tmp_path):
    exe = str(tmp_path / "host_ring_test")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I", os.path.join(ROOT, "relux_b200", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "host_ring_test.cpp"), "-o", exe])
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr
