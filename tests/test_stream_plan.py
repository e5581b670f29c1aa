"""The plan that the latent decode kernel runs: its items cover every page once, every worker's are its own, and the counts that the host
hands to the launch are those of the device's builder; which calls go in pieces and which in ranges."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("plan") / "stream_plan_test")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Werror", "-I", os.path.join(ROOT, "relux_b200", "csrc"),
                           os.path.join(ROOT, "tests", "cpp", "stream_plan_test.cpp"), "-o", path])
    return path


def test_items_of_random_calls(exe):
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.stdout + out.stderr


@pytest.mark.parametrize("tokens,workers,plan", [
    ([300], 74, "pieces"), ([64, 65, 128, 129], 74, "pieces"), ([600] * 9, 74, "pieces"), ([129] * 38, 74, "ranges"), ([4096] * 64, 74, "pieces"),
    ([200] * 75, 74, "ranges"), ([2000] * 20, 74, "ranges"), ([32768] * 64, 74, "ranges"), ([1500, 100, 900], 18, "pieces"), ([0, 0], 74, "ranges")])
def test_which_plan_a_call_gets(exe, tokens, workers, plan):
    pages = [str((t + 63) // 64) for t in tokens]
    out = subprocess.run([exe, str(workers)] + pages, capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.split()[0] == plan, out.stdout


def test_scratch_serves_both_plans(exe):
    """64 sequences that grow from one plan into the other: what the call after the change needs is there already, but for the few items
    by which ranges change from length to length."""
    plans = []
    for pages in range(20, 560, 4):
        out = subprocess.run([exe, "74"] + [str(pages)] * 64, capture_output=True, text=True, timeout=60).stdout.split()
        plans.append((out[0], int(out[3]), int(out[4])))
    borders = [(a, b) for a, b in zip(plans, plans[1:]) if a[0] != b[0]]
    assert borders
    for (_, _, room), (_, items, _) in borders:
        assert items <= room + 10
