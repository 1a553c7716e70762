"""Launches whose blocks wait for one another, from any engine, stream and
thread of a process (psdm::CoopLedger): those that may run side by side never
hold more blocks together than the device has, every launch gets its turn, and
small ones do run side by side.  tests/coop_order_check.cpp is compiled against
the engine's headers and run here, without a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("cooporder") / "coop_order_check")
    r = subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I",
                        os.path.join(ROOT, "psdm_b200", "csrc"), os.path.join(ROOT, "tests", "coop_order_check.cpp"),
                        "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return out


@pytest.mark.parametrize("wide", [0, 1])
@pytest.mark.parametrize("streams,most", [(1, 148), (3, 148), (8, 30), (8, 60), (24, 24), (12, 100)])
def test_side_by_side_launches_fit_the_device(checker, streams, most, wide):
    for seed in range(8):
        r = subprocess.run([checker, "148", str(streams), str(most), "400", str(seed), str(wide)], capture_output=True,
                           text=True, timeout=60)
        worst, never, side, ids = (int(v) for v in r.stdout.split())
        assert worst <= 148 and never == 0 and ids <= 148, r.stdout
        if streams >= 8 and most <= 30 and not wide:
            assert side >= 4, r.stdout
