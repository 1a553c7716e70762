"""The slots that keep the region plans (psdm::KeyedSlots, two per shot of the
largest group): a group's plans stay its own until the whole group is
prepared, whatever was asked for before it; keys that recur within the last 32
are not made again.  tests/plan_slots_check.cpp is compiled against the
engine's headers and run here, without a GPU."""
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
    out = str(tmp_path_factory.mktemp("planslots") / "plan_slots_check")
    r = subprocess.run([cxx, "-O1", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I",
                        os.path.join(ROOT, "psdm_b200", "csrc"), os.path.join(ROOT, "tests", "plan_slots_check.cpp"),
                        "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return out


@pytest.mark.parametrize("keys,groups,fixed", [(48, 0, 1), (33, 5000, 0), (60, 5000, 0), (1000, 2000, 1)])
def test_a_group_keeps_its_plans(checker, keys, groups, fixed):
    r = subprocess.run([checker, str(keys), str(groups), str(fixed)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.split()[0] == "0", r.stdout


def test_recurring_plans_are_made_once(checker):
    r = subprocess.run([checker, "32", "500", "0"], capture_output=True, text=True, timeout=60)
    assert r.stdout.split() == ["0", "32"], r.stdout
