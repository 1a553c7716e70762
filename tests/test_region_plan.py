"""The region form's planner on the CPU: psdm::plan_regions covers every live
cell of the padded grid by exactly one region within the shared-memory limit,
one exchange of its packets fills every ring cell that a neighbour owns (and
leaves rows above a free surface and cells outside the grid at zero), the
stencils of the cells updated before the ring arrives end inside the region,
and
psdm::region_loads names each injection point and receiver in the region that
owns it.  tests/region_plan_check.cpp is compiled against the built engine
library and run here, without a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def checker(engine_lib, tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("regionplan") / "region_plan_check")
    libdir = os.path.join(ROOT, "psdm_b200", "lib")
    cmd = [cxx, "-O1", "-std=c++17", "-I", os.path.join(ROOT, "include"), "-I",
           os.path.join(ROOT, "psdm_b200", "csrc"), os.path.join(ROOT, "tests", "region_plan_check.cpp"), "-o", out,
           "-L", libdir, "-lpsdm_rtm", "-Wl,-rpath," + libdir]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    return out


FLOATS = 57500  # a B200 block's dynamic shared memory beside the kernel's own


@pytest.mark.parametrize("ny,nx,dPML,fs,regions", [
    (3, 14, 8, 0, 148),        # the fewest rows
    (36, 59, 8, 0, 148),
    (41, 97, 9, 1, 148),       # ny and dn not multiples of 4
    (150, 317, 11, 0, 148),
    (200, 228, 40, 1, 148),
    (331, 321, 25, 0, 37),     # a quarter of the device
    (1200, 1136, 50, 1, 148),
    (1199, 1137, 50, 0, 148),
    (1500, 1210, 40, 1, 148),
    (200, 400, 12, 1, 148),    # corners cut to their narrowest columns
])
def test_regions_cover_grid_and_exchange_rings(checker, ny, nx, dPML, fs, regions):
    r = subprocess.run([checker, *map(str, (ny, nx, dPML, fs, regions, FLOATS))], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, r.stderr
    got = [int(v) for v in r.stdout.split()]
    assert got[0] == 1 and 1 <= got[1] <= regions, got
    assert got[2:] == [0, 0, 0, 0, 0], got


def test_regions_refuse_grids_that_do_not_fit(checker):
    for ny, nx, dPML, regions in ((2, 40, 8, 148), (3000, 2620, 50, 148), (1200, 1136, 50, 4)):
        r = subprocess.run([checker, *map(str, (ny, nx, dPML, 1, regions, FLOATS))], capture_output=True, text=True)
        assert r.returncode == 0 and r.stdout.split() == ["0"], (ny, nx, r.stdout)
