"""A small window whose record keeps more 16-bit snapshots than one launch
may convert at once (65535 rows of a grid), against the oracle's emulation bit
for bit."""
import numpy as np
import pytest

from tests.cases import make_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt", [65536, 65537, 65700])
def test_mixed_shot_with_many_snapshots(engine_lib, oracle, nt):
    from psdm_b200.rtm import Engine, Params
    c = make_case(ny=9, nx_model=60, nt=nt, dPML=8, fs=1, strategy=2, nrec=3, sou_x=30, sou_z=3, rec_z=3, added_space=20.0, seed=5)
    prm = Params(dPML=c["dPML"], fs=c["fs"], strategy=c["strategy"], precision=1)
    with Engine(0) as e:
        got = e.rtm_shot(prm, c["nxSou"], c["nySou"], c["nxRec"], c["nyRec"], c["src"], c["tgt"], c["dd"], c["dt"],
                         c["ny"], c["nx"], c["nx_w"], c["vp_w"], c["added_space"], 1, c["nt_taper"], c["nt_prop2"],
                         c["nt_taper"], 0, 1, 0)
        assert e.stats()["launches"] < 100  # region launches and conversions
    want = oracle.rtm_shot_mixed(dPML=c["dPML"], fs=c["fs"], nxSou=c["nxSou"], nySou=c["nySou"], nxRec=c["nxRec"],
                                 nyRec=c["nyRec"], Data_source=c["src"], Data_target=c["tgt"], dd=c["dd"], dt=c["dt"],
                                 nx=c["nx"], vp_w=c["vp_w"], added_space=c["added_space"], store_snap=1, nt_prop2=nt,
                                 nt_taper=nt, q16=1, kahan=1, disk_mode=1)
    assert np.isfinite(want).all() and np.abs(want).max() > 0
    bad = np.flatnonzero(~(got == want))
    assert bad.size == 0, f"{bad.size} of {got.size} values differ"
