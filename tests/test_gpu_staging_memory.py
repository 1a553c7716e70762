"""Device memory of 16-bit batches whose FP32 snapshots are staged: what an
engine holds after batches of one to four shots is what it holds after the one
of four, whatever the sizes of the groups before (the staging is one buffer of
512 MB at most, inside the 1 GB that the memory plan leaves free)."""
import numpy as np
import pytest

from tests.cases import make_case

pytestmark = pytest.mark.gpu


def _batch(e, c, n):
    from psdm_b200.rtm import Params
    d = dict(nxSou=c["nxSou"], nySou=c["nySou"], nxRec=c["nxRec"], nyRec=c["nyRec"], nx_w=c["nx_w"],
             nt_prop2=c["nt_prop2"], nt_taper=c["nt_taper"], Vp_w=c["vp_w"], Data_target=c["tgt"])
    prm = Params(dPML=c["dPML"], fs=c["fs"], strategy=c["strategy"], precision=1)
    return e.rtm_batch(prm, [d] * n, c["src"], c["dd"], c["dt"], c["ny"], c["nx"], c["added_space"], 1, 0, 1, 0,
                       max_slots=4)


def test_batches_of_all_sizes_share_one_staging_buffer(engine_lib):
    from psdm_b200.rtm import Engine, plan_memory, Params
    # 3000 FP32 snapshots of 200 x 252 cells: 600 MB a shot
    c = make_case(ny=200, nx_model=400, nt=3001, dPML=40, fs=1, strategy=1, nrec=60, sou_x=300, added_space=640.0)
    with Engine(0) as once, Engine(0) as often:
        want = _batch(once, c, 4)
        assert once.batch_slots() == 4 and np.abs(want[0]).max() > 0
        for n in (1, 2, 3, 4):
            for img in _batch(often, c, n):
                assert np.array_equal(img, want[0]), n
        plan = plan_memory(Params(dPML=40, fs=1, strategy=1, precision=1), c["ny"], c["nx_w"], c["nt"], c["nt"], 1,
                           len(c["nxRec"]), 1 << 37)
        print(once.device_bytes(), often.device_bytes(), 4 * plan["bytes_per_slot"])
        assert often.device_bytes() - once.device_bytes() < 64 << 20
        assert often.device_bytes() < 4 * plan["bytes_per_slot"] + (1 << 30)
