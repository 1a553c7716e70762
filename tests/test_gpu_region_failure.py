"""The region launches' failure path, exercised without a GPU fault: the
regions of a pass wait, within their time limit, for packets of a region that
was not launched, give up together and report through the engine's error word;
the engine's next shots are the oracle's, on the same board."""
import time

import numpy as np
import pytest

from tests.cases import make_case

pytestmark = pytest.mark.gpu


def test_packet_wait_times_out_and_engine_recovers(engine_lib, oracle):
    from psdm_b200._lib import PSDM_ERR_CUDA, PsdmError
    from psdm_b200.rtm import Engine, Params
    c = make_case(fs=1, nt=120, seed=21)
    prm = Params(dPML=c["dPML"], fs=c["fs"], strategy=c["strategy"])
    want = oracle.rtm_shot(dPML=c["dPML"], fs=c["fs"], nxSou=c["nxSou"], nySou=c["nySou"], nxRec=c["nxRec"],
                           nyRec=c["nyRec"], Data_source=c["src"], Data_target=c["tgt"], dd=c["dd"], dt=c["dt"],
                           nx=c["nx"], vp_w=c["vp_w"], added_space=c["added_space"], store_snap=1,
                           nt_snap=c["nt_taper"], nt_prop2=c["nt"], nt_taper=c["nt_taper"])

    def shot(e):
        return e.rtm_shot(prm, c["nxSou"], c["nySou"], c["nxRec"], c["nyRec"], c["src"], c["tgt"], c["dd"], c["dt"],
                          c["ny"], c["nx"], c["nx_w"], c["vp_w"], c["added_space"], 1, c["nt_taper"], c["nt_prop2"],
                          c["nt_taper"], 0, 1, 0)

    with Engine(0) as e:
        for _ in range(2):
            t = time.monotonic()
            with pytest.raises(PsdmError, match="timed out waiting for neighbouring") as ei:
                e.check_region_timeout()
            assert ei.value.code == PSDM_ERR_CUDA and 1.5 < time.monotonic() - t < 8.0
            assert np.array_equal(shot(e), want)
