"""The launch form of an engine can be set and taken back: one launch a step
(0), the engine's own choice (-1, which it starts with), seen in the number of
launches of the same shot, whose image does not change; other values are
refused and leave the form."""
import numpy as np
import pytest

from tests.cases import make_case

pytestmark = pytest.mark.gpu


def test_own_choice_can_be_had_back(engine_lib):
    from psdm_b200._lib import PsdmError
    from psdm_b200.rtm import Engine, Params
    c = make_case(ny=40, nx_model=120, nt=180, dPML=8, fs=1, strategy=1, seed=2)
    prm = Params(dPML=c["dPML"], fs=c["fs"], strategy=c["strategy"])
    with Engine(0) as e:
        def shot():
            e.reset_stats()
            img = e.rtm_shot(prm, c["nxSou"], c["nySou"], c["nxRec"], c["nyRec"], c["src"], c["tgt"], c["dd"], c["dt"],
                             c["ny"], c["nx"], c["nx_w"], c["vp_w"], c["added_space"], 1, c["nt_taper"], c["nt_prop2"],
                             c["nt_taper"], 0, 1, 0)
            return img, e.stats()["launches"]

        first, few = shot()
        assert np.abs(first).max() > 0 and few < 20
        for form, steps in ((0, True), (-1, False), (2, False), (0, True), (1, False), (-1, False)):
            e.set_pass_launch(form)
            img, n = shot()
            assert np.array_equal(img, first), form
            assert n >= 2 * (c["nt"] - 1) if steps else n < 20, (form, n)
            if form == -1:
                assert n == few
        for form in (-2, 3, 100):
            with pytest.raises(PsdmError):
                e.set_pass_launch(form)
        assert shot()[1] == few
