"""Passes and checkpoint segments around the fewest steps for which a region
launch is taken (2 and one more for each 120000 padded cells), seen in the
number of launches, against one launch a step bit for bit."""
import numpy as np
import pytest

from tests.cases import make_case

pytestmark = pytest.mark.gpu

SMALL = dict(ny=36, nx_model=90, dPML=8, fs=0, strategy=1)                        # 2 steps
MIDDLE = dict(ny=500, nx_model=900, dPML=30, fs=1, strategy=2, nrec=100, rec_step=5, sou_x=800,
              added_space=300.0)                                                     # 572 x 631 padded cells: 5 steps


@pytest.fixture(scope="module")
def engines():
    from psdm_b200.rtm import Engine
    auto, steps = Engine(0), Engine(0)
    steps.set_pass_launch(0)
    yield auto, steps
    auto.close()
    steps.close()


def _shot(e, c, nt, precision=0):
    from psdm_b200.rtm import Params
    prm = Params(dPML=c["dPML"], fs=c["fs"], strategy=c["strategy"], precision=precision)
    e.reset_stats()
    img = e.rtm_shot(prm, c["nxSou"], c["nySou"], c["nxRec"], c["nyRec"], c["src"][:nt], c["tgt"][:, :nt], c["dd"],
                     c["dt"], c["ny"], c["nx"], c["nx_w"], c["vp_w"], c["added_space"], 1, nt, nt, nt, 0, 1, 0)
    return img, e.stats()["launches"]


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("kw,least", [(SMALL, 2), (MIDDLE, 5)])
def test_short_shots(engines, kw, least, precision):
    auto, steps = engines
    c = make_case(nt=30, **kw)
    dn = kw["dPML"] + 6
    assert least == 2 + (kw["ny"] + 2 * dn) * (c["nx_w"] + 2 * dn) // 120000
    for nt in (2, least, least + 1, least + 2, 30):
        got, n = _shot(auto, c, nt, precision)
        want, m = _shot(steps, c, nt, precision)
        assert np.array_equal(got, want), nt
        if nt - 1 < least:
            assert n == m, (nt, n, m)  # the same launches
    assert np.abs(want).max() > 0 and n < m


@pytest.mark.parametrize("kw,least", [(SMALL, 2), (MIDDLE, 5)])
def test_short_segments(engines, kw, least):
    c = make_case(nt=61, **kw)
    for interval in (1, least - 1, least, least + 1):
        got = []
        for e in engines:
            e.set_checkpointing(interval)
            try:
                got.append(_shot(e, c, 61))
            finally:
                e.set_checkpointing(0)
        assert np.abs(got[1][0]).max() > 0 and np.array_equal(got[0][0], got[1][0]), interval
        assert (got[0][1] == got[1][1]) == (interval < least), (interval, got[0][1], got[1][1])
