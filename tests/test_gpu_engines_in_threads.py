"""Several engines of one process at work at once, a thread and a stream each,
whose launches' blocks wait for one another: the engine's own choice on
windows that take part of the device and all of it, both explicit forms of one
launch a pass, and a window too large for any of them.  Every image must be
that of the engine alone."""
import threading

import numpy as np
import pytest

from tests.cases import make_case

pytestmark = pytest.mark.gpu

SMALL = dict(ny=36, nx_model=90, nt=200, dPML=8, fs=0, strategy=1, seed=1)
MIDDLE = dict(ny=150, nx_model=420, nt=200, dPML=20, fs=1, strategy=1, nrec=60, rec_step=3, sou_x=380,
              added_space=200.0, seed=4)
LARGE = dict(ny=500, nx_model=800, nt=150, dPML=30, fs=1, strategy=1, nrec=150, rec_step=4, sou_x=760,
             added_space=350.0, seed=5)
HUGE = dict(ny=700, nx_model=4300, nt=60, dPML=8, fs=1, strategy=1, nrec=100, rec_step=40, sou_x=4200, seed=6)


def _shot(e, c):
    from psdm_b200.rtm import Params
    prm = Params(dPML=c["dPML"], fs=c["fs"], strategy=c["strategy"])
    return e.rtm_shot(prm, c["nxSou"], c["nySou"], c["nxRec"], c["nyRec"], c["src"], c["tgt"], c["dd"], c["dt"],
                      c["ny"], c["nx"], c["nx_w"], c["vp_w"], c["added_space"], 1, c["nt_taper"], c["nt_prop2"],
                      c["nt_taper"], 0, 1, 0)


@pytest.mark.parametrize("mix", [
    [(SMALL, None)] * 8,
    [(SMALL, None), (MIDDLE, None), (MIDDLE, None), (LARGE, None), (LARGE, None)],
    [(LARGE, None), (LARGE, 2), (MIDDLE, 1), (SMALL, None), (SMALL, 2)],
    [(LARGE, None), (HUGE, None), (SMALL, None), (MIDDLE, 0)],
])
def test_engines_side_by_side_match_alone(engine_lib, mix):
    from psdm_b200.rtm import Engine
    cases = [make_case(**kw) for kw, _ in mix]
    engines = [Engine(0) for _ in mix]
    try:
        for e, (_, form) in zip(engines, mix):
            if form is not None:
                e.set_pass_launch(form)
        want = [_shot(e, c) for e, c in zip(engines, cases)]
        assert all(np.abs(w).max() > 0 for w in want)
        bad = []

        def work(k):
            try:
                for _ in range(12):
                    if not np.array_equal(_shot(engines[k], cases[k]), want[k]):
                        bad.append((k, "image differs"))
            except Exception as err:  # noqa: BLE001
                bad.append((k, err))

        threads = [threading.Thread(target=work, args=(k,)) for k in range(len(mix))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad, bad
    finally:
        for e in engines:
            e.close()
