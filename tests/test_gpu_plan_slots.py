"""Batches on an engine that has planned more grids than it keeps plans for:
groups of one window planned long ago and new ones, and the same batches
again, every image equal to the shot alone."""
import numpy as np
import pytest

from tests.cases import make_case

pytestmark = pytest.mark.gpu


def _case(k, nt):
    return make_case(ny=30, nx_model=400, nt=nt, dPML=8, fs=1, strategy=1, nrec=14 + k, rec_step=4, near=4, sou_x=340,
                     seed=k)


def _single(e, prm, c, src):
    return e.rtm_shot(prm, c["nxSou"], c["nySou"], c["nxRec"], c["nyRec"], src[:c["nt"]], c["tgt"], c["dd"], c["dt"],
                      c["ny"], c["nx"], c["nx_w"], c["vp_w"], c["added_space"], 1, c["nt_taper"], c["nt_prop2"],
                      c["nt_taper"], 0, 1, 0)


def test_groups_of_old_and_new_windows(engine_lib):
    from psdm_b200.rtm import Engine, Params
    cs = [_case(k, 60) for k in range(44)]
    assert len({c["nx_w"] for c in cs}) == len(cs)
    src = cs[0]["src"]
    prm = Params(dPML=8, fs=1, strategy=1)
    with Engine(0) as alone:
        want = [_single(alone, prm, c, src) for c in cs]
    c0 = cs[0]

    def batch(e, ks):
        descs = [dict(nxSou=cs[k]["nxSou"], nySou=cs[k]["nySou"], nxRec=cs[k]["nxRec"], nyRec=cs[k]["nyRec"],
                      nx_w=cs[k]["nx_w"], nt_prop2=60, nt_taper=60, Vp_w=cs[k]["vp_w"], Data_target=cs[k]["tgt"])
                 for k in ks]
        got = e.rtm_batch(prm, descs, src, c0["dd"], c0["dt"], c0["ny"], c0["nx"], c0["added_space"], 1, 0, 1, 0)
        for k, img in zip(ks, got):
            bad = np.flatnonzero(~(img == want[k]))
            assert bad.size == 0, f"window {k}: {bad.size} of {img.size} values differ"

    with Engine(0) as e:
        for k in range(32):  # a plan each
            batch(e, [k])
        rng = np.random.default_rng(5)
        for first in range(8):  # the oldest windows beside ones that are new or long gone
            batch(e, [first, 43 - first, 32 + first // 2])
        for _ in range(12):
            batch(e, rng.choice(len(cs), size=int(rng.integers(2, 7)), replace=False).tolist())
