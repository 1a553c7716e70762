"""Host-array batches whose shots take different routes: windows that fit the
region form run as region launches, and from the first one that does not on,
the rest runs as a work list on the same slots.  Every image must be that of
the shot alone, whichever route it took and whatever its slot held before;
more shots than slots, so that slots of both routes are refilled."""
import numpy as np
import pytest

from tests.cases import make_case

pytestmark = pytest.mark.gpu

KW = dict(ny=500, nx_model=5400, dPML=8, fs=1, strategy=1, sou_x=5300, sou_z=3, rec_z=2)
NARROW = [dict(nt=50 + 7 * k, nrec=20 + 3 * k, rec_step=2 + k, seed=k) for k in range(5)]
WIDE = dict(nt=44, nrec=100, rec_step=50, seed=9)  # ~2.7 M padded cells


@pytest.fixture(scope="module")
def shots():
    narrow = [make_case(**KW, **g) for g in NARROW]
    return narrow[:2] + [make_case(**KW, **WIDE)] + narrow[2:]


@pytest.fixture(scope="module")
def engine():
    from psdm_b200.rtm import Engine
    with Engine(0) as e:
        yield e


def _single(e, prm, c, src, ks):
    return e.rtm_shot(prm, c["nxSou"], c["nySou"], c["nxRec"], c["nyRec"], src[:c["nt"]], c["tgt"], c["dd"], c["dt"],
                      c["ny"], c["nx"], c["nx_w"], c["vp_w"], c["added_space"], ks, c["nt_taper"], c["nt_prop2"],
                      c["nt_taper"], 0, 1, 0)


@pytest.mark.parametrize("order", ["mixed", "wide_last"])
@pytest.mark.parametrize("precision,ks,slots", [(0, 1, 1), (0, 1, 2), (1, 4, 2)])
def test_batch_of_both_routes_matches_single_shots(engine, shots, order, precision, ks, slots):
    from psdm_b200.rtm import Params
    cs = shots if order == "mixed" else shots[:2] + shots[3:] + shots[2:3]
    c0 = cs[0]
    prm = Params(dPML=c0["dPML"], fs=c0["fs"], strategy=c0["strategy"], precision=precision)
    src = max((c["src"] for c in cs), key=len)
    descs = [dict(nxSou=c["nxSou"], nySou=c["nySou"], nxRec=c["nxRec"], nyRec=c["nyRec"], nx_w=c["nx_w"],
                  nt_prop2=c["nt_prop2"], nt_taper=c["nt_taper"], Vp_w=c["vp_w"], Data_target=c["tgt"]) for c in cs]
    engine.reset_stats()
    got = engine.rtm_batch(prm, descs, src, c0["dd"], c0["dt"], c0["ny"], c0["nx"], c0["added_space"], ks, 0, 1, 0,
                           max_slots=slots)
    assert engine.batch_slots() == slots
    assert engine.stats()["launches"] >= 2 * (WIDE["nt"] - 1)  # the wide shot took a launch a step
    for i, (c, img) in enumerate(zip(cs, got)):
        want = _single(engine, prm, c, src, ks)
        assert np.abs(want).max() > 0
        bad = np.flatnonzero(~(img == want))
        assert bad.size == 0, f"shot {i}: {bad.size} of {img.size} values differ"
