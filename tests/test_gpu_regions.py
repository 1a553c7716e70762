"""Passes as region launches (the engine's own choice until a launch form is
set) against one launch per time step: images, receiver traces and snapshots
bit for bit, over windows whose rows, columns and C-PML width leave partial
float4s, one region or many, injection rows at the edges of regions, both
statement orders and both kinds of surface.  The launch counts show which
form ran."""
import numpy as np
import pytest

from tests.cases import make_case

pytestmark = pytest.mark.gpu

CASES = [
    dict(ny=9, nx_model=60, nt=120, dPML=8, fs=0, strategy=2, nrec=9, sou_x=40, sou_z=2, rec_z=2, seed=1),
    dict(ny=37, nx_model=90, nt=200, dPML=8, fs=1, strategy=1, seed=2, collide=True),
    dict(ny=64, nx_model=150, nt=170, dPML=11, fs=0, strategy=1, nrec=40, sou_x=120, sou_z=33, rec_z=64, seed=3),
    dict(ny=129, nx_model=330, nt=140, dPML=25, fs=1, strategy=2, nrec=90, sou_x=280, sou_z=110, rec_z=129, seed=4,
         taper_option=1, N_taper=30, N_zeros=12),
    dict(ny=261, nx_model=700, nt=110, dPML=41, fs=1, strategy=1, nrec=200, rec_step=3, sou_x=660, sou_z=2, rec_z=3,
         seed=5),
    dict(ny=502, nx_model=420, nt=90, dPML=30, fs=0, strategy=1, nrec=120, rec_step=2, sou_x=330, sou_z=250,
         rec_z=251, seed=6),
]


@pytest.fixture(scope="module")
def engines():
    from psdm_b200.rtm import Engine
    auto, steps = Engine(0), Engine(0)
    steps.set_pass_launch(0)
    yield auto, steps
    auto.close()
    steps.close()


def _prm(c):
    from psdm_b200.rtm import Params
    return Params(dPML=c["dPML"], fs=c["fs"], strategy=c["strategy"])


def _shot(e, c):
    return e.rtm_shot(_prm(c), c["nxSou"], c["nySou"], c["nxRec"], c["nyRec"], c["src"], c["tgt"], c["dd"], c["dt"],
                      c["ny"], c["nx"], c["nx_w"], c["vp_w"], c["added_space"], 1, c["nt_taper"], c["nt_prop2"],
                      c["nt_taper"], c["taper_option"], c["N_taper"], c["N_zeros"])


def _forward(e, c):
    F = np.zeros((c["nt"], c["nx_w"], c["ny"]), np.float32)
    rec = np.zeros((c["nxRec"].size, c["nt"]), np.float32)
    e.dynamic_window_solver_forward_ram(_prm(c), [c["nxSou"]], [c["nySou"]], c["nxRec"], c["nyRec"], c["src"], c["dd"],
                                        c["dt"], c["ny"], c["nx"], c["nx_w"], c["vp_w"], c["added_space"], 1, c["nt"],
                                        c["nt"], Fields=F, Data_synth=rec)
    return F, rec


def _same(a, b, what):
    assert a.shape == b.shape and np.abs(b).max() > 0, what
    bad = np.flatnonzero(~(a == b))
    assert bad.size == 0, f"{what}: {bad.size} of {a.size} values differ (first at flat {bad[:1]})"


@pytest.mark.parametrize("ci", range(len(CASES)))
def test_regions_match_steps(engines, ci):
    auto, steps = engines
    c = make_case(**CASES[ci])
    for fn, what in ((_shot, ("image",)), (_forward, ("snapshots", "traces"))):
        got = []
        for e in (auto, steps):
            e.reset_stats()
            r = fn(e, c)
            got.append((r if isinstance(r, tuple) else (r,), e.stats()["launches"]))
        assert got[0][1] < 20 and got[1][1] >= c["nt"] - 1, (got[0][1], got[1][1])
        for a, b, w in zip(got[0][0], got[1][0], what):
            _same(a, b, w)


def _batch(e, cs, precision, ks):
    from psdm_b200.rtm import Params
    c0 = cs[0]
    prm = Params(dPML=c0["dPML"], fs=c0["fs"], strategy=c0["strategy"], precision=precision)
    shots = [dict(nxSou=c["nxSou"], nySou=c["nySou"], nxRec=c["nxRec"], nyRec=c["nyRec"], nx_w=c["nx_w"],
                  nt_prop2=c["nt_prop2"], nt_taper=c["nt_taper"], Vp_w=c["vp_w"], Data_target=c["tgt"]) for c in cs]
    src = max((c["src"] for c in cs), key=len)
    return e.rtm_batch(prm, shots, src, c0["dd"], c0["dt"], c0["ny"], c0["nx"], c0["added_space"], ks,
                       c0["taper_option"], c0["N_taper"], c0["N_zeros"])


@pytest.mark.parametrize("precision,ks", [(0, 1), (1, 1), (1, 4), (2, 3)])
def test_regions_batch_match_steps(engines, precision, ks):
    """Shots of different windows and records side by side, and one shot in each precision alone."""
    auto, steps = engines
    for n in (5, 1):
        cs = [make_case(ny=45, nx_model=400, nt=160 + 17 * k, dPML=10, fs=1, strategy=1, nrec=20 + 9 * k, rec_step=2,
                        sou_x=200 + 30 * k, sou_z=2, rec_z=2, seed=20 + k, taper_option=1, N_taper=20, N_zeros=8)
              for k in range(n)]
        got = []
        for e in (auto, steps):
            e.reset_stats()
            got.append((_batch(e, cs, precision, ks), e.stats()["launches"]))
        assert got[0][1] < 60 and got[1][1] >= 2 * 159, (got[0][1], got[1][1])
        for a, b in zip(got[0][0], got[1][0]):
            _same(a, b, "image")


@pytest.mark.parametrize("interval", [1, 37, 199, 500])
def test_regions_checkpointed_match_steps(engines, interval):
    c = make_case(ny=61, nx_model=150, nt=200, dPML=9, fs=0, strategy=2, nrec=30, seed=8, taper_option=1, N_taper=15,
                  N_zeros=6)
    got = []
    for e in engines:
        e.set_checkpointing(interval)
        try:
            got.append(_shot(e, c))
        finally:
            e.set_checkpointing(0)
    _same(got[0], got[1], "image")
    _same(got[0], _shot(engines[0], c), "image of the shot that keeps every snapshot")
