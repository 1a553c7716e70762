"""The snapshots of the region launches, (p3 - p1) * 0.5 / dt, against the
IEEE FP32 expression (numpy's, every operation rounded to nearest) and against
the step kernels', bit for bit: over every binary exponent, both signs, signed
zeros, halved subnormals (the smallest one rounds to a zero that keeps the
sign), ties between subnormal quotients, infinities and NaN; and the whole
wavefield of a shot, whose onset is full of such values."""
import numpy as np
import pytest

from tests.cases import make_case
from tests.test_gpu_dt_quotients import DTS, _inputs, _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", DTS + [2.0, 0.1])
@pytest.mark.parametrize("form", ["twice", "alone", "mixed"])
def test_region_snapshot_is_the_ieee_expression(engine, dt, form):
    x = _inputs(dt, seed=int(dt * 1e7) + 1)
    if form == "twice":  # p3 - p1 = 2 x: every x is a halved difference
        p3, p1 = x, -x
    elif form == "alone":  # halves of subnormals round
        p3, p1 = x, np.zeros_like(x)
    else:
        p3, p1 = x, np.roll(x, 5)
    with np.errstate(all="ignore"):
        want = ((p3 - p1) * np.float32(0.5) / np.float32(dt)).astype(np.float32)
    _same(engine.snapshot_quotients(dt, p3, p1), want)


def test_region_snapshot_rejects_ragged_input(engine):
    from psdm_b200._lib import PsdmError
    with pytest.raises(PsdmError):
        engine.snapshot_quotients(1e-3, np.ones(6, np.float32), np.ones(6, np.float32))


@pytest.mark.parametrize("kw", [dict(ny=37, nx_model=90, nt=200, dPML=8, fs=1, strategy=1, seed=2),
                                dict(ny=64, nx_model=150, nt=170, dPML=11, fs=0, strategy=2, nrec=40, sou_x=120,
                                     sou_z=33, rec_z=64, seed=3)])
def test_region_wavefield_has_the_step_kernels_bits(engine_lib, kw):
    from psdm_b200.rtm import Engine, Params
    c = make_case(**kw)
    prm = Params(dPML=c["dPML"], fs=c["fs"], strategy=c["strategy"])
    got = []
    for form in (None, 0):
        with Engine(0) as e:
            if form is not None:
                e.set_pass_launch(form)
            F = np.zeros((c["nt"], c["nx_w"], c["ny"]), np.float32)
            e.dynamic_window_solver_forward_ram(prm, [c["nxSou"]], [c["nySou"]], c["nxRec"], c["nyRec"], c["src"],
                                                c["dd"], c["dt"], c["ny"], c["nx"], c["nx_w"], c["vp_w"],
                                                c["added_space"], 1, c["nt"], c["nt"], Fields=F)
            got.append(F)
    assert (np.signbit(got[1]) & (got[1] == 0)).any()  # zeros with a sign among them
    bad = np.flatnonzero(got[0].view(np.uint32) != got[1].view(np.uint32))
    assert bad.size == 0, f"{bad.size} of {got[0].size} differ in their bits"
