"""One launch per time step on windows with more tiles than resident blocks
(where the step kernel spreads its boundary tiles over the list, takes the
interior tiles in reverse every other step and loads through the shared ring),
bit for bit against the oracle: windows that are mostly boundary tiles, mostly
interior ones, and just around one wave, FP32 and 16-bit snapshots, an odd and
an even number of steps."""
import numpy as np
import pytest

from tests.cases import make_case

pytestmark = pytest.mark.gpu


def _wide(ny, nx, nt, dPML, fs, strategy, seed, depth=2):
    return make_case(ny=ny, nx_model=nx, nt=nt, dPML=dPML, fs=fs, strategy=strategy, nrec=90,
                     rec_step=(nx - 160) // 90, sou_x=nx - 60, sou_z=depth, rec_z=depth + 1, seed=seed)


CASES = [
    dict(ny=41, nx=7300, nt=41, dPML=8, fs=0, strategy=2, seed=1, depth=20),
    dict(ny=300, nx=4900, nt=30, dPML=9, fs=1, strategy=1, seed=2),
    dict(ny=387, nx=3400, nt=31, dPML=11, fs=1, strategy=1, seed=3),
]


@pytest.fixture(scope="module")
def steps():
    from psdm_b200.rtm import Engine
    e = Engine(0)
    e.set_pass_launch(0)
    yield e
    e.close()


@pytest.mark.parametrize("precision,ks", [(0, 1), (1, 3)])
@pytest.mark.parametrize("ci", range(len(CASES)))
def test_many_tiles_match_oracle(steps, oracle, ci, precision, ks):
    from psdm_b200.rtm import Params
    c = _wide(**CASES[ci])
    prm = Params(dPML=c["dPML"], fs=c["fs"], strategy=c["strategy"], precision=precision)
    got = steps.rtm_shot(prm, c["nxSou"], c["nySou"], c["nxRec"], c["nyRec"], c["src"], c["tgt"], c["dd"], c["dt"],
                         c["ny"], c["nx"], c["nx_w"], c["vp_w"], c["added_space"], ks, c["nt_taper"], c["nt_prop2"],
                         c["nt_taper"], c["taper_option"], c["N_taper"], c["N_zeros"])
    kw = dict(dPML=c["dPML"], fs=c["fs"], nxSou=c["nxSou"], nySou=c["nySou"], nxRec=c["nxRec"], nyRec=c["nyRec"],
              Data_source=c["src"], Data_target=c["tgt"], dd=c["dd"], dt=c["dt"], nx=c["nx"], vp_w=c["vp_w"],
              added_space=c["added_space"], store_snap=ks, nt_prop2=c["nt_prop2"], nt_taper=c["nt_taper"],
              taper_option=c["taper_option"], N_taper=c["N_taper"], N_zeros=c["N_zeros"],
              disk_mode=int(c["strategy"] == 2))
    want = oracle.rtm_shot_mixed(q16=precision, kahan=1, **kw) if precision else oracle.rtm_shot(nt_snap=c["nt_taper"], **kw)
    assert got.shape == want.shape and np.abs(want).max() > 0
    bad = np.flatnonzero(~(got == want))
    assert bad.size == 0, f"{bad.size} of {got.size} values differ"
