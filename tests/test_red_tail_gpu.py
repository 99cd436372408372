"""The rms an update leaves to the next kernel (knob red_tail), where the
number of block partials or the place of the fold could go wrong.  With the
knob at 0 each update folds its own partials in the same order, so every rms
must be equal bit for bit."""
import numpy as np
import pytest

from oplus2_matlab_b200 import api, apps
from oplus2_matlab_b200 import mesh as M

pytestmark = pytest.mark.gpu

STAGE = ("res_calc", "bres_calc", "update")


@pytest.fixture(autouse=True)
def knobs():
    yield
    api.lib().op2b_set_tuning(b"red_tail", 1)
    api.set_gbl_deferred(0)


def start(mesh, dt, strategy, tail):
    api.set_strategy(strategy)
    api.lib().op2b_set_tuning(b"red_tail", tail)
    # every cell's residual well away from zero, so that each partial counts
    n, rng = mesh.ncell, np.random.default_rng(5)
    qinf = np.asarray(apps.airfoil_consts(dt)["qinf"], dt)
    q = qinf * (1 + rng.uniform(-0.01, 0.01, (n, 4)))
    return apps.Airfoil(mesh, dt, state=dict(q=q, qold=q, res=np.zeros((n, 4)), adt=np.ones(n)))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("strategy", [api.STRATEGY_GATHER, api.STRATEGY_COLOURED])
def test_graph_launched_when_res_is_not_zero(op2, dt, strategy):
    """Two stages with adt frozen, captured while res is known zero and
    launched after res_calc and bres_calc alone wrote it: the launch puts the
    update that reads res in the captured one's place, and the flux pass
    behind it folds the partials of that one.  86,400 cells: more than both
    fit in one wave of CTAs."""
    mesh = M.naca0012(180, 160)
    lib = api.lib()

    def run(tail):
        A = start(mesh, dt, strategy, tail)
        A.iterate(2)
        api.sync()
        assert lib.op2b_capture_begin(0) == 1, api.last_error()
        for nm in STAGE + STAGE:
            A.loop(nm)
        h = lib.op2b_capture_end()
        assert h, api.last_error()
        out = []
        for disturbed in (False, True, True, False):
            if disturbed:
                A.loop("res_calc")
                A.loop("bres_calc")
                api.sync()
            A.rms[0] = 0
            assert lib.op2b_graph_launch(h) == 0, api.last_error()
            api.sync()
            out.append(float(A.rms[0]))
        lib.op2b_graph_destroy(h)
        return out

    want = run(0)
    api.op_exit()
    api.op_init([], 0)
    assert run(1) == want
