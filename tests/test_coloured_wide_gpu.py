"""COLOURED on meshes whose contribution lists cannot be had: a cell on more
edges than its list may hold (the loops run by block colours), up to more than
an ordered list can be made for at all, which COLOURED never needed.  Against
knob coloured_fold 0, fields bit for bit and the plan's count of uses."""
import numpy as np
import pytest

from oplus2_matlab_b200 import api, apps
from oplus2_matlab_b200 import mesh as M

pytestmark = pytest.mark.gpu

INDS = {"res_calc": [0, 0, 1, 1, 2, 2, 3, 3], "bres_calc": [0, 0, 1, 2, 3, -1]}


def solve(fold, mesh, dt):
    api.set_error_mode(api.ERRORS_RETURN)
    api.op_init(["OP_PART_SIZE=512", "OP_BLOCK_SIZE=512"], 0)
    old = api.set_strategy(api.STRATEGY_COLOURED)
    lib = api.lib()
    lib.op2b_set_tuning(b"coloured_fold", fold)
    try:
        n, rng = mesh.ncell, np.random.default_rng(4)
        qinf = np.asarray(apps.airfoil_consts(dt)["qinf"], dt)
        q = qinf * (1 + rng.uniform(-0.01, 0.01, (n, 4)))
        A = apps.Airfoil(mesh, dt, state=dict(q=q, qold=q, res=np.zeros((n, 4)), adt=np.ones(n)))
        for nm in ("adt_calc", "res_calc", "bres_calc", "save_soln", "res_calc", "update"):
            A.loop(nm)
        st = {k: v.copy() for k, v in A.fetch().items()}
        assert api.last_error() == "", api.last_error()
        counts = []
        for nm, inds in INDS.items():
            s, args = A.loops[nm]
            counts.append(api.op_plan_core(nm, s, 512, args, inds).contents.count)
        return st, counts
    finally:
        lib.op2b_set_tuning(b"coloured_fold", 1)
        api.set_strategy(old)
        api.op_exit()
        api.op_init(["OP_PART_SIZE=0", "OP_BLOCK_SIZE=512"], 0)
        api.op_exit()
        api.clear_error()


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("shared", [0, 6, 100, 33000])
def test_a_cell_on_many_edges(shared, dt):
    mesh = M.naca0012(110, 60)
    assert mesh.nedge > 33000
    mesh.ecell = mesh.ecell.copy()
    mesh.ecell[:shared, 0] = 5  # edges 0 ... shared - 1 all increment cell 5
    (a, ca), (b, cb) = solve(0, mesh, dt), solve(1, mesh, dt)
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k
    assert ca == cb
