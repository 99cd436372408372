"""COLOURED res_calc as a flux pass and a per-cell fold in the plan's order
(knob coloured_fold, the default) against one launch per block colour: every
field bit for bit, and with SEQ reductions every rms, over both precisions,
numberings, part and block sizes (strips of OP_BLOCK_SIZE edges inside a
block), loops fused or not, run ahead, deferred and captured."""
import numpy as np
import pytest

from oplus2_matlab_b200 import api, apps
from oplus2_matlab_b200 import mesh as M

pytestmark = pytest.mark.gpu


def solve(fold, mesh, dt, mode, part=0, block=512):
    api.set_error_mode(api.ERRORS_RETURN)
    api.op_init(["OP_PART_SIZE=%d" % part, "OP_BLOCK_SIZE=%d" % block], 0)
    lib = api.lib()
    old = api.set_strategy(api.STRATEGY_COLOURED)
    lib.op2b_set_tuning(b"coloured_fold", fold)
    api.set_reduction(api.REDUCE_TREE if mode == "graph" else api.REDUCE_SEQ)
    try:
        rng = np.random.default_rng(3)
        qinf = np.asarray(apps.airfoil_consts(dt)["qinf"], dt)
        q = (qinf * (1 + rng.uniform(-0.01, 0.01, (mesh.ncell, 4)))).astype(dt)
        res = rng.uniform(-1e-3, 1e-3, (mesh.ncell, 4)).astype(dt)  # not zero at first
        A = apps.Airfoil(mesh, dt, state=dict(q=q, qold=q, res=res, adt=np.ones((mesh.ncell, 1))))
        rms = []
        if mode == "loops":  # a residual, then loops in an order that does not fuse
            for nm in ("adt_calc", "res_calc", "bres_calc", "adt_calc", "res_calc", "adt_calc",
                       "bres_calc", "save_soln", "res_calc", "update"):
                A.loop(nm)
        elif mode == "eager":
            rms = list(A.iterate(4))
        else:
            A.iterate(1)
            assert lib.op2b_capture_begin(0) == 1
            for nm in ("save_soln",) + 2 * ("adt_calc", "res_calc", "bres_calc", "update"):
                A.loop(nm)
            g = lib.op2b_capture_end()
            assert g, api.last_error()
            for _ in range(3):
                assert lib.op2b_graph_launch(g) == 0
            api.sync()
            lib.op2b_graph_destroy(g)
        st = {k: v.copy() for k, v in A.fetch().items()}
        assert api.last_error() == ""
        return st, rms
    finally:
        lib.op2b_set_tuning(b"coloured_fold", 1)
        api.set_strategy(old)
        api.set_reduction(api.REDUCE_TREE)
        api.op_exit()
        # op_init keeps the sizes it is not given
        api.op_init(["OP_PART_SIZE=0", "OP_BLOCK_SIZE=512"], 0)
        api.op_exit()
        api.clear_error()


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("mode", ["eager", "loops", "graph"])
@pytest.mark.parametrize("I,J,scramble,part,block", [
    (3, 5, False, 0, 512), (17, 31, False, 64, 64), (21, 40, True, 128, 512),
    (40, 60, False, 512, 128), (40, 60, True, 256, 96)])
def test_fold_equals_block_colours(dt, mode, I, J, scramble, part, block):
    mesh = M.naca0012(I, J, scramble=scramble)
    a, ra = solve(0, mesh, dt, mode, part, block)
    b, rb = solve(1, mesh, dt, mode, part, block)
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k
    assert ra == rb
