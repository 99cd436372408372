"""The airfoil-shaped per-cell pass (knob fold_cells) against the general one,
and the rms left to the next flux pass (knob red_tail) against the one the
pass folds itself: every field bit for bit, every rms too where only red_tail
differs.  Sizes below a CTA, around one and over a whole wave; eager (the rms
waited for on its flag), deferred and captured; two solves taking turns."""
import numpy as np
import pytest

from oplus2_matlab_b200 import api, apps
from oplus2_matlab_b200 import mesh as M

pytestmark = pytest.mark.gpu
LOOPS = ("save_soln",) + 2 * ("adt_calc", "res_calc", "bres_calc", "update")


def solve(mesh, dt, mode, cells, tail):
    api.set_error_mode(api.ERRORS_RETURN)
    api.op_init([], 0)
    lib = api.lib()
    old = api.set_strategy(api.STRATEGY_GATHER)
    api.set_reduction(api.REDUCE_TREE)
    lib.op2b_set_tuning(b"fold_cells", cells)
    lib.op2b_set_tuning(b"red_tail", tail)
    try:
        A = apps.Airfoil(mesh, dt)
        rms = []
        if mode == "eager":
            rms = list(A.iterate(5))
        elif mode == "two":  # another solve between the iterations
            B = apps.Airfoil(mesh, dt)
            for _ in range(4):
                rms += [A.iteration(), B.iteration(), B.iteration()]
        elif mode == "deferred":
            A.iteration()
            api.set_gbl_deferred(1)
            A.rms[0] = 0
            for _ in range(3):
                for nm in LOOPS:
                    A.loop(nm)
            api.sync()
            rms = [A.rms[0]]
            A.loop("save_soln")  # not the loop the held update expects next
            A.loop("update")
            api.sync()
            rms.append(A.rms[0])
        else:
            A.iteration()
            assert lib.op2b_capture_begin(0) == 1
            for nm in LOOPS:
                A.loop(nm)
            g = lib.op2b_capture_end()
            assert g, api.last_error()
            for _ in range(3):
                A.rms[0] = 0
                assert lib.op2b_graph_launch(g) == 0
                api.sync()
                rms.append(A.rms[0])
            n = lib.op2b_graph_nkernels(g)
            lib.op2b_graph_destroy(g)
            rms.append(n)
        st = {k: v.copy() for k, v in A.fetch().items()}
        assert api.last_error() == ""
        return st, rms
    finally:
        lib.op2b_set_tuning(b"fold_cells", 1)
        lib.op2b_set_tuning(b"red_tail", 1)
        api.set_gbl_deferred(0)
        api.set_strategy(old)
        api.op_exit()
        api.clear_error()


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("mode", ["eager", "two", "deferred", "graph"])
@pytest.mark.parametrize("I,J,scramble", [(2, 4, False), (17, 5, False), (4, 21, True), (64, 4, False),
                                          (120, 250, True)])
def test_same_fields_and_rms(dt, mode, I, J, scramble):
    mesh = M.naca0012(I, J, scramble=scramble)
    a, ra = solve(mesh, dt, mode, 0, 0)
    b, rb = solve(mesh, dt, mode, 1, 0)
    c, rc = solve(mesh, dt, mode, 1, 1)
    for k in a:
        assert a[k].tobytes() == b[k].tobytes() == c[k].tobytes(), k
    assert rb == rc  # the same partials in the same order, and as many kernels
    # another grid's partials: a tree sum of 4 n terms, n * eps at the worst
    n = mesh.ncell
    assert np.allclose(np.array(ra, np.float64), np.array(rc, np.float64), rtol=4 * n * np.finfo(dt).eps, atol=0)
