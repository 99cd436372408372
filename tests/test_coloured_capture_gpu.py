"""COLOURED loops captured before the lists of their two passes are there: a
capture cannot make them, so the loops run by block colours in it, and what a
call outside the capture uses is made outside.  Every field bit for bit as with
the block colours alone (knob coloured_fold 0)."""
import ctypes as C

import numpy as np
import pytest

from oplus2_matlab_b200 import _lib, api, apps
from oplus2_matlab_b200 import mesh as M

pytestmark = pytest.mark.gpu

ITERATION = ("save_soln",) + 2 * ("adt_calc", "res_calc", "bres_calc", "update")


def cudart():
    for name in ("libcudart.so.12", "libcudart.so"):
        try:
            rt = C.CDLL(name)
            break
        except OSError:
            continue
    P = C.c_void_p
    rt.cudaStreamBeginCapture.argtypes = [P, C.c_int]
    rt.cudaStreamEndCapture.argtypes = [P, C.POINTER(P)]
    rt.cudaGraphDestroy.argtypes = [P]
    return rt


def solve(case, fold, dt, scramble):
    mesh = M.naca0012(24, 40, scramble=scramble)
    lib = api.lib()
    api.set_error_mode(api.ERRORS_RETURN)
    api.op_init(["OP_PART_SIZE=128", "OP_BLOCK_SIZE=512"], 0)
    old = api.set_strategy(api.STRATEGY_COLOURED)
    block = _lib.global_int("OP_block_size")
    try:
        # lists that are not there yet: none at all, or none for this block size
        lib.op2b_set_tuning(b"coloured_fold", 0 if case == "first" else fold)
        A = apps.Airfoil(mesh, dt)
        A.iterate(2)
        api.sync()
        lib.op2b_set_tuning(b"coloured_fold", fold)
        if case != "first":
            block.value = 64
        if case == "callers":  # recorded and thrown away
            rt, s, g = cudart(), C.c_void_p(api.get_stream()), C.c_void_p()
            api.set_gbl_deferred(1)
            assert rt.cudaStreamBeginCapture(s, 2) == 0
            for nm in ("adt_calc", "res_calc", "bres_calc", "adt_calc"):
                A.loop(nm)
            assert rt.cudaStreamEndCapture(s, C.byref(g)) == 0
            assert rt.cudaGraphDestroy(g) == 0
            api.set_gbl_deferred(0)
        else:
            assert lib.op2b_capture_begin(0) == 1, api.last_error()
            for nm in ITERATION:
                A.loop(nm)
            g = lib.op2b_capture_end()
            assert g, api.last_error()
        A.iterate(1)  # before the first launch
        if case != "callers":
            for _ in range(2):
                assert lib.op2b_graph_launch(g) == 0, api.last_error()
            api.sync()
            lib.op2b_graph_destroy(g)
        A.iterate(1)
        st = {k: v.copy() for k, v in A.fetch().items()}
        assert api.last_error() == ""
        return st
    finally:
        block.value = 512
        api.set_gbl_deferred(0)
        lib.op2b_set_tuning(b"coloured_fold", 1)
        api.set_strategy(old)
        api.op_exit()
        api.op_init(["OP_PART_SIZE=0", "OP_BLOCK_SIZE=512"], 0)
        api.op_exit()
        api.clear_error()


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("scramble", [False, True])
@pytest.mark.parametrize("case", ["first", "block size", "callers"])
def test_capture_before_the_lists(case, scramble, dt):
    a = solve(case, 0, dt, scramble)
    b = solve(case, 1, dt, scramble)
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k
