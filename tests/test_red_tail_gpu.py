"""The rms an update leaves to the next kernel (knob red_tail), where the
number of block partials or the place of the fold could go wrong.  With the
knob at 0 each update folds its own partials in the same order, so every rms
must be equal bit for bit."""
import ctypes as C

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
    rt.cudaStreamSynchronize.argtypes = [P]
    return rt


RELAXED = 2  # cudaStreamCaptureModeRelaxed


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_a_callers_capture_records_no_fold_of_an_earlier_update(op2, dt):
    """A deferred update, then a stream capture of the caller's own (never
    launched) of loops whose flux pass could take the update's rms along:
    op2b_sync delivers the rms all the same."""
    mesh = M.naca0012(41, 61)
    rt = cudart()

    def run(tail, capture):
        A = start(mesh, dt, api.STRATEGY_GATHER, tail)
        A.iterate(2)
        for nm in ("adt_calc", "res_calc", "bres_calc", "adt_calc"):  # plans without update
            A.loop(nm)
        A.iterate(1)
        api.set_gbl_deferred(1)
        A.rms[0] = 0
        for nm in ("save_soln", "adt_calc") + STAGE + ("adt_calc",):
            A.loop(nm)  # the last call runs the held update
        if capture:
            s = C.c_void_p(api.get_stream())
            assert rt.cudaStreamBeginCapture(s, RELAXED) == 0
            for nm in ("res_calc", "bres_calc", "adt_calc"):
                A.loop(nm)
            g = C.c_void_p()
            assert rt.cudaStreamEndCapture(s, C.byref(g)) == 0
            assert rt.cudaGraphDestroy(g) == 0
        api.sync()
        assert api.last_error() == ""
        return float(A.rms[0])

    want = run(0, False)
    assert want > 0
    for tail, capture in ((1, False), (0, True), (1, True)):
        api.set_gbl_deferred(0)
        api.op_exit()
        api.op_init([], 0)
        assert run(tail, capture) == want, (tail, capture)


def test_a_jac_update_before_a_callers_capture(op2):
    """The same with jac1's sum and maximum and the res behind them."""
    rt = cudart()

    def run(tail, capture):
        api.set_strategy(api.STRATEGY_GATHER)
        api.lib().op2b_set_tuning(b"red_tail", tail)
        api.lib().op2b_set_tuning(b"jac_step", 0)
        J = apps.Jac(M.jac(40, 1), 1)
        J.iterate(2)
        api.set_gbl_deferred(1)
        api.op_par_loop("res", J.edges, *J.res_args)
        J.u_sum[0] = J.u_max[0] = 0
        api.op_par_loop("update", J.nodes, *J.upd_args)
        if capture:
            s = C.c_void_p(api.get_stream())
            assert rt.cudaStreamBeginCapture(s, RELAXED) == 0
            api.op_par_loop("res", J.edges, *J.res_args)
            g = C.c_void_p()
            assert rt.cudaStreamEndCapture(s, C.byref(g)) == 0
            assert rt.cudaGraphDestroy(g) == 0
        api.sync()
        assert api.last_error() == ""
        return float(J.u_sum[0]), float(J.u_max[0])

    try:
        want = run(0, False)
        assert want[0] > 0
        for tail, capture in ((1, False), (0, True), (1, True)):
            api.set_gbl_deferred(0)
            api.op_exit()
            api.op_init([], 0)
            assert run(tail, capture) == want, (tail, capture)
    finally:
        api.lib().op2b_set_tuning(b"jac_step", 1)


def test_a_capture_after_one_that_failed(op2):
    """jac1's update twice in a capture: the second has the first fold its own
    partials, which is put into the graph at the capture's end.  A
    synchronisation breaks the capture before that; the next capture holds
    nothing of it and its sums are those of the loops."""
    rt, lib = cudart(), api.lib()

    def run(failed, tail):
        lib.op2b_set_tuning(b"red_tail", tail)
        lib.op2b_set_tuning(b"jac_step", 0)
        J = apps.Jac(M.jac(40, 1), 1)
        J.iterate(2)

        def update():
            api.op_par_loop("update", J.nodes, *J.upd_args)

        if failed:
            assert lib.op2b_capture_begin(0) == 1
            update()
            update()
            assert rt.cudaStreamSynchronize(C.c_void_p(api.get_stream())) != 0
            assert not lib.op2b_capture_end()
            assert "capture failed" in api.last_error()
            api.clear_error()
        assert lib.op2b_capture_begin(0) == 1
        api.op_par_loop("res", J.edges, *J.res_args)
        update()
        api.op_par_loop("res", J.edges, *J.res_args)
        update()
        h = lib.op2b_capture_end()
        assert h, api.last_error()
        out = []
        for _ in range(3):
            J.u_sum[0] = J.u_max[0] = 0
            assert lib.op2b_graph_launch(h) == 0
            api.sync()
            out.append((float(J.u_sum[0]), float(J.u_max[0])))
        lib.op2b_graph_destroy(h)
        assert api.last_error() == ""
        return out

    try:
        want = run(False, 0)
        for failed, tail in ((True, 1), (False, 1)):
            api.op_exit()
            api.op_init([], 0)
            assert run(failed, tail) == want
    finally:
        lib.op2b_set_tuning(b"jac_step", 1)
