"""The flux pass's own order of the edges (knob flux_order) against the loop's:
every field bit for bit, over sizes around a chunk of 1024 edges, numberings
with and without locality, both precisions, GATHER and COLOURED, the residual
alone and the fused chain; node datasets that are no coordinates; and the knob
changed between two loops whose flux pass has run ahead."""
import numpy as np
import pytest

from oplus2_matlab_b200 import api, apps
from oplus2_matlab_b200 import mesh as M

pytestmark = pytest.mark.gpu


def solve(mesh, dt, strategy, order, flip=False):
    api.set_error_mode(api.ERRORS_RETURN)
    api.op_init([], 0)
    lib = api.lib()
    old = api.set_strategy(strategy)
    api.set_reduction(api.REDUCE_TREE)
    lib.op2b_set_tuning(b"flux_order", order)
    try:
        A = apps.Airfoil(mesh, dt)
        for nm in ("adt_calc", "res_calc", "bres_calc"):
            A.loop(nm)
        api.sync()
        rms = list(A.iterate(3))
        if flip:
            lib.op2b_set_tuning(b"flux_order", 2 - order if order else 1)
        rms += list(A.iterate(2))
        st = {k: v.copy() for k, v in A.fetch().items()}
        assert api.last_error() == ""
        return st, rms
    finally:
        lib.op2b_set_tuning(b"flux_order", 1)
        api.set_strategy(old)
        api.op_exit()
        api.clear_error()


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("I,J,scramble", [(2, 4, False), (17, 10, False), (19, 9, False), (40, 60, False),
                                          (17, 10, True), (60, 90, True), (131, 77, True)])
def test_same_fields(dt, I, J, scramble):
    mesh = M.naca0012(I, J, scramble=scramble)
    for strategy in (api.STRATEGY_GATHER, api.STRATEGY_COLOURED):
        a, ra = solve(mesh, dt, strategy, 0)
        b, rb = solve(mesh, dt, strategy, 1)
        c, rc = solve(mesh, dt, strategy, 2, flip=True)
        d, rd = solve(mesh, dt, strategy, 2)
        for k in a:
            assert a[k].tobytes() == b[k].tobytes() == c[k].tobytes() == d[k].tobytes(), (strategy, k)
        assert ra == rb == rc == rd


@pytest.mark.parametrize("what", ["nan", "inf", "same", "noise"])
def test_node_data_that_are_no_coordinates(what):
    mesh = M.naca0012(50, 70, scramble=True)
    x = mesh.x32.copy()
    if what == "nan":
        x[::3] = np.nan
    elif what == "inf":
        x[::5, 0], x[::7, 1] = np.inf, -np.inf
    elif what == "same":
        x[:] = 1.5
    else:
        x[:] = np.random.default_rng(1).uniform(-1, 1, x.shape)
    mesh.x32 = x
    a, _ = solve(mesh, np.float32, api.STRATEGY_GATHER, 0)
    b, _ = solve(mesh, np.float32, api.STRATEGY_GATHER, 2)
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k


@pytest.mark.parametrize("strategy", [api.STRATEGY_GATHER, api.STRATEGY_COLOURED])
@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_made_during_the_run_or_by_a_capture(dt, strategy):
    """60k edges: made by the 105th pass (between an update and the chain whose
    flux pass it ran ahead), or by the capture of an iteration before that."""
    mesh = M.naca0012(131, 77, scramble=True)
    rot = ("res_calc", "bres_calc", "update", "adt_calc", "res_calc", "bres_calc", "update", "save_soln", "adt_calc")

    def run(order, capture):
        api.set_error_mode(api.ERRORS_RETURN)
        api.op_init([], 0)
        lib = api.lib()
        old = api.set_strategy(strategy)
        lib.op2b_set_tuning(b"flux_order", order)
        try:
            A = apps.Airfoil(mesh, dt)
            rms = list(A.iterate(2 if capture else 60))
            if capture:
                A.loop("save_soln")
                A.loop("adt_calc")
                api.sync()
                assert lib.op2b_capture_begin(0) == 1
                for nm in rot:
                    A.loop(nm)
                g = lib.op2b_capture_end()
                assert g, api.last_error()
                for _ in range(3):
                    lib.op2b_graph_launch(g)
                api.sync()
                lib.op2b_graph_destroy(g)
            st = {k: v.copy() for k, v in A.fetch().items()}
            assert api.last_error() == ""
            return st, rms
        finally:
            lib.op2b_set_tuning(b"flux_order", 1)
            api.set_strategy(old)
            api.op_exit()
            api.clear_error()

    for capture in (False, True):
        a, ra = run(0, capture)
        b, rb = run(1, capture)
        for k in a:
            assert a[k].tobytes() == b[k].tobytes(), (capture, k)
        assert ra == rb
