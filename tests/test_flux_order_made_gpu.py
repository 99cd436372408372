"""That the flux pass's own order of the edges is made and taken where it
should be (op2b_flux_orders), and gives every field bit for bit as the loop's
order does: edge counts around multiples of the 1024 edges of a sampled chunk
and around the least for which an order is made, and node data that are no
coordinates, whose order the sample rejects."""
import copy
import ctypes as C

import numpy as np
import pytest

from oplus2_matlab_b200 import api, apps
from oplus2_matlab_b200 import mesh as M
from test_autotune_gpu import DEFAULTS

pytestmark = pytest.mark.gpu

LEAST = 16384


def orders():
    kept = C.c_int()
    return api.lib().op2b_flux_orders(C.byref(kept)), kept.value


def with_edges(n, scramble=True):
    m = copy.copy(M.naca0012(80, 60, scramble=scramble))
    assert m.nedge > n
    m.edge, m.ecell = np.ascontiguousarray(m.edge[:n]), np.ascontiguousarray(m.ecell[:n])
    m.nedge = n
    return m


def solve(mesh, dt, strategy, order, steps=3):
    """the fields after some iterations, and the orders made and kept"""
    api.set_error_mode(api.ERRORS_RETURN)
    api.op_init([], 0)
    old = api.set_strategy(strategy)
    api.lib().op2b_set_tuning(b"flux_order", order)
    try:
        A = apps.Airfoil(mesh, dt)
        for nm in ("adt_calc", "res_calc", "bres_calc"):
            A.loop(nm)
        rms = list(A.iterate(steps))
        made = orders()
        st = {k: v.copy() for k, v in A.fetch().items()}
        assert api.last_error() == ""
        return [v.tobytes() for v in st.values()] + rms, made
    finally:
        api.lib().op2b_set_tuning(b"flux_order", 1)
        api.set_strategy(old)
        api.op_exit()
        api.clear_error()


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", [LEAST - 1, LEAST, LEAST + 1, LEAST + 1023, LEAST + 1024, LEAST + 1025, 28500])
def test_made_and_kept(dt, n):
    mesh = with_edges(n)
    for strategy in (api.STRATEGY_GATHER, api.STRATEGY_COLOURED):
        a, made = solve(mesh, dt, strategy, 0)
        assert made == (0, 0)
        b, made = solve(mesh, dt, strategy, 2)
        assert made == ((1, 1) if n >= LEAST else (0, 0))
        assert a == b


def test_made_once_it_has_paid():
    """1.05M edges, knob 1: after 24 passes, two an iteration, whatever the
    size above or below a million edges."""
    mesh = M.naca0012(480, 366, scramble=True)
    assert mesh.nedge > 1 << 20
    a, _ = solve(mesh, np.float32, api.STRATEGY_GATHER, 0, 16)
    for steps, want in ((4, (0, 0)), (10, (0, 0)), (16, (1, 1))):
        b, made = solve(mesh, np.float32, api.STRATEGY_GATHER, 1, steps)
        assert made == want, steps
    assert a == b


def test_made_before_the_autotuner_times(op2):
    api.set_strategy(api.STRATEGY_GATHER)
    A = apps.Airfoil(with_edges(28500), np.float32)
    A.iterate(1)
    assert orders() == (0, 0)
    try:
        assert api.lib().op2b_autotune(None, 1, 0) == 0, api.last_error()
        assert orders() == (1, 1)
    finally:
        for k, v in DEFAULTS.items():
            api.lib().op2b_set_tuning(k.encode(), v)


def test_numbering_with_locality():
    assert solve(with_edges(LEAST, scramble=False), np.float32, api.STRATEGY_GATHER, 2)[1] == (0, 0)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("strategy", [api.STRATEGY_GATHER, api.STRATEGY_COLOURED])
def test_rejected(dt, strategy):
    mesh = with_edges(LEAST + 500)
    mesh.x32 = np.random.default_rng(1).uniform(-1, 1, mesh.x32.shape).astype(np.float32)
    mesh.x64 = mesh.x32.astype(np.float64)
    a, _ = solve(mesh, dt, strategy, 0)
    b, made = solve(mesh, dt, strategy, 2)
    assert made == (1, 0)
    assert a == b
