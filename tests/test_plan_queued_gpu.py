"""Kernels that read plan arrays before they wait for the kernel in front of
them (programmatic dependent launch), where that kernel is the one that has
just filled the arrays: the fold behind coloured lists made for a new block
size after its flux pass has run ahead, the flux pass behind an order that is
rejected, and jac's first res behind its pairs.  Against the same calls with
programmatic launches off (knob pdl), bit for bit."""
import numpy as np
import pytest

from oplus2_matlab_b200 import _lib, api, apps
from oplus2_matlab_b200 import mesh as M

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def knobs(op2):
    api.op_exit()
    api.op_init(["OP_PART_SIZE=128", "OP_BLOCK_SIZE=512"], 0)
    yield
    api.lib().op2b_set_tuning(b"pdl", 1)
    api.lib().op2b_set_tuning(b"flux_order", 1)
    _lib.global_int("OP_block_size").value = 512
    _lib.global_int("OP_part_size").value = 0


def both(run):
    out = []
    for pdl in (0, 1):
        api.lib().op2b_set_tuning(b"pdl", pdl)
        out.append(run())
        assert api.last_error() == ""
        api.op_exit()
        api.op_init(["OP_PART_SIZE=128", "OP_BLOCK_SIZE=512"], 0)
    a, b = out
    for k in a:
        assert a[k].tobytes() == b[k].tobytes(), k


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("scramble", [False, True])
def test_lists_for_a_new_block_size_after_the_flux_pass(dt, scramble):
    mesh = M.naca0012(60, 90, scramble=scramble)

    def run():
        api.set_strategy(api.STRATEGY_COLOURED)
        A = apps.Airfoil(mesh, dt)
        A.iterate(3)
        for block in (64, 32, 96):
            A.loop("save_soln")
            A.loop("adt_calc")
            _lib.global_int("OP_block_size").value = block  # its flux pass has run ahead
            for nm in ("res_calc", "bres_calc", "update"):
                A.loop(nm)
            A.iterate(1)
        _lib.global_int("OP_block_size").value = 512
        return {k: v.copy() for k, v in A.fetch().items()}

    both(run)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_first_pass_of_a_rejected_order(dt):
    mesh = M.naca0012(131, 77, scramble=True)
    mesh.x32 = np.random.default_rng(1).uniform(-1, 1, mesh.x32.shape).astype(np.float32)
    mesh.x64 = mesh.x32.astype(np.float64)

    def run():
        api.set_strategy(api.STRATEGY_GATHER)
        api.lib().op2b_set_tuning(b"flux_order", 2)
        A = apps.Airfoil(mesh, dt)
        for nm in ("adt_calc", "res_calc", "bres_calc"):
            A.loop(nm)
        return {k: v.copy() for k, v in A.fetch().items()}

    both(run)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("noise", [False, True])
def test_order_made_by_a_capture_that_is_not_launched(dt, noise):
    """The loops recorded behind the making of the order run no kernel; the
    next flux pass is an eager one (noise: its rows are the rejected order's)."""
    mesh = M.naca0012(131, 77, scramble=True)
    if noise:
        mesh.x32 = np.random.default_rng(1).uniform(-1, 1, mesh.x32.shape).astype(np.float32)
        mesh.x64 = mesh.x32.astype(np.float64)

    def run():
        lib = api.lib()
        api.set_strategy(api.STRATEGY_GATHER)
        A = apps.Airfoil(mesh, dt)
        for nm in ("adt_calc", "res_calc", "bres_calc"):
            A.loop(nm)
        api.sync()
        assert lib.op2b_flux_orders(None) == 0
        assert lib.op2b_capture_begin(0) == 1, api.last_error()
        for nm in ("adt_calc", "res_calc", "bres_calc"):
            A.loop(nm)
        h = lib.op2b_capture_end()
        assert h, api.last_error()
        for nm in ("res_calc", "bres_calc"):
            A.loop(nm)
        out = {k: v.copy() for k, v in A.fetch().items()}
        assert lib.op2b_flux_orders(None) == 1
        lib.op2b_graph_destroy(h)
        return out

    both(run)


@pytest.mark.parametrize("variant", [1, 2])
def test_pairs_are_not_made_in_a_capture(variant):
    """A capture's first res through another column of the map, then the same
    loop outside before the graph is launched; against the loop alone."""
    mesh = M.jac(100, variant)

    def run(capture):
        lib = api.lib()
        api.set_strategy(api.STRATEGY_GATHER)
        J = apps.Jac(mesh, variant)
        J.iterate(2)
        args = list(J.res_args)
        args[1] = api.op_arg_dat(J.p_u, 0, J.ppedge, J.u.shape[1], "float", api.OP_READ)
        if capture:
            assert lib.op2b_capture_begin(0) == 1, api.last_error()
            api.op_par_loop("res", J.edges, *args)
            h = lib.op2b_capture_end()
            assert h, api.last_error()
        api.op_par_loop("res", J.edges, *args)
        if capture:
            assert lib.op2b_graph_launch(h) == 0
            api.sync()
            lib.op2b_graph_destroy(h)
        else:
            api.op_par_loop("res", J.edges, *args)
        api.op_fetch_data(J.p_du)
        assert api.last_error() == ""
        return J.du.copy()

    want = run(False)
    api.op_exit()
    api.op_init([], 0)
    assert np.any(want != 0)
    assert run(True).tobytes() == want.tobytes()


@pytest.mark.parametrize("variant", [1, 2])
def test_first_res_of_jac(variant):
    mesh = M.jac(200, variant)

    def run():
        api.set_strategy(api.STRATEGY_GATHER)
        J = apps.Jac(mesh, variant)
        J.u[...] = np.random.default_rng(2).uniform(-1, 1, J.u.shape)
        J.p_u = api.op_decl_dat(J.nodes, J.u.shape[1], "float", J.u, "p_u2")
        J.res_args[1] = api.op_arg_dat(J.p_u, 1, J.ppedge, J.u.shape[1], "float", api.OP_READ)
        api.op_par_loop("res", J.edges, *J.res_args)
        api.op_fetch_data(J.p_du)
        assert np.any(J.du != 0)
        return {"du": J.du.copy()}

    both(run)
