"""op2b_autotune on a mesh with a cell on more edges than a contribution list
holds: the two passes of the chain do not apply, COLOURED by block colours
does, and is what the tuner finds when sums may be reordered."""
import numpy as np
import pytest

from oplus2_matlab_b200 import api, apps
from oplus2_matlab_b200 import mesh as M
from test_autotune_gpu import DEFAULTS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_block_colours_are_a_candidate(op2, dt):
    mesh = M.naca0012(20, 30)
    mesh.ecell = mesh.ecell.copy()
    mesh.ecell[:12, 0] = 5
    lib = api.lib()
    part, block = api.global_int("OP_part_size"), api.global_int("OP_block_size")
    A = apps.Airfoil(mesh, dt)
    try:
        A.iterate(1)
        api.sync()
        before = {k: v.copy() for k, v in A.fetch().items()}
        assert lib.op2b_autotune(None, 2, 1) == 0, api.last_error()
        assert api.set_strategy(api.STRATEGY_COLOURED) == api.STRATEGY_COLOURED
        after = A.fetch()
        for k in before:
            assert after[k].tobytes() == before[k].tobytes(), k
        A.iterate(2)  # runs (its fields mean nothing on such a mesh)
        api.sync()
        assert api.last_error() == ""
    finally:
        for k, v in DEFAULTS.items():
            lib.op2b_set_tuning(k.encode(), v)
        api._lib.global_int("OP_part_size").value = part
        api._lib.global_int("OP_block_size").value = block
