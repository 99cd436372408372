"""op2b_group_autotune a few iterations before solves stop: its trials run
whole graphs of eight or single iterations and put everything back, so the
solves go on as if it had not run."""
import numpy as np
import pytest

from oplus2_matlab_b200 import group as G
from oplus2_matlab_b200 import mesh as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("left", [1, 7, 8, 9, 21])
def test_autotune_before_the_end(op2, dtype, left):
    ms, before = [M.naca0012(20, 30), M.naca0012(12, 17)], 3
    out = []
    for iters in (0, 1, 7, 8, 17):
        g = G.Group(dtype)
        ids = [g.add(m, 0.4 + 0.1 * k, 1.0, before + left + 30 * k) for k, m in enumerate(ms)]
        g.run(before)
        if iters:
            assert g.autotune(iters) == g.edge_tile
            assert [g.iterations(i) for i in ids] == [before, before]
        g.run(before + left + 30)
        g.sync()
        out.append([(g.fetch_q(i).tobytes(), g.history(i).tobytes()) for i in ids])
        g.close()
    assert all(o == out[0] for o in out)
