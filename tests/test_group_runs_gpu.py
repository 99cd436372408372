"""The group's cell pass over runs of 256 to 1024 cells per CTA and its
iterations issued one by one, singly or eight to a graph.

A solve's fields equal the plain solve's bit for bit whatever its lists' width,
and its rms history does not depend on the run its cells fall into (a solve
alone has short runs, the same one beside a large one long ones) nor on how the
iterations were issued.
"""
import copy

import numpy as np
import pytest

from oplus2_matlab_b200 import group as G
from oplus2_matlab_b200 import mesh as M

pytestmark = pytest.mark.gpu


def with_width(width):
    """A small mesh whose longest list has `width` entries: edges left out of
    (below 4) or listed again at (above 4) some cells."""
    m = copy.copy(M.naca0012(6, 9))
    if width < 4:
        count = np.zeros(m.ncell, int)
        np.add.at(count, m.becell, 1)
        keep = []
        for e, (a, b) in enumerate(m.ecell):
            if count[a] < width and count[b] < width:
                count[a] += 1
                count[b] += 1
                keep.append(e)
    else:
        keep = list(range(m.nedge)) + [0] * (width - 4)
        count = np.zeros(m.ncell, int)
        np.add.at(count, m.becell, 1)
        np.add.at(count, m.ecell[keep].ravel(), 1)
    m.edge = np.ascontiguousarray(m.edge[keep])
    m.ecell = np.ascontiguousarray(m.ecell[keep])
    m.nedge = len(keep)
    assert count.max() == width
    return m


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("width", [2, 3, 4, 5, 7])
def test_lists_of_any_width(op2, width, dtype):
    m = with_width(width)
    g = G.Group(dtype)
    i = g.add(m, 0.4, 1.0, 3)
    g.run(3)
    want = G.plain_solve(m, 0.4, 1.0, 3, dtype)[0]
    assert np.isfinite(want).all()
    assert g.fetch_q(i).tobytes() == want.astype(dtype).tobytes()
    g.close()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
# cells: below, at and above one partial; a ragged number of them
@pytest.mark.parametrize("ij", [(3, 5), (8, 32), (16, 16), (1 + 16, 16), (40, 61)])
def test_rms_does_not_depend_on_the_run(op2, ij, dtype):
    m, n = M.naca0012(*ij), 5
    alone = G.Group(dtype)
    a = alone.add(m, 0.5, 2.0, n)
    alone.run(n)
    want = alone.fetch_q(a).tobytes(), alone.history(a).tobytes()
    alone.close()
    mix = G.Group(dtype)
    mix.add(M.naca0012(300, 450), 0.4, 0.0, n)  # long runs for every solve
    b = mix.add(m, 0.5, 2.0, n)
    mix.run(n)
    assert (mix.fetch_q(b).tobytes(), mix.history(b).tobytes()) == want
    mix.close()


@pytest.mark.parametrize("parts", [[19], [1] * 19, [8, 11], [2, 16, 1], [11, 8]])
def test_iterations_however_issued(op2, parts):
    ms, n = [M.naca0012(20, 30), M.naca0012(12, 17)], 19
    ref = G.Group()
    ids = [ref.add(x, 0.4 + 0.1 * k, 1.0, n) for k, x in enumerate(ms)]
    ref.run(n + 64)  # graphs of eight; every solve stops at n
    want = [(ref.fetch_q(i).tobytes(), ref.history(i).tobytes()) for i in ids]
    ref.close()
    g = G.Group()
    ids = [g.add(x, 0.4 + 0.1 * k, 1.0, n) for k, x in enumerate(ms)]
    for p in parts:
        g.run(p)
    g.sync()
    assert [g.iterations(i) for i in ids] == [n, n]
    assert [(g.fetch_q(i).tobytes(), g.history(i).tobytes()) for i in ids] == want
    g.close()
