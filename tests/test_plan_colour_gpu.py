"""The block colouring from the blocks' conflicts against the oracle's
op_plan_core, where its parts meet their limits: rows narrower and wider than
the narrow greedy holds, more than 32 colours, targets of many blocks, one
block, two incremented datasets, more blocks than the conflicts are kept for."""
import numpy as np
import pytest

import oracle_lib as O
from oplus2_matlab_b200 import mesh as M

pytestmark = pytest.mark.gpu
R, INC = 0, 3


def check(op2, name, n, maps, part):
    """maps: (array [n, dim], target set size), every column an INC argument."""
    s = op2.op_decl_set(n, "elements")
    args, inds, spec = [], [], []
    for k, (m, size) in enumerate(maps):
        m = np.ascontiguousarray(m, np.int32)
        to = op2.op_decl_set(size, "targets%d" % k)
        mp = op2.op_decl_map(s, to, m.shape[1], m, "map%d" % k)
        d = op2.op_decl_dat(to, 1, "float", np.zeros((size, 1), np.float32), "d%d" % k)
        for c in range(m.shape[1]):
            args.append(op2.op_arg_dat(d, c, mp, 1, "float", op2.OP_INC))
            inds.append(k)
            spec.append((m, m.shape[1], c, size, 4, INC))
    p = op2.op_plan_core(name, s, part, args, inds)
    assert p, op2.last_error()
    got = op2.plan_arrays(p, args, inds)
    ref, checks, colours = O.plan_core(O.LoopSpec(n, spec, inds), part)
    try:
        assert checks == 0 and colours == 0
        assert (got["nblocks"], got["ncolors"]) == (ref["nblocks"], ref["ncolors"])
        for key in ("blkmap", "ncolblk", "thrcol", "nthrcol"):
            assert np.array_equal(got[key], ref[key]), key
    finally:
        O.plan_free(ref)
    return got


@pytest.mark.parametrize("scramble,part", [(False, 16), (True, 16), (False, 5000), (True, 64)])
def test_mesh_blocks(op2, scramble, part):
    m = M.naca0012(100, 150, scramble=scramble)
    check(op2, "mesh", m.nedge, [(m.ecell, m.ncell)], part)


@pytest.mark.parametrize("n,targets,part", [(70, 3, 1), (3000, 2, 1), (5000, 40, 8), (33000, 900, 2)])
def test_targets_of_many_blocks(op2, n, targets, part):
    rng = np.random.default_rng(n)
    got = check(op2, "many", n, [(rng.integers(0, targets, (n, 2)), targets)], part)
    assert got["ncolors"] > 32


def test_two_incremented_datasets_and_one_block(op2):
    rng = np.random.default_rng(1)
    n = 4000
    near = (np.arange(n)[:, None] + rng.integers(0, 5, (n, 2))) % n
    far = rng.integers(0, n, (n, 1))
    check(op2, "two", n, [(near, n), (far, n)], 16)
    check(op2, "one", 100, [(near[:100] % 100, 100)], 0)


def test_more_blocks_than_conflicts_are_kept_for(op2):
    n = 20000
    ring = (np.arange(n)[:, None] + np.array([[0, 1]])) % n
    check(op2, "ring", n, [(ring, n)], 1)
