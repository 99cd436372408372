"""SEQ reductions: the rms of airfoil's update, added in element order, must
equal numpy's one-at-a-time sum bit for bit (np.add.accumulate adds in order
with one rounding per addition), whatever the values do to the running sum:
ties, subnormals, jumps over many binades, infinities, NaN, a negative start."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CELLS = [1, 511, 512, 513, 1023, 1024, 1025, 4097, 70001]  # 2048 / 4096 values: the head / a tile


def values(kind, n, t, rng):
    """res values whose squares (adt = 1) are the addends; the start value."""
    u = rng.random(n)
    if kind == "uniform":
        return u, 0.0
    if kind == "ties":  # multiples of 1/8 onto a sum of 2^20 or more
        return np.sqrt(rng.integers(0, 9, n) / 8.0), 2.0 ** (21 if t == np.float32 else 50) + 1.0
    if kind == "wide":
        return np.exp(20 * (u - 0.5)), 0.0
    if kind == "powers":
        return 2.0 ** -rng.integers(0, 20, n).astype(np.float64), 3.0
    if kind == "subnormal":
        return np.sqrt(np.finfo(t).smallest_subnormal.astype(np.float64) if t == np.float32 else 1e-160) * (1 + 9 * u), 0.0
    if kind == "stuck":  # addends below half an ulp of the sum
        return 1e-3 * u, 1e12 if t == np.float32 else 1e30
    if kind == "jumps":
        return np.where(u < 0.001, 1e9, u), 0.0
    if kind == "overflow":
        return u * np.sqrt(np.finfo(t).max / 50), 0.0
    if kind == "nan":
        v = u.copy()
        v[n // 2] = np.nan
        return v, 0.0
    if kind == "inf":
        v = u.copy()
        v[n // 3] = np.inf
        return v, 0.0
    return u, -0.4 * n / 3  # negative: the sum starts below zero


@pytest.mark.parametrize("t", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["uniform", "ties", "wide", "powers", "subnormal", "stuck", "jumps",
                                  "overflow", "nan", "inf", "negative"])
def test_update_rms_is_the_serial_sum(op2, t, kind):
    op2.set_reduction(op2.REDUCE_SEQ)
    tn = "float" if t == np.float32 else "double"
    keep = []
    for k, n in enumerate(CELLS):
        rng = np.random.default_rng(100 * k + len(kind))
        v, init = values(kind, 4 * n, t, rng)
        cells = op2.op_decl_set(n, "cells")
        res = np.ascontiguousarray(v.reshape(n, 4), dtype=t)
        qold, q, adt = np.zeros((n, 4), t), np.zeros((n, 4), t), np.ones((n, 1), t)
        rms = np.array([init], t)
        with np.errstate(all="ignore"):
            want = np.add.accumulate(np.concatenate([rms, (res * res).ravel()]), dtype=t)[-1]
        d = [op2.op_decl_dat(cells, a.shape[1], tn, a, nm)
             for a, nm in ((qold, "qold"), (q, "q"), (res, "res"), (adt, "adt"))]
        keep += [res, qold, q, adt, rms]
        op2.op_par_loop("update", cells,
                        op2.op_arg_dat(d[0], -1, None, 4, tn, op2.OP_READ),
                        op2.op_arg_dat(d[1], -1, None, 4, tn, op2.OP_WRITE),
                        op2.op_arg_dat(d[2], -1, None, 4, tn, op2.OP_RW),
                        op2.op_arg_dat(d[3], -1, None, 1, tn, op2.OP_READ),
                        op2.op_arg_gbl(rms, 1, tn, op2.OP_INC))
        op2.sync()
        assert rms[0] == want or (np.isnan(want) and np.isnan(rms[0])), (n, rms[0], want)
