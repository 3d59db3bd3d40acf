"""complex128 product over rows (qr_apply_rows.cu): edges of its splits.

Rows per thread and group slices follow from the number of rows (states
times 2^n), descriptors come in chunks of 32 groups, and factors that are
real or imaginary throughout take half the multiply-adds unless an amplitude
is infinite or NaN.  Tolerance: a row sums at most ~300 products of FP64
rounding 2^-53 each, so 1e-12 of the result's norm leaves two digits.
"""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _run(cuda, op, psi, **kw):
    import torch
    y = op.apply(torch.from_numpy(psi).to(cuda), **kw)
    op.sync_check()
    return y.cpu().numpy()


def _want(oracle, t, c, psi):
    cp = oracle.make_params(t.phase, c)
    return np.stack([oracle.apply(t.n, t.x, t.z, cp, p) for p in psi])


# every rows-per-thread / slices choice (2^12 ... 2^21 rows) and its edges,
# states smaller than a warp's rows, one to several states
@pytest.mark.parametrize("n,states", [(1, 1), (4, 3), (5, 1), (6, 300), (11, 1), (12, 1), (12, 3),
                                      (13, 1), (13, 3), (14, 3), (15, 3), (16, 1), (8, 9000),
                                      (19, 5)])
@pytest.mark.parametrize("scale", [1.0, 0.6 - 0.8j])
def test_row_splits(cuda, oracle, n, states, scale):
    rng = np.random.default_rng(100 * n + states)
    t = W.random_letters_op(rng, n, 45)
    c = t.coeff * scale
    psi = W.random_state(rng, 1 << n, nstates=max(2, states))[:states]
    op = PauliOperator(n, t.x, t.z, t.phase, c)
    got = _run(cuda, op, psi)
    pick = sorted(rng.choice(states, min(states, 3), replace=False))
    want = _want(oracle, t, c, psi[pick])
    assert np.linalg.norm(got[pick] - want) <= TOL * np.linalg.norm(want)


@pytest.mark.parametrize("groups", [1, 31, 32, 33, 64, 65, 97])
@pytest.mark.parametrize("n", [9, 14])
def test_descriptor_chunks(cuda, oracle, n, groups):
    rng = np.random.default_rng(groups)
    x = rng.choice(1 << n, groups, replace=False).astype(np.uint64)
    # two terms per group, z masks differing: some factors vary within a warp's rows
    t = W.Terms(n, np.concatenate([x, x]), rng.integers(0, 1 << n, 2 * groups).astype(np.uint64),
                rng.integers(0, 4, 2 * groups).astype(np.uint8), rng.standard_normal(2 * groups))
    psi = W.random_state(rng, 1 << n, nstates=2)
    got = _run(cuda, PauliOperator(n, t.x, t.z, t.phase, t.coeff), psi)
    want = _want(oracle, t, t.coeff, psi)
    assert np.linalg.norm(got - want) <= TOL * np.linalg.norm(want)


def test_infinite_and_nan_amplitudes(cuda):
    """Every product D psi keeps its 0 * inf and 0 * nan parts."""
    n = 10
    rng = np.random.default_rng(7)
    t = W.random_letters_op(rng, n, 30)
    psi = W.random_state(rng, 1 << n)
    psi[17] = complex(np.inf, 1.0)
    psi[300] = complex(2.0, -np.inf)
    psi[901] = complex(np.nan, 0.0)
    got = _run(cuda, PauliOperator(n, t.x, t.z, t.phase, t.coeff), psi)
    rows = np.arange(1 << n, dtype=np.uint64)
    re, im = np.zeros(1 << n), np.zeros(1 << n)
    unit = np.array([1, -1j, -1, 1j])[t.phase]
    with np.errstate(invalid="ignore"):
        for x in np.unique(t.x):
            d = np.zeros(1 << n, dtype=np.complex128)
            for k in np.flatnonzero(t.x == x):
                sign = 1.0 - 2.0 * (np.bitwise_count(rows & t.z[k]) & 1)
                d += sign * (unit[k].real * t.coeff[k].real + 1j * unit[k].imag * t.coeff[k].real)
            p = psi[(rows ^ x).astype(np.int64)]
            re += d.real * p.real - d.imag * p.imag
            im += d.real * p.imag + d.imag * p.real
    for g, w in ((got.real, re), (got.imag, im)):
        assert np.array_equal(np.isnan(g), np.isnan(w))
        assert np.array_equal(g[np.isinf(w)], w[np.isinf(w)])
        fine = np.isfinite(w)
        assert np.allclose(g[fine], w[fine], rtol=0, atol=1e-13)
