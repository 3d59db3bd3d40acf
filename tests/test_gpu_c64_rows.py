"""complex64 products around the number of rows at which they change from the
rows kernel (qr_apply_rows.cu) to the tile kernels, and the rows kernel's own
splits.  Tolerance: 1e-6 of the FP64 result's norm, the module's bound."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _dense_groups(n, groups, per, rng):
    """x groups of `per` strings with random z masks (rank up to per - 1)."""
    x = np.repeat(rng.choice(1 << n, groups, replace=False), per).astype(np.uint64)
    T = len(x)
    c = rng.standard_normal(T) + 1j * rng.standard_normal(T)
    return W.Terms(n, x, rng.integers(0, 1 << n, T).astype(np.uint64),
                   rng.integers(0, 4, T).astype(np.uint8), c)


def _check(cuda, oracle, t, states, rows=2048):
    import torch
    rng = np.random.default_rng(t.T + states)
    psi = W.random_state(rng, 1 << t.n, nstates=max(2, states))[:states].astype(np.complex64)
    op = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff)
    p = torch.from_numpy(psi).to(cuda)
    got = op.apply(p)
    host = op.apply(psi.reshape(-1)).reshape(psi.shape)
    res = op.apply_axpby(p, p, 2.0, -0.5j).cpu().numpy()
    op.sync_check()
    got = got.cpu().numpy()
    assert np.array_equal(got, host)  # state by state on the host path, same bits
    cp = oracle.make_params(t.phase, t.coeff)
    for s in sorted(rng.choice(states, min(states, 3), replace=False)):
        lo = 0 if 1 << t.n <= rows else int(rng.integers(0, (1 << t.n) - rows))
        hi = min(1 << t.n, lo + rows)
        p64 = psi[s].astype(np.complex128)
        ref = oracle.apply_rows(t.x, t.z, cp, p64, lo, hi)
        assert np.linalg.norm(got[s, lo:hi] - ref) <= TOL * np.linalg.norm(ref)
        ref = 2.0 * ref - 0.5j * p64[lo:hi]
        assert np.linalg.norm(res[s, lo:hi] - ref) <= TOL * np.linalg.norm(ref)


# rows = states * 2^n: one per split of the rows kernel, the limits and beyond
@pytest.mark.parametrize("n,states", [(1, 1), (3, 5), (6, 1), (8, 1), (8, 128), (8, 130), (11, 4),
                                      (11, 16), (11, 17), (12, 2), (12, 3), (13, 1), (14, 1)])
def test_random_letters(cuda, oracle, n, states):
    rng = np.random.default_rng(n + states)
    t = W.random_letters_op(rng, n, 90)
    t.coeff = t.coeff * (0.8 + 0.6j)
    _check(cuda, oracle, t, states)


@pytest.mark.parametrize("n,states", [(7, 2), (12, 1), (12, 4), (13, 4), (15, 2), (15, 4), (17, 1),
                                      (17, 2), (18, 1)])
@pytest.mark.parametrize("groups,per", [(33, 3), (64, 40), (300, 6)])
def test_many_strings_per_group(cuda, oracle, n, states, groups, per):
    """Ranks up to 4 in one table, above it split; beyond the rows limit the
    paired kernel (33 groups) and the table rebuilt per chunk (the others)."""
    rng = np.random.default_rng(n * groups)
    if groups > 1 << n:
        groups = 1 << n
    _check(cuda, oracle, _dense_groups(n, groups, per, rng), states)


@pytest.mark.parametrize("n", [13, 16])
def test_infinite_and_nan_amplitudes(cuda, n):
    """Rows that meet one are NaN in both parts, all others finite."""
    import torch
    t, _ = W.cfg1(with_state=False, n=n)
    rng = np.random.default_rng(n)
    psi = W.random_state(rng, 1 << n).astype(np.complex64)
    bad = np.array([9, 1 << (n - 1)])
    psi[bad] = [complex(-np.inf, 1), complex(0, np.nan)]
    y = PauliOperator(n, t.x, t.z, t.phase, t.coeff).apply(torch.from_numpy(psi).to(cuda))
    y = y.cpu().numpy()
    hit = np.zeros(1 << n, dtype=bool)
    for x in t.x.astype(np.int64):
        hit[bad ^ x] = True
    assert np.isnan(y.real[hit]).all() and np.isnan(y.imag[hit]).all()
    assert np.isfinite(y[~hit]).all()
