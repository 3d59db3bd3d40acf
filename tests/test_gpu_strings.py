"""Compensated complex64 product string by string (qr_apply_strings.cu): the
edges of its blocks (255 strings, one or two partner tiles), of the split over
a cluster (few tiles), and of its register and thread bits.  Tolerance: the
module's bound for complex64 products, 1e-6 of the FP64 result's norm."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _op(n, x, rng, z=None):
    T = len(x)
    z = rng.integers(0, 1 << n, T) if z is None else z
    c = rng.standard_normal(T) + 1j * rng.standard_normal(T)
    c[::3] = c[::3].real
    c[1::3] = 1j * c[1::3].imag
    return W.Terms(n, np.asarray(x, np.uint64), np.asarray(z, np.uint64),
                   rng.integers(0, 4, T).astype(np.uint8), c)


def _check(cuda, oracle, t, states, adjoint=False, rows=4096):
    import torch
    rng = np.random.default_rng(t.T)
    psi = W.random_state(rng, 1 << t.n, nstates=max(2, states))[:states].astype(np.complex64)
    op = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff)
    p = torch.from_numpy(psi).to(cuda)
    got = op.apply(p, adjoint=adjoint)
    again = op.apply(p, adjoint=adjoint)
    v = op.apply_axpby(p, p, 0.5 - 2j, 1.25j) if not adjoint else None
    op.sync_check()
    assert torch.equal(got, again)
    cp = oracle.make_params(t.phase, t.coeff)
    if adjoint:  # (H^dagger) has the conjugated strings
        flip = 1.0 - 2.0 * (np.bitwise_count(t.x & t.z) & 1)
        cp = np.conj(cp) * flip
    lo = 0 if t.n <= 13 else int(rng.integers(0, (1 << t.n) - rows))
    hi = min(1 << t.n, lo + rows) if t.n > 13 else 1 << t.n
    got = got.cpu().numpy()
    for s in range(states):
        p64 = psi[s].astype(np.complex128)
        ref = oracle.apply_rows(t.x, t.z, cp, p64, lo, hi)
        assert np.linalg.norm(got[s, lo:hi] - ref) <= TOL * np.linalg.norm(ref)
        if v is not None:
            ref = (0.5 - 2j) * ref + 1.25j * p64[lo:hi]
            assert np.linalg.norm(v[s].cpu().numpy()[lo:hi] - ref) <= TOL * np.linalg.norm(ref)


@pytest.mark.parametrize("n", [12, 13, 16, 18, 19, 20])
@pytest.mark.parametrize("states", [1, 2, 5])
def test_sizes(cuda, oracle, n, states):
    rng = np.random.default_rng(n)
    _check(cuda, oracle, _op(n, rng.choice(np.arange(1, 1 << n), 300, replace=False), rng), states)


@pytest.mark.parametrize("n", [12, 19])
@pytest.mark.parametrize("strings", [1, 2, 3, 7, 8, 9, 15, 16, 17, 254, 255, 256, 257, 511])
def test_strings_of_one_tile(cuda, oracle, n, strings):
    """All strings on one partner tile: odd and even counts, block capacity."""
    rng = np.random.default_rng(strings)
    x = rng.choice(4096, strings, replace=False) | (rng.integers(0, 2) << (n - 1) & ~4095)
    _check(cuda, oracle, _op(n, x, rng), 1)


@pytest.mark.parametrize("first", [100, 254, 255])
def test_two_tiles_share_a_block(cuda, oracle, first):
    rng = np.random.default_rng(first)
    n = 19
    x = np.concatenate([rng.choice(4096, first, replace=False) | tile << 12
                        for tile in (1, 2, 5, 127)] + [[3 << 12, 9 << 12]])
    _check(cuda, oracle, _op(n, x, rng), 1, adjoint=True)


@pytest.mark.parametrize("n", [12, 14, 19])
def test_with_a_diagonal(cuda, oracle, n):
    """x = 0 strings of z rank > 4 become a diagonal, here beside strings on
    tile 0 or with none there."""
    rng = np.random.default_rng(n)
    zero = np.zeros(9, dtype=np.int64)
    for other in (rng.choice(np.arange(1, 4096), 40, replace=False),
                  rng.choice(np.arange(1, 4096), 40, replace=False) | 1 << (n - 1)):
        _check(cuda, oracle, _op(n, np.concatenate([zero, other]), rng), 2)


@pytest.mark.parametrize("n", [13, 19])
def test_infinite_and_nan_amplitudes(cuda, oracle, n):
    """A row that meets an infinite or NaN amplitude is NaN in both parts (the
    compensated sum of 0 * inf and inf), every other row stays finite."""
    import torch
    rng = np.random.default_rng(n)
    t = _op(n, rng.choice(np.arange(1, 1 << n), 60, replace=False), rng)
    t.coeff = t.coeff.real.astype(np.complex128)
    psi = W.random_state(rng, 1 << n).astype(np.complex64)
    bad = np.array([3, 1 << 11, (1 << n) - 1])
    psi[bad] = [complex(np.inf, 1), complex(0, -np.inf), complex(np.nan, 2)]
    op = PauliOperator(n, t.x, t.z, t.phase, t.coeff)
    y = op.apply(torch.from_numpy(psi).to(cuda)).cpu().numpy()
    op.sync_check()
    hit = np.zeros(1 << n, dtype=bool)
    for x in t.x.astype(np.int64):
        hit[bad ^ x] = True
    assert np.isnan(y.real[hit]).all() and np.isnan(y.imag[hit]).all()
    psi[bad] = 0
    cp = oracle.make_params(t.phase, t.coeff)
    ref = oracle.apply(n, t.x, t.z, cp, psi.astype(np.complex128))[~hit]
    assert np.linalg.norm(y[~hit] - ref) <= TOL * np.linalg.norm(ref)
