"""complex64 products by cosets of the row bits 8-11 (qr_apply_cosets.cu): x and
z masks with every pattern on those bits, Jordan-Wigner hops complete and with
strings missing, one and many partner tiles, the diagonal alone and beside
sub-groups.  Many states of few qubits reach the kernel too.  Tolerance: 1e-6
of the FP64 result's norm, the module's bound for complex64 products."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _check(cuda, oracle, t, states, adjoint=False):
    import torch
    rng = np.random.default_rng(t.T)
    psi = W.random_state(rng, 1 << t.n, nstates=max(2, states))[:states].astype(np.complex64)
    op = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff)
    p = torch.from_numpy(psi).to(cuda)
    got = op.apply(p, adjoint=adjoint).cpu().numpy()
    res = op.apply_axpby(p, p, 0.5j, 2.0).cpu().numpy()
    c1 = rng.standard_normal(t.T) + 1j * rng.standard_normal(t.T)
    op.set_coeffs_device(torch.from_numpy(c1).to(cuda))  # rewrites the tables in place
    upd = op.apply(p)
    op.sync_check()
    fresh = PauliOperator(t.n, t.x, t.z, t.phase, c1).apply(p)
    assert torch.equal(torch.view_as_real(upd), torch.view_as_real(fresh))
    cp = oracle.make_params(t.phase, t.coeff)
    ca = cp
    if adjoint:
        ca = np.conj(cp) * (1.0 - 2.0 * (np.bitwise_count(t.x & t.z) & 1))
    for s in sorted(rng.choice(states, min(states, 2), replace=False)):
        lo = 0 if t.n <= 12 else int(rng.integers(0, (1 << t.n) - 4096))
        hi = lo + min(4096, 1 << t.n)
        p64 = psi[s].astype(np.complex128)
        ref = oracle.apply_rows(t.x, t.z, ca, p64, lo, hi)
        assert np.linalg.norm(got[s, lo:hi] - ref) <= TOL * np.linalg.norm(ref)
        ref = 0.5j * oracle.apply_rows(t.x, t.z, cp, p64, lo, hi) + 2.0 * p64[lo:hi]
        assert np.linalg.norm(res[s, lo:hi] - ref) <= TOL * np.linalg.norm(ref)


def _terms(n, x, z, rng):
    T = len(x)
    c = rng.standard_normal(T) + 1j * rng.standard_normal(T)
    return W.Terms(n, np.asarray(x, np.uint64), np.asarray(z, np.uint64),
                   rng.integers(0, 4, T).astype(np.uint8), c)


def _hops(n, pairs, rng, letters=4):
    """X / Y at i and j with Z between: `letters` of the four combinations."""
    xs, zs = [], []
    for i, j in pairs:
        for k in rng.choice(4, letters, replace=False):
            xs.append(1 << i | 1 << j)
            zs.append(((1 << j) - (1 << (i + 1))) | (int(k) & 1) << i | (int(k) >> 1) << j)
    return _terms(n, xs, zs, rng)


@pytest.mark.parametrize("n,states", [(18, 1), (13, 20), (12, 40)])
@pytest.mark.parametrize("letters", [4, 3, 2])
def test_jordan_wigner_hops(cuda, oracle, n, states, letters):
    """Every pair: complete hops take the quads, the others the dispatch."""
    rng = np.random.default_rng(n + letters)
    pairs = [(i, j) for i in range(n) for j in range(i + 1, n)]
    if letters == 2:  # still more strings than the string-by-string kernel takes
        pairs = [q for q in pairs if q[0] in (8, 9, 10, 11) or q[1] in (8, 9, 10, 11)] * 2
    _check(cuda, oracle, _hops(n, pairs, rng, letters), states, adjoint=letters == 3)


@pytest.mark.parametrize("n,states", [(18, 1), (14, 9)])
@pytest.mark.parametrize("seed", range(4))
def test_every_register_pattern(cuda, oracle, n, states, seed):
    """x over all patterns of bits 8-11 on few outer masks (cosets of several x
    groups), two to five strings each."""
    rng = np.random.default_rng(seed)
    xs, zs = [], []
    for outer in rng.choice(1 << (n - 4), 5, replace=False):
        out = (int(outer) & 255) | (int(outer) >> 8) << 12
        for reg in rng.choice(16, 11, replace=False):
            k = int(rng.integers(2, 6))
            z = int(rng.integers(0, 1 << n))
            flips = [0] + [1 << int(b) for b in rng.choice(n, 4, replace=False)]
            xs += [out | int(reg) << 8] * k
            zs += [z ^ flips[q] for q in range(k)]
    _check(cuda, oracle, _terms(n, xs, zs, rng), states, adjoint=bool(seed & 1))


@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 7])
@pytest.mark.parametrize("diag", [False, True])
def test_few_partner_tiles(cuda, oracle, tiles, diag):
    """Odd and even numbers of partner tiles; the diagonal on a tile without
    sub-groups or beside them."""
    n, rng = 18, np.random.default_rng(tiles)
    xs, zs = [], []
    for h in rng.choice(np.arange(1, 64), tiles, replace=False):
        x = int(h) << 12 | int(rng.integers(0, 4096))
        z = int(rng.integers(0, 1 << n))
        for b in (0, 1 << 9, 1 << 17, 1 << 9 | 1 << 17):
            xs.append(x)
            zs.append(z ^ b)
    if diag:
        xs += [0] * 8
        zs += [1 << b for b in (0, 3, 8, 9, 11, 12, 15, 17)]
    _check(cuda, oracle, _terms(n, xs, zs, rng), 1)


def test_chain_with_infinite_and_nan_amplitudes(cuda):
    import torch
    t, _ = W.cfg1(with_state=False, n=18)
    rng = np.random.default_rng(1)
    psi = W.random_state(rng, 1 << 18).astype(np.complex64)
    bad = np.array([5, 1 << 17])
    psi[bad] = [complex(np.inf, 1), complex(0, np.nan)]
    y = PauliOperator(18, t.x, t.z, t.phase, t.coeff).apply(torch.from_numpy(psi).to(cuda))
    y = y.cpu().numpy()
    hit = np.zeros(1 << 18, dtype=bool)
    for x in t.x.astype(np.int64):
        hit[bad ^ x] = True
    assert np.isnan(y.real[hit]).all() and np.isnan(y.imag[hit]).all()
    assert np.isfinite(y[~hit]).all()


def test_withheld_copy(cuda):
    """A partner copy that never comes: the bounded wait runs out, the error is
    reported, and the next product is right."""
    import torch
    from qrusty_gb300 import QrError
    t = W.cfg2(n=18, npair=900, nz=300)
    op = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff)
    psi = torch.randn(1 << 18, 2, device=cuda, dtype=torch.float32)
    psi = torch.view_as_complex(psi)
    want = op.apply(psi)
    op.sync_check()
    for step in (0, 2, 5):
        op.set_test_hooks(wait_ns=50_000_000, withhold_step=step)
        op.apply(psi)
        with pytest.raises(QrError, match="bounded mbarrier wait expired"):
            op.sync_check()
        op.set_test_hooks()
        assert torch.equal(torch.view_as_real(op.apply(psi)), torch.view_as_real(want))
        op.sync_check()
