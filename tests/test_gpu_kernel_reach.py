"""Each kernel family of the product reached by name (``apply_form``): its bounded
waits run out, its 64-bit row words, and the edges of its blocks.

An expired wait is made as in the failure tests: one ring step's copy is never
issued, and the wait bound is 50 ms."""
import numpy as np
import pytest

from qrusty_gb300 import Batch, PauliOperator, QrError
from qrusty_gb300 import workloads as W
from tests.test_gpu_batch import check_against_oracle, make_batch

pytestmark = pytest.mark.gpu

WAIT_NS = 50_000_000


def _two_body(n, quads, seed):
    """Four-index Jordan-Wigner terms: eight strings on each x."""
    rng = np.random.default_rng(seed)
    xs, zs = [], []
    for _ in range(quads):
        i, j, k, l = sorted(int(v) for v in rng.choice(n, 4, replace=False))
        x = 1 << i | 1 << j | 1 << k | 1 << l
        between = ((1 << j) - (1 << (i + 1))) | ((1 << l) - (1 << (k + 1)))
        for bits in range(16):
            if bin(bits).count("1") % 2 == 0:
                z = between
                for b, q in enumerate((i, j, k, l)):
                    z ^= (bits >> b & 1) << q
                xs.append(x)
                zs.append(z)
    x, z = np.array(xs, np.uint64), np.array(zs, np.uint64)
    return W.Terms(n, x, z, (np.bitwise_count(x & z) % 4).astype(np.uint8),
                   rng.standard_normal(len(x)).astype(np.complex128))


def _letters(n, strings, seed):
    return W.random_letters_op(np.random.default_rng(seed), n, strings)


# form, dtype, states, terms, ring steps to withhold (-1: the first tile's last)
KERNELS = {
    "tables, one tile": ("tables", "complex64", 20, lambda: _letters(11, 200, 1), (0,)),
    "tables, several chunks": ("tables", "complex64", 1, lambda: _two_body(18, 250, 2), (0, 5, -1)),
    "strings over a cluster": ("strings", "complex64", 2, lambda: _letters(14, 300, 3), (0, 3, 11)),
    "strings, several rounds": ("strings", "complex64", 40, lambda: _letters(15, 200, 4), (0, 20)),
    "strings, two tiles a block": ("strings", "complex64", 1, lambda: _letters(20, 700, 5),
                                   (0, 3, 60)),
    "cosets": ("cosets", "complex64", 1, lambda: W.cfg2(n=18, npair=900, nz=300), (0, 4)),
    "rows, complex64": ("rows", "complex64", 1, lambda: W.cfg2(n=14, npair=600, nz=200), (0, 1)),
    "rows, complex128": ("rows", "complex128", 2, lambda: _letters(12, 300, 6), (0, 2, -1)),
}


def _case(cuda, name):
    import torch
    form, dtype, states, terms, steps = KERNELS[name]
    t = terms()
    op = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff)
    dt = getattr(torch, dtype)
    assert op.apply_form(dt, states) == form
    psi = W.random_state(np.random.default_rng(7), 1 << t.n, nstates=max(2, states))[:states]
    return t, op, torch.from_numpy(psi).to(cuda, dt), steps


@pytest.mark.parametrize("name", sorted(KERNELS))
def test_withheld_copy(cuda, name):
    import torch
    t, op, psi, steps = _case(cuda, name)
    want = torch.view_as_real(op.apply(psi))
    op.sync_check()
    info = op.info()
    last = info["nblocks"] - 1 if psi.dtype == torch.complex64 else (info["ngroups"] - 1) // 32
    for step in (last if k < 0 else k for k in steps):
        op.set_test_hooks(wait_ns=WAIT_NS, withhold_step=step)
        op.apply(psi)
        with pytest.raises(QrError, match="bounded mbarrier wait expired"):
            op.sync_check()
        op.set_test_hooks()
        for _ in range(2):
            assert torch.equal(torch.view_as_real(op.apply(psi)), want)
            op.sync_check()


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("name", sorted(KERNELS))
def test_wide_rows_are_identical(cuda, oracle, name, adjoint):
    import torch
    t, op, psi, _ = _case(cuda, name)
    narrow = op.apply(psi, adjoint=adjoint)
    op.set_test_hooks(force_wide=True)
    wide = op.apply(psi, adjoint=adjoint)
    op.sync_check()
    assert torch.equal(torch.view_as_real(narrow), torch.view_as_real(wide))
    cp = oracle.make_params(t.phase, t.coeff)
    if adjoint:
        cp = np.conj(cp) * (1.0 - 2.0 * (np.bitwise_count(t.x & t.z) & 1))
    p = psi[-1].cpu().numpy().astype(np.complex128)
    hi = min(1 << t.n, 8192)
    ref = oracle.apply_rows(t.x, t.z, cp, p, 0, hi)
    got = wide[-1, :hi].cpu().numpy()
    assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref)


# string kernel: one partner tile (n = 12, 33 states are above the rows limit),
# blocks at their capacity of 255 strings (a 32nd of the strings below 19 qubits,
# so from 8,160 on) and dense tiles at 19
@pytest.mark.parametrize("n,states,strings", [(12, 33, k) for k in (1, 2, 3, 15, 16, 17, 33, 512)] +
                         [(14, 2, 8159), (14, 2, 8160), (14, 3, 9000), (19, 1, 10000)])
def test_string_blocks(cuda, oracle, n, states, strings):
    import torch
    t = _letters(n, strings, strings)
    t.x[t.x == 0] = 1  # no diagonal
    op = PauliOperator(n, t.x, t.z, t.phase, t.coeff)
    assert op.apply_form(torch.complex64, states) == "strings"
    psi = W.random_state(np.random.default_rng(n), 1 << n, nstates=max(2, states))[:states]
    psi = psi.astype(np.complex64)
    y = op.apply(torch.from_numpy(psi).to(cuda)).cpu().numpy()
    op.sync_check()
    cp = oracle.make_params(t.phase, t.coeff)
    lo = (1 << n) - 4096
    for s in {0, states - 1}:
        ref = oracle.apply_rows(t.x, t.z, cp, psi[s].astype(np.complex128), lo, 1 << n)
        assert np.linalg.norm(y[s, lo:] - ref) <= 1e-6 * np.linalg.norm(ref)


@pytest.mark.parametrize("strings", [8159, 8160, 8161])
def test_string_batch_blocks(cuda, oracle, strings):
    terms = [_letters(14, strings, 1), _letters(13, 300, 2), _letters(6, 20, 3)]
    for t in terms[:2]:
        t.x[t.x == 0] = 1
    states = [10, 2, 1]
    ops, psis, ys = make_batch(terms, states, cuda, 4)
    b = Batch(ops, states)
    b.set_mode(2)
    b.apply(psis, ys)
    assert check_against_oracle(oracle, terms, psis, ys, range(3), rows=2048) <= 1e-6
