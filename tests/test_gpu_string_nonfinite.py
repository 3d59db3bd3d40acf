"""String kernel, states of infinite or NaN amplitudes: the rows that meet one
cost no more than the bounded waits allow, however many strings there are."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu

WAIT_NS = 2_000_000  # a ring step takes microseconds


@pytest.mark.parametrize("value", [complex(np.nan, 0), complex(0, np.inf)])
def test_state_of_one_nonfinite_part(cuda, value):
    import torch
    t = W.random_letters_op(np.random.default_rng(9), 20, 20000)
    op = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff)
    psi = torch.full((1 << t.n,), value, dtype=torch.complex64, device=cuda)
    op.apply(psi)  # plan
    op.sync_check()
    op.set_test_hooks(wait_ns=WAIT_NS)
    y = op.apply(psi)
    op.sync_check()
    assert bool(torch.isnan(torch.view_as_real(y)).all())


def _terms(n, strings, seed):
    """Distinct x, real coefficients."""
    rng = np.random.default_rng(seed)
    x = rng.choice(np.arange(1, 1 << n), strings, replace=False).astype(np.uint64)
    z = rng.integers(0, 1 << n, strings).astype(np.uint64)
    phase = (np.bitwise_count(x & z) % 4).astype(np.uint8)  # c' real or imaginary
    return W.Terms(n, x, z, phase, rng.standard_normal(strings).astype(np.complex128))


# one state of 15-18 qubits is split over a cluster, larger ones are not
@pytest.mark.parametrize("n,strings", [(15, 300), (16, 1000), (18, 64), (20, 500)])
def test_rows_that_meet_one(cuda, oracle, n, strings):
    """They are NaN in both parts, every other row is what it was."""
    import torch
    t = _terms(n, strings, n)
    op = PauliOperator(n, t.x, t.z, t.phase, t.coeff)
    assert op.apply_form(torch.complex64) == "strings"
    psi = W.random_state(np.random.default_rng(1), 1 << n).astype(np.complex64)
    clean = op.apply(torch.from_numpy(psi).to(cuda)).cpu().numpy()
    bad = np.array([3, 1 << 11, 1 << (n - 1), (1 << n) - 1])
    psi[bad] = [complex(np.inf, 1), complex(0, -np.inf), complex(np.nan, 2), complex(1, np.nan)]
    p = torch.from_numpy(psi).to(cuda)
    hit = np.zeros(1 << n, bool)
    for b in bad:
        hit[(np.int64(b) ^ t.x.astype(np.int64))] = True
    for y in (op.apply(p), op.apply_axpby(p, torch.zeros_like(p), 1.0, 0.0)):
        y = y.cpu().numpy()
        assert np.isnan(y.real[hit]).all() and np.isnan(y.imag[hit]).all()
        assert np.array_equal(y[~hit], clean[~hit])
    op.sync_check()


@pytest.mark.parametrize("n,strings", [(15, 300), (20, 500)])
def test_overflow_stays_in_its_part(cuda, n, strings):
    """A finite amplitude whose products leave the range: NaN in the part that
    they are added to, the other part as with any real amplitude there."""
    import torch
    t = _terms(n, strings, n + 1)
    t.z[:] = 0  # real coefficients throughout
    t.phase[:] = 0
    t.coeff[:] = 2.0
    op = PauliOperator(n, t.x, t.z, t.phase, t.coeff)
    assert op.apply_form(torch.complex64) == "strings"
    psi = W.random_state(np.random.default_rng(2), 1 << n).astype(np.complex64)
    at = 77
    psi[at] = complex(1.0, psi[at].imag)
    want = op.apply(torch.from_numpy(psi).to(cuda)).cpu().numpy()
    psi[at] = complex(3e38, psi[at].imag)
    y = op.apply(torch.from_numpy(psi).to(cuda)).cpu().numpy()
    op.sync_check()
    hit = np.zeros(1 << n, bool)
    hit[at ^ t.x.astype(np.int64)] = True
    assert np.isnan(y.real[hit]).all()
    assert np.array_equal(y.imag, want.imag)
    assert np.array_equal(y.real[~hit], want.real[~hit])
