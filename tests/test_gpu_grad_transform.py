"""complex128 term gradients on both sides of the work from which x groups of many
strings take the Walsh-Hadamard transform."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,strings", [(5, 32), (12, 511), (12, 590), (12, 700), (13, 257),
                                       (13, 300), (13, 500)])
@pytest.mark.parametrize("states", [1, 3])
def test_against_fp64(cuda, n, strings, states):
    import torch
    rng = np.random.default_rng(strings)
    x = np.concatenate([np.full(strings, 5), rng.integers(0, 1 << n, 7)]).astype(np.uint64)
    z = np.concatenate([rng.choice(1 << n, strings, replace=False),
                        rng.integers(0, 1 << n, 7)]).astype(np.uint64)
    T = len(x)
    phase = rng.integers(0, 4, T).astype(np.uint8)
    psi = W.random_state(rng, 1 << n, nstates=max(2, states))[:states]
    g = W.random_state(rng, 1 << n, nstates=max(2, states))[:states]
    op = PauliOperator(n, x, z, phase, np.ones(T, np.complex128))
    got = op.term_grad(torch.from_numpy(psi).to(cuda), torch.from_numpy(g).to(cuda))
    op.sync_check()
    got = got.cpu().numpy()
    r = np.arange(1 << n, dtype=np.int64)
    unit = np.array([1, 1j, -1, -1j])  # conjugates of 1, -i, -1, i
    # unit-norm states: the products' moduli add to at most 1 per state, a sum in
    # any order is off by at most a rounding of that per addition (both sides)
    tol = 2.0 * states * (1 << n) * 2.0 ** -53
    for k in rng.choice(T, 12, replace=False).tolist() + [0, strings - 1, strings, T - 1]:
        sign = 1.0 - 2.0 * (np.bitwise_count(r & np.int64(z[k])) & 1)
        want = unit[phase[k]] * (np.conj(psi[:, r ^ np.int64(x[k])]) * sign * g).sum()
        assert abs(got[k] - want) <= tol
