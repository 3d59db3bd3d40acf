"""complex128 products of many states: a row is split over as many warps as the
rows of the call leave idle, at the edges of that rule."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu


# 16 slices up to 2^14 rows, 8 to 2^15, 4 below 2^20, 2 below 2^21 and for states
# of fewer than 512 rows, then none
@pytest.mark.parametrize("n,states", [(9, 32), (9, 33), (9, 64), (9, 65), (9, 2047), (9, 2048),
                                      (9, 4095), (9, 4096), (8, 8192), (3, 5000), (1, 40000)])
def test_states_against_fp64(cuda, oracle, n, states):
    import torch
    rng = np.random.default_rng(n + states)
    t = W.random_letters_op(rng, n, 3 if n == 1 else 40)
    t.coeff = t.coeff + 1j * rng.standard_normal(t.T)
    psi = W.random_state(rng, 1 << n, nstates=states)
    op = PauliOperator(n, t.x, t.z, t.phase, t.coeff)
    y = op.apply(torch.from_numpy(psi).to(cuda)).cpu().numpy()
    op.sync_check()
    assert np.array_equal(y, op.apply(psi))  # host states, one launch each: the same split
    cp = oracle.make_params(t.phase, t.coeff)
    # a row's sum of T products in any order: at most a rounding of the moduli's
    # sum per operation, twice (both sides)
    tol = 2.0 * (4 * t.T) * 2.0 ** -53 * np.abs(cp).sum()
    for s in sorted({0, 1, states // 2, states - 1}):
        ref = oracle.apply(n, t.x, t.z, cp, psi[s])
        assert np.abs(y[s] - ref).max() <= tol * np.abs(psi[s]).max()
