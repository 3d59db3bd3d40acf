"""complex64 products of many states of fewer rows than a warp has lanes."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,states", [(1, 1), (1, 20000), (2, 9000), (3, 4097), (4, 2049),
                                      (4, 40000), (5, 1025), (5, 20000)])
def test_many_states(cuda, n, states):
    import torch
    rng = np.random.default_rng(n)
    t = W.random_letters_op(rng, n, 3 * n)
    op = PauliOperator(n, t.x, t.z, t.phase, t.coeff)
    assert n >= 5 or op.apply_form(torch.complex64, states) == "rows"
    psi = torch.from_numpy(W.random_state(rng, 1 << n, nstates=max(2, states))[:states]
                           .astype(np.complex64)).to(cuda)
    y = op.apply(psi)
    op.sync_check()
    want = op.apply(psi.to(torch.complex128))
    assert float(torch.linalg.vector_norm(y - want)) <= 1e-6 * float(torch.linalg.vector_norm(want))
