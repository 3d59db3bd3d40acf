"""The hybrid batch form's string kernel keeps what a launch per operator
refuses and reports: overlapping states, and an expired wait on the operator."""
import numpy as np
import pytest

from qrusty_gb300 import Batch, PauliOperator, QrError
from qrusty_gb300 import workloads as W
from tests.test_gpu_batch import make_batch

pytestmark = pytest.mark.gpu

STATES = [120, 2, 4]


def _batch(cuda):
    rng = np.random.default_rng(7)
    terms = [W.random_letters_op(rng, 14, 120), W.random_letters_op(rng, 6, 30),
             W.random_letters_op(rng, 13, 90)]
    # 480 tiles (more than two per SM, so the first CTA has some), 2 and 8
    ops, psis, ys = make_batch(terms, STATES, cuda, 8)
    b = Batch(ops, STATES)
    b.set_mode(2)
    return ops, psis, ys, b


def test_overlapping_states_are_refused(cuda):
    _, psis, ys, b = _batch(cuda)
    with pytest.raises(QrError, match="overlap"):
        b.apply([psis[0], psis[1], psis[2]], [psis[0], ys[1], ys[2]])
    b.apply(psis, ys)
    with pytest.raises(QrError, match="overlap"):  # also once the graph is made
        b.apply([ys[0], psis[1], psis[2]], [ys[0], ys[1], ys[2]])


@pytest.mark.parametrize("step", [0, 3, 5])
def test_withheld_copy_is_reported_by_the_operators(cuda, step):
    """A partner copy that never comes: the bounded wait runs out, every string
    operator of the batch reports it, and the next call is right."""
    import torch
    ops, psis, ys, b = _batch(cuda)
    ops[0].set_test_hooks(wait_ns=50_000_000, withhold_step=step)
    b.apply(psis, ys)
    for k in (0, 2):
        with pytest.raises(QrError, match="bounded mbarrier wait expired"):
            ops[k].sync_check()
    ops[1].sync_check()  # of six qubits, in the persistent kernel
    ops[0].set_test_hooks()
    again = [torch.empty_like(y) for y in ys]
    b.apply(psis, again)  # other pointers: the graph is made anew
    for op, p, y in zip(ops, psis, again):
        op.sync_check()
        want = op.apply(p.to(torch.complex128))
        assert float(torch.linalg.vector_norm(y - want)) <= 1e-6 * float(
            torch.linalg.vector_norm(want))
