"""The hybrid batch form's string kernel keeps what a launch per operator
refuses and reports: overlapping states, and an expired wait on the operator."""
import numpy as np
import pytest

from qrusty_gb300 import Batch, PauliOperator, QrError
from qrusty_gb300 import workloads as W
from tests.test_gpu_batch import make_batch

pytestmark = pytest.mark.gpu


def _batch(cuda):
    rng = np.random.default_rng(7)
    terms = [W.random_letters_op(rng, 14, 120), W.random_letters_op(rng, 6, 30),
             W.random_letters_op(rng, 13, 90)]
    ops, psis, ys = make_batch(terms, [25, 2, 4], cuda, 8)  # 100, 2 and 8 tiles
    b = Batch(ops, [25, 2, 4])
    b.set_mode(2)
    return ops, psis, ys, b


def test_overlapping_states_are_refused(cuda):
    _, psis, ys, b = _batch(cuda)
    with pytest.raises(QrError, match="overlap"):
        b.apply([psis[0], psis[1], psis[2]], [psis[0], ys[1], ys[2]])
    b.apply(psis, ys)
    with pytest.raises(QrError, match="overlap"):  # also once the graph is made
        b.apply([ys[0], psis[1], psis[2]], [ys[0], ys[1], ys[2]])
