"""The hybrid batch form's string kernel: operators of about one string per x
group share one launch, taking (operator, state, tile) items from a counter.
Against the FP64 oracle at the edges of its blocks and lists; the bound is the
batch's, 1e-6."""
import numpy as np
import pytest

from qrusty_gb300 import Batch
from qrusty_gb300 import workloads as W
from tests.test_gpu_batch import check_against_oracle, make_batch

pytestmark = pytest.mark.gpu


def _op(rng, n, T, diagonal=0, complex_coeff=False):
    t = W.random_letters_op(rng, n, T)
    if diagonal:
        x, z = t.x.copy(), t.z.copy()
        x[:diagonal] = 0
        z[:diagonal] = rng.choice(1 << n, diagonal, replace=False).astype(np.uint64)
        t = W.Terms(n, x, z, t.phase, t.coeff)
    if complex_coeff:
        t.coeff = t.coeff * (1 + 0.4j)
    return t


def _run(cuda, terms, nstates, seed=5):
    ops, psis, ys = make_batch(terms, nstates, cuda, seed)
    b = Batch(ops, nstates)
    b.set_mode(2)
    b.apply(psis, ys)
    return ops, psis, ys, b


# fewer items than SMs and several rounds of them; strings around a block's
# 16 and 255; a diagonal; complex coefficients; beside small operators (their
# own persistent kernel), a few-rows one and a spin chain (their own launches)
@pytest.mark.parametrize("states", [3, 9])
@pytest.mark.parametrize("strings", [5, 16, 17, 255, 256, 700])
def test_items(cuda, oracle, states, strings):
    rng = np.random.default_rng(strings + states)
    terms = [_op(rng, 12, strings), _op(rng, 14, strings, diagonal=40 if strings > 100 else 0),
             _op(rng, 15, strings, complex_coeff=True), _op(rng, 13, 2 * strings),
             _op(rng, 5, 20), _op(rng, 10, 60), W.cfg1(with_state=False, n=14)[0]]
    _, psis, ys, _ = _run(cuda, terms, [states] * len(terms))
    assert check_against_oracle(oracle, terms, psis, ys, range(len(terms))) <= 1e-6


def test_follows_coefficients(cuda, oracle):
    import torch
    rng = np.random.default_rng(11)
    terms = [_op(rng, 14, 300, diagonal=30), _op(rng, 13, 200), _op(rng, 15, 90)]
    ops, psis, ys, b = _run(cuda, terms, [4, 5, 3])
    for k, (op, t) in enumerate(zip(ops, terms)):
        t.coeff = t.coeff * (0.5 + k) + 0.25
        if k == 1:
            op.set_coeffs_device(torch.as_tensor(t.coeff, device=cuda))
        else:
            op.set_coeffs(t.coeff)
    b.apply(psis, ys)
    assert check_against_oracle(oracle, terms, psis, ys, range(len(terms))) <= 1e-6


def test_infinite_and_nan_amplitudes(cuda):
    """Rows that meet one are NaN in both parts, the others as without it."""
    rng = np.random.default_rng(3)
    terms = [_op(rng, 13, 120), _op(rng, 14, 60)]
    ops, psis, ys, b = _run(cuda, terms, [3, 2])
    clean = [y.cpu().numpy().copy() for y in ys]
    bad = [7, (1 << 13) + 5000]  # states 0 and 1 of the first operator
    psis[0][bad[0]] = complex(np.inf, 1)
    psis[0][bad[1]] = complex(0, np.nan)
    b.apply(psis, ys)
    got = [y.cpu().numpy() for y in ys]
    xs = np.unique(terms[0].x).astype(np.int64)
    hit = np.zeros(len(clean[0]), bool)
    for r in bad:
        hit[(r >> 13 << 13) + ((r & 8191) ^ xs)] = True
    assert np.isnan(got[0][hit].real).all() and np.isnan(got[0][hit].imag).all()
    assert np.array_equal(got[0][~hit], clean[0][~hit])
    assert np.array_equal(got[1], clean[1])
