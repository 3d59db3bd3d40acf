"""Term gradients of x groups with many strings (one Walsh-Hadamard transform
per 256 rows, qr_reduce.cu): the group sizes at which strings change over and
batches split, states smaller than a transform, both dtypes, beside strings
that go one by one.  Tolerances as for the other term gradients: 1e-12
(complex128) and 1e-5 (complex64) relative to the FP64 definition."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _terms(rng, n, sizes):
    xs, zs = [], []
    for x, k in zip(rng.choice(1 << n, len(sizes), replace=False), sizes):
        k = min(k, 1 << n)
        xs.append(np.full(k, x))
        zs.append(rng.choice(1 << n, k, replace=False))
    x, z = np.concatenate(xs), np.concatenate(zs)
    at = rng.permutation(len(x))
    x, z = x[at], z[at]
    x, z = np.concatenate([x, x[:3]]), np.concatenate([z, z[:3]])  # merged duplicates
    T = len(x)
    return (x.astype(np.uint64), z.astype(np.uint64), rng.integers(0, 4, T).astype(np.uint8),
            rng.standard_normal(T).astype(np.complex128))


@pytest.mark.parametrize("n,states,sizes", [
    (3, 1, [8, 7, 1]), (5, 3, [32, 9, 8, 7, 2]), (7, 1, [128, 100, 1]), (8, 2, [256, 31, 33, 3]),
    (9, 1, [255, 256, 257, 8]), (12, 1, [600, 64, 7, 8, 1, 1, 1]), (13, 3, [40, 8, 1, 2]),
    (14, 1, [513, 16]), (15, 1, [95] + [3] * 30)])
def test_groups(cuda, oracle, n, states, sizes):
    import torch
    rng = np.random.default_rng(n)
    x, z, ph, c = _terms(rng, n, sizes)
    op = PauliOperator(n, x, z, ph, c)
    psi = W.random_state(rng, 1 << n, nstates=max(2, states))[:states]
    g = W.random_state(rng, 1 << n, nstates=max(2, states))[:states]
    for dt, tol in ((np.complex128, 1e-12), (np.complex64, 1e-5)):
        p, q = psi.astype(dt), g.astype(dt)
        want = sum(oracle.term_grad(n, x, z, ph, p[s].astype(np.complex128),
                                    q[s].astype(np.complex128)) for s in range(states))
        pt, gt = torch.from_numpy(p.reshape(-1)).to(cuda), torch.from_numpy(q.reshape(-1)).to(cuda)
        got = op.term_grad(pt, gt)
        assert torch.equal(torch.view_as_real(got), torch.view_as_real(op.term_grad(pt, gt)))
        assert np.linalg.norm(got.cpu().numpy() - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("n", [6, 12, 14, 16, 20, 21])
@pytest.mark.parametrize("scale", [1.0, 1j, 0.5 - 2j])
def test_diagonal_of_the_apply_plans(cuda, n, scale):
    """The diagonal's transform on every tile width, real coefficients (whose
    imaginary half is left out) and complex ones: a pure-Z operator's product
    against the operator diagonal."""
    import torch
    rng = np.random.default_rng(n)
    z = rng.choice(1 << n, 30, replace=False).astype(np.uint64)
    c = rng.standard_normal(30) * scale
    op = PauliOperator(n, np.zeros(30, np.uint64), z, np.zeros(30, np.uint8), c)
    psi = torch.randn(1 << n, 2, device=cuda, dtype=torch.float64)
    psi = torch.view_as_complex(psi)
    want = op.diagonal() * psi
    got = op.apply(psi)
    assert torch.linalg.vector_norm(got - want) <= 1e-13 * torch.linalg.vector_norm(want)
    got = op.apply(psi.to(torch.complex64)).to(torch.complex128)
    assert torch.linalg.vector_norm(got - want) <= 1e-6 * torch.linalg.vector_norm(want)
