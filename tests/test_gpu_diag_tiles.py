"""The precomputed diagonal of many Z strings over the tile sizes of its
transform: each entry is the sum of the signed coefficients."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator

pytestmark = pytest.mark.gpu


# tiles of all rows, of 2^8, 2^9, 2^10, 2^11 and 2^12, by rows and by terms
@pytest.mark.parametrize("n,terms", [(5, 31), (8, 255), (9, 300), (14, 300), (15, 20000),
                                     (16, 60000), (18, 500), (18, 5000), (19, 5000), (20, 5000)])
@pytest.mark.parametrize("imaginary", [False, True])
def test_every_entry(cuda, n, terms, imaginary):
    import torch
    rng = np.random.default_rng(terms)
    z = rng.choice(1 << n, terms, replace=False).astype(np.uint64)
    c = rng.standard_normal(terms) + (1j * rng.standard_normal(terms) if imaginary else 0)
    op = PauliOperator(n, np.zeros(terms, np.uint64), z, np.zeros(terms, np.uint8), c)
    one = torch.ones(1 << n, dtype=torch.complex128, device=cuda)
    y = op.apply(one).cpu().numpy()
    op.set_coeffs_device(torch.from_numpy(2.0 * c + 0j).to(cuda))
    y2 = op.apply(one).cpu().numpy()
    op.sync_check()
    w = np.zeros(1 << n, np.complex128)
    w[z.astype(np.int64)] = c
    for b in range(n):  # Walsh-Hadamard transform
        w = w.reshape(-1, 2, 1 << b)
        w = np.stack([w[:, 0] + w[:, 1], w[:, 0] - w[:, 1]], axis=1)
    w = w.reshape(-1)
    # two sums of the same terms, each off by a rounding of the moduli's sum per
    # addition at most, along chains of at most terms (bins) + n (transform)
    tol = 2.0 * (terms + n) * 2.0 ** -53 * np.abs(c).sum()
    assert np.abs(y - w).max() <= tol
    assert np.array_equal(y2, 2.0 * y)
