"""CSR x vector: which loop a matrix takes is read off its first row; every other
row's sum is the same bits in both, and right."""
import numpy as np
import pytest

from qrusty_gb300 import _lib

pytestmark = pytest.mark.gpu


def _spmv(cuda, indptr, indices, data, v):
    import torch
    t = [torch.from_numpy(a).to(cuda) for a in (indptr, indices, data, v)]
    y = torch.empty(len(indptr) - 1, dtype=torch.complex128, device=cuda)
    _lib.check(_lib.load().qr_csr_spmv(y.numel(), v.size, *(a.data_ptr() for a in t),
                                       y.data_ptr(), torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    return y.cpu().numpy()


# below and above the 2^14 rows where a row's lanes go from 16 to 4; lengths of
# one to several steps, ragged, and rows that are empty
@pytest.mark.parametrize("rows", [1, 33, 1000, (1 << 14) + 5])
@pytest.mark.parametrize("mean", [1, 5, 24, 97])
def test_both_loops_agree(cuda, rows, mean):
    rng = np.random.default_rng(rows + mean)
    ncols = rows + 7
    length = rng.poisson(mean, rows)
    length[0] = mean
    if rows > 2:
        length[rows // 2] = 0
    indptr = np.concatenate([[0], np.cumsum(length)]).astype(np.int64)
    nnz = int(indptr[-1])
    indices = rng.integers(0, ncols, nnz)
    data = rng.standard_normal(nnz) + 1j * rng.standard_normal(nnz)
    kind = rng.integers(0, 3, nnz)  # real, imaginary, both
    data[kind == 0] = data[kind == 0].real
    data[kind == 1] = 1j * data[kind == 1].imag
    v = rng.standard_normal(ncols) + 1j * rng.standard_normal(ncols)
    row = np.repeat(np.arange(rows), length)
    data[:mean] = data[:mean].real
    if nnz > mean + 3:  # columns out of range are skipped, whatever is stored there
        indices[mean], data[mean] = ncols + 3, complex(np.inf, np.nan)
        v[3] = complex(np.inf, 1.0)  # rows that meet it keep 0 * inf
        indices[:mean][indices[:mean] == 3] = 4
        indices[mean + 1], data[mean + 1] = 3, 2.0
    real_first = _spmv(cuda, indptr, indices, data, v)
    other = data.copy()
    other[:mean] += 0.5j
    mixed_first = _spmv(cuda, indptr, indices, other, v)
    assert np.array_equal(real_first[1:], mixed_first[1:], equal_nan=True)
    assert np.array_equal(np.isnan(real_first.real), np.isnan(mixed_first.real))
    ok = indices < ncols
    with np.errstate(invalid="ignore"):
        for d, got in ((data, real_first), (other, mixed_first)):
            want = np.zeros(rows, np.complex128)
            prod = d[ok] * v[indices[ok]]
            np.add.at(want, row[ok], prod)
            size = np.zeros(rows)
            np.add.at(size, row[ok], np.abs(d[ok]) * np.abs(v[indices[ok]]))
            fin = np.isfinite(want)
            # a row's sum in another order: at most a rounding of the moduli's
            # sum per product and addition
            tol = 4.0 * (length + 2) * 2.0 ** -53 * size
            assert (np.abs(got - want)[fin] <= tol[fin]).all()
            assert not np.isfinite(got[~fin]).any()
