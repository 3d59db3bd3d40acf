"""Real factors on the complex128 paths: CSR * vector, ax / axpy / axpby and
precond2 leave out the products of a zero part, and must return what the full
products give -- the helpers bit for bit (signed zeros, infinities and NaNs
included), CSR * vector within 1e-12 and with the same infinite and NaN rows."""
import numpy as np
import pytest

from qrusty_gb300 import _lib, ax, axpby, axpy, precond2

pytestmark = pytest.mark.gpu

SPECIAL = np.array([0.0, -0.0, 1.0, -1.0, 3e-310, -5e-324, 1e300, -1e-300, np.inf, -np.inf,
                    np.nan, 0.3, -7.25])


def _vectors():
    a, b = np.meshgrid(SPECIAL, SPECIAL)
    v = np.empty(a.size, dtype=np.complex128)
    v.real, v.imag = a.ravel(), b.ravel()
    return np.repeat(v, v.size), np.tile(v, v.size)


def _same(got, want):
    for g, w in ((got.real, want.real), (got.imag, want.imag)):
        nan = np.isnan(w)
        assert np.array_equal(np.isnan(g), nan)
        assert np.array_equal(g[~nan].view(np.uint64), w[~nan].view(np.uint64))


@pytest.mark.parametrize("a,b", [(1.0, -2.5), (-1.0, 1.0), (0.0, 3.0), (-0.0, 0.0),
                                 (1e-300, complex(2.0, -0.0)), (2.0, 1j), (1 - 1j, 1.0)])
def test_scalars_bit_exact(cuda, oracle, a, b):
    import torch
    x, y = _vectors()
    xd, yd = torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda)
    with np.errstate(all="ignore"):
        _same(ax(a, xd).cpu().numpy(), oracle.vec("ax", x, a=a))
        _same(axpy(a, xd, yd).cpu().numpy(), oracle.vec("axpy", x, y, a))
        _same(axpby(a, xd, b, yd).cpu().numpy(), oracle.vec("axpby", x, y, a, b))


@pytest.mark.parametrize("e", [0.0, -0.5, 0.25 + 0.5j])
@pytest.mark.parametrize("tol", [0.0, 1e-14, 0.1, np.inf, np.nan, -1.0])
def test_precond2_bit_exact(cuda, oracle, e, tol):
    import torch
    x, y = _vectors()
    # pivots on both sides of tol, real and complex, away from it by 1 %
    t = 0.1 if not 0 < tol < 1 else tol
    near = e + t * np.array([0.3, 0.99, 1.01, 1.5, 1.99, 2.01, 0.7 + 0.69j, 0.7 + 0.73j, 1.4 + 1.45j])
    x = np.concatenate([x, near])
    y = np.concatenate([y, np.full(len(near), 1.5 - 0.5j)])
    got = precond2(torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda), e, tol)
    _same(got.cpu().numpy(), oracle.vec("precond2", x, y, e, tol=tol))


@pytest.mark.parametrize("kind", ["real", "imag", "complex", "mixed"])
@pytest.mark.parametrize("row", [1, 3, 4, 5, 44, 64, 70])
def test_spmv_parts(cuda, kind, row):
    import torch
    rng = np.random.default_rng(row)
    nrows, ncols = 517, 700
    col = np.stack([rng.choice(ncols, row, replace=False) for _ in range(nrows)])
    d = rng.standard_normal((nrows, row)) + 1j * rng.standard_normal((nrows, row))
    if kind == "real":
        d = d.real + 0j
    elif kind == "imag":
        d = 1j * d.imag
    elif kind == "mixed":
        d[::2] = d[::2].real
        d[1::4] = 1j * d[1::4].imag
    v = rng.standard_normal(ncols) + 1j * rng.standard_normal(ncols)
    v[5] = complex(np.inf, 1.0)
    v[9] = complex(2.0, np.nan)
    ip = np.arange(nrows + 1, dtype=np.int64) * row
    dev = [torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
           for a in (ip, col.ravel().astype(np.int64), d.ravel(), v)]
    out = torch.empty(nrows, dtype=torch.complex128, device=cuda)
    _lib.check(_lib.load().qr_csr_spmv(nrows, ncols, *[a.data_ptr() for a in dev],
                                       out.data_ptr(), None))
    got = out.cpu().numpy()
    with np.errstate(invalid="ignore"):
        x = v[col]
        re = (d.real * x.real - d.imag * x.imag).sum(axis=1)
        im = (d.real * x.imag + d.imag * x.real).sum(axis=1)
    for g, w in ((got.real, re), (got.imag, im)):
        fine = np.isfinite(w)
        assert np.array_equal(np.isnan(g), np.isnan(w))
        assert np.array_equal(g[np.isinf(w)], w[np.isinf(w)])
        assert np.linalg.norm(g[fine] - w[fine]) <= 1e-12 * np.linalg.norm(w[fine])
