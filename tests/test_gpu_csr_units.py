"""CSR rows written in units and stages: bit-exact against the oracle at the
edges of stage geometry, unit tails and the in-pass fold of one group."""
import numpy as np
import pytest

from qrusty_gb300 import workloads as W
from tests.test_gpu_csr import check_csr

pytestmark = pytest.mark.gpu


def _rows(rng, n, count=48):
    return sorted({0, 1, 63, 64, (1 << n) - 1} | {int(v) for v in rng.integers(0, 1 << n, count)})


def _groups(rng, n, groups, terms):
    """terms strings over exactly `groups` distinct x masks."""
    xs = rng.choice(1 << n, groups, replace=False).astype(np.uint64)
    x = np.concatenate([xs, rng.choice(xs, terms - groups)])
    z = rng.integers(0, 1 << n, terms).astype(np.uint64)
    return x, z, rng.integers(0, 4, terms).astype(np.uint8), \
        (rng.standard_normal(terms) + 1j * rng.standard_normal(terms))


# one group per row up to the most the staged rows take (256), around the
# sizes where the chunk's rows and the stage's parts change
@pytest.mark.parametrize("groups", [1, 2, 10, 11, 12, 23, 46, 47, 64, 128, 255, 256, 257])
@pytest.mark.parametrize("n", [9, 13])
def test_stage_sizes(cuda, oracle, n, groups):
    rng = np.random.default_rng(groups * 31 + n)
    x, z, ph, c = _groups(rng, n, groups, groups + groups // 2)
    check_csr(oracle, n, x, z, ph, c, sample_rows=_rows(rng, n))


# one wide diagonal group of m terms among narrow ones: prefix only, a few and
# the most terms after it that are folded in the pass, and one more
@pytest.mark.parametrize("m", [6, 12, 13, 14, 19, 29, 30, 31, 40, 76, 77, 78, 90])
@pytest.mark.parametrize("kind", ["real", "imag", "complex", "zeros"])
def test_one_wide_group(cuda, oracle, m, kind):
    n, groups = 14, 70
    rng = np.random.default_rng(m)
    x = np.concatenate([np.zeros(m, np.uint64),
                        rng.choice((1 << n) - 1, groups, replace=False).astype(np.uint64) + np.uint64(1)])
    z = rng.integers(0, 1 << n, len(x)).astype(np.uint64)
    order = rng.permutation(len(x))
    x, z = x[order], z[order]
    ph = np.zeros(len(x), np.uint8)
    c = rng.standard_normal(len(x)) + 0j
    if kind == "imag":
        c = c * 1j
    elif kind == "complex":
        c = c + 1j * rng.standard_normal(len(x))
    elif kind == "zeros":
        c = np.where(rng.random(len(x)) < 0.5, -0.0, 0.0) + \
            1j * np.where(rng.random(len(x)) < 0.5, -0.0, 0.0)
    check_csr(oracle, n, x, z, ph, c, sample_rows=_rows(rng, n))


# several wide groups: values through the value buffer, few (kept ahead in
# shared memory) and many (read at their stage)
@pytest.mark.parametrize("wide", [1, 2, 3, 15, 16, 17, 40])
@pytest.mark.parametrize("narrow", [4, 60])
def test_several_wide_groups(cuda, oracle, wide, narrow):
    n = 12
    rng = np.random.default_rng(100 * wide + narrow)
    xs = rng.choice(1 << n, wide + narrow, replace=False).astype(np.uint64)
    x = np.concatenate([xs, np.repeat(xs[:wide], 30)])
    x = x[rng.permutation(len(x))]
    z = rng.integers(0, 1 << n, len(x)).astype(np.uint64)
    c = rng.standard_normal(len(x)) + 1j * rng.standard_normal(len(x))
    check_csr(oracle, n, x, z, np.zeros(len(x), np.uint8), c, sample_rows=_rows(rng, n))


# several units per block and a block that takes many of them
def test_many_units(cuda, oracle):
    rng = np.random.default_rng(5)
    t, _ = W.cfg1(with_state=False, n=18)
    check_csr(oracle, t.n, t.x, t.z, t.phase, t.coeff, sample_rows=_rows(rng, t.n, 300))
