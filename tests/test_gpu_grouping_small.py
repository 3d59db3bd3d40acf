"""Short term lists are grouped by counting, longer ones by the sorts; few
groups get their CSR tables from one block.  Both sides of each line, and the
tile and block edges, against numpy and the oracle."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from tests.test_gpu_csr import check_csr
from tests.test_gpu_grouping import _case, _expected

pytestmark = pytest.mark.gpu


def check_groups(t):
    got = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff).groups()
    gx, goff, order, mmap, _ = _expected(t.x, t.z)
    for name, want in (("gx", gx), ("goff", goff), ("order", order), ("mmap", mmap)):
        assert np.array_equal(got[name], want), name


@pytest.mark.parametrize("T", [1, 2, 127, 128, 129, 1023, 1024, 1025, 2049, 4095, 4096, 4097])
@pytest.mark.parametrize("n,xbits,zbits", [(63, 63, 63), (20, 2, 3), (13, 13, 1)])
def test_lengths(cuda, T, n, xbits, zbits):
    check_groups(_case(np.random.default_rng(T), n, T, xbits, zbits))


# top-bit masks through the sorts' eighth pass
def test_long_top_bit(cuda):
    check_groups(_case(np.random.default_rng(3), 63, 5000, 63, 63))


@pytest.mark.parametrize("groups", [1, 31, 32, 33, 511, 512, 513])
@pytest.mark.parametrize("wide", [0, 1, 9])
def test_structure(cuda, oracle, groups, wide):
    n = 10
    rng = np.random.default_rng(groups + wide)
    wide = min(wide, groups)
    xs = rng.choice(1 << n, groups, replace=False).astype(np.uint64)
    x = np.concatenate([xs, np.repeat(xs[:wide], 25), rng.choice(xs, groups // 2)])
    x = x[rng.permutation(len(x))]
    z = rng.integers(0, 1 << n, len(x)).astype(np.uint64)
    ph = rng.integers(0, 4, len(x)).astype(np.uint8)
    c = rng.standard_normal(len(x)) + 1j * rng.standard_normal(len(x))
    check_csr(oracle, n, x, z, ph, c, sample_rows=[0, 1, 511, 512, 700, 1023])
