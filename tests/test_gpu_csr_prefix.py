"""Memory of the CSR's prefix tables: 32 KB per x group folded term by term
where there are many such groups or few rows."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,groups", [(14, 2000), (13, 200)])
def test_prefix_tables_are_bounded(cuda, n, groups):
    import torch
    rng = np.random.default_rng(n)
    x = np.repeat(rng.choice(1 << n, groups, replace=False), 30).astype(np.uint64)
    z = rng.integers(0, 1 << n, x.size).astype(np.uint64)
    op = PauliOperator(n, x, z, np.zeros(x.size, np.uint8), rng.standard_normal(x.size))
    out = torch.empty(1 << n, dtype=torch.complex128, device=cuda)
    del out
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    op.diagonal()  # builds the CSR tables, no matrix
    torch.cuda.synchronize()
    used = before - torch.cuda.mem_get_info()[0]
    # 2^11 classes of 16 bytes per group, descriptors (some 400 bytes and 2 per
    # term), and the allocators' granularity
    assert used <= groups * (2048 * 16 + 1024) + (24 << 20)
