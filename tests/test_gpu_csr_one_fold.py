"""CSR of operators with one x group folded term by term: by the staged fill, from
a value buffer, or in place after it; sampled rows bit for bit against make_row."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _with_diagonal(n, others, zs, seed):
    rng = np.random.default_rng(seed)
    x = np.concatenate([rng.choice(np.arange(1, 1 << n), others, replace=False), np.zeros(zs)])
    z = rng.integers(0, 1 << n, others + zs)
    return W.Terms(n, x.astype(np.uint64), z.astype(np.uint64),
                   rng.integers(0, 4, others + zs).astype(np.uint8),
                   rng.standard_normal(others + zs) + 1j * rng.standard_normal(others + zs))


# several classes per group: in place from 18 qubits on; else from 20
@pytest.mark.parametrize("t", [W.cfg2(n=17, npair=700, nz=150), W.cfg2(n=18, npair=700, nz=150),
                               _with_diagonal(19, 6, 120, 1), _with_diagonal(20, 6, 120, 2),
                               _with_diagonal(18, 40, 90, 3)], ids=lambda t: "n%d_%d" % (t.n, t.T))
def test_sampled_rows(cuda, oracle, t):
    op = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff)
    indptr, indices, data = op.csr_device()
    op.sync_check()
    G = int(indptr[1])
    cp = oracle.make_params(t.phase, t.coeff)
    rng = np.random.default_rng(4)
    last = (1 << t.n) - 1
    for r in [0, 1, last] + [int(v) for v in rng.integers(0, last, 60)]:
        cols, vals = oracle.make_row(t.x, t.z, cp, r)
        got_c = indices[r * G:(r + 1) * G].cpu().numpy().view(np.uint64)
        got_v = data[r * G:(r + 1) * G].cpu().numpy()
        assert np.array_equal(got_c, cols)
        assert np.array_equal(got_v.view(np.uint64), np.ascontiguousarray(vals).view(np.uint64))
