"""CSR of one x group (a single Pauli among them), chunks of 512 rows from 18 qubits
on: bit for bit against the oracle, on the device and over the host."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8, 9, 10, 17, 18])
@pytest.mark.parametrize("terms", [1, 3, 40])  # class tables, and folded term by term
def test_one_group(cuda, oracle, n, terms):
    rng = np.random.default_rng(n + terms)
    x = np.full(terms, rng.integers(0, 1 << n), np.uint64)
    z = rng.integers(0, 1 << n, terms).astype(np.uint64)
    phase = rng.integers(0, 4, terms).astype(np.uint8)
    c = rng.standard_normal(terms) + 1j * rng.standard_normal(terms)
    op = PauliOperator(n, x, z, phase, c)
    want = oracle.csr_build(n, x, z, oracle.make_params(phase, c))
    dev = [t.cpu().numpy() for t in op.csr_device()]
    op.sync_check()
    for got in (dev, op.csr_host()):
        for a, b in zip(got, want):
            assert np.array_equal(np.ascontiguousarray(a).view(np.uint64),
                                  np.ascontiguousarray(b).view(np.uint64))
