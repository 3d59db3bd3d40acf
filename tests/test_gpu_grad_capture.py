"""Term gradients captured into a CUDA graph without an earlier call, where the
kernels need nothing that is made on the host: complex128, and complex64 below
12 qubits."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n", [("complex128", 13), ("complex128", 6), ("complex64", 11)])
def test_first_call_inside_a_capture(cuda, dtype, n):
    import torch
    t = W.cfg2(n=n, npair=120, nz=60)  # x = 0 has many strings
    psi = W.random_state(np.random.default_rng(1), 1 << n, nstates=2)
    g = W.random_state(np.random.default_rng(2), 1 << n, nstates=2)
    p = torch.from_numpy(psi).to(cuda, getattr(torch, dtype))
    gg = torch.from_numpy(g).to(cuda, getattr(torch, dtype))
    op = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = op.term_grad(p, gg)
    graph.replay()
    op.sync_check()
    want = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff).term_grad(p, gg)
    # two unit-norm states: the products' moduli add to at most 1 each, and a
    # sum in any order is off by at most 2^n roundings of that, so two sums by 4
    # times 2^n; below 12 qubits complex64 takes the same sums in the same order
    tol = 4.0 * (1 << n) * 2.0 ** -53 if dtype == "complex128" else 0.0
    assert float((out - want).abs().max()) <= tol
