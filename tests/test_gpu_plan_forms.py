"""complex64 products of one operator over calls of few and of many states: the
number of states picks the kernel, but the operator's coefficients and what may
be captured into a CUDA graph do not depend on it."""
import numpy as np
import pytest

from qrusty_gb300 import PauliOperator
from qrusty_gb300 import workloads as W

pytestmark = pytest.mark.gpu

# few states run over rows, many over tiles (cosets, strings, per-tile tables)
CASES = {
    "cosets": lambda: W.cfg2(n=14, npair=300, nz=100),
    "strings": lambda: W.random_letters_op(np.random.default_rng(1), 12, 200),
    "tables": lambda: W.random_letters_op(np.random.default_rng(2), 10, 150),
}


def _setup(cuda, name):
    import torch
    t = CASES[name]()
    op = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff)
    few = torch.from_numpy(W.random_state(np.random.default_rng(3), 1 << t.n)
                           .astype(np.complex64)).to(cuda)
    states = {14: 16, 12: 40, 10: 80}[t.n]
    many = torch.from_numpy(W.random_state(np.random.default_rng(4), 1 << t.n, nstates=states)
                            .astype(np.complex64)).to(cuda)
    return t, op, few, many


@pytest.mark.parametrize("adjoint", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_replayed_update_reaches_every_call(cuda, name, adjoint):
    """A graph that updates the coefficients, captured when only calls of few
    states had been made, serves a call of many states made outside it."""
    import torch
    t, op, few, many = _setup(cuda, name)
    c = torch.from_numpy(t.coeff.copy()).to(cuda)
    out = torch.empty_like(few)

    def step():
        op.set_coeffs_device(c)
        op.apply(few, out=out, adjoint=adjoint)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    op.apply(many, adjoint=adjoint)  # with today's coefficients
    c1 = np.random.default_rng(5).standard_normal(t.T) + 0.5j
    c.copy_(torch.from_numpy(c1).to(cuda))
    graph.replay()
    got = op.apply(many, adjoint=adjoint)
    op.sync_check()
    want = PauliOperator(t.n, t.x, t.z, t.phase, c1).apply(many, adjoint=adjoint)
    assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))


@pytest.mark.parametrize("warm,call", [("few", "many"), ("many", "few")])
@pytest.mark.parametrize("name", sorted(CASES))
def test_capture_after_a_call_of_another_size(cuda, name, warm, call):
    import torch
    t, op, few, many = _setup(cuda, name)
    psi = {"few": few, "many": many}
    op.apply(psi[warm])
    out = torch.empty_like(psi[call])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        op.apply(psi[call], out=out)
    graph.replay()
    op.sync_check()
    want = PauliOperator(t.n, t.x, t.z, t.phase, t.coeff).apply(psi[call])
    assert torch.equal(torch.view_as_real(out), torch.view_as_real(want))


# about one string per x group: the string kernel above 2^14 rows (2^23 over the
# groups where they are few), whatever the few groups of several strings and those
# on the diagonal
@pytest.mark.parametrize("n,strings,diagonal", [(12, 400, 0), (12, 1000, 0), (12, 2000, 0),
                                                (13, 2000, 0), (14, 2000, 0), (14, 900, 600)])
def test_string_operators_leave_the_rows_kernel(cuda, oracle, n, strings, diagonal):
    import torch
    rng = np.random.default_rng(strings)
    t = W.random_letters_op(rng, n, strings)
    if diagonal:
        x, z = t.x.copy(), t.z.copy()
        x[:diagonal], z[:diagonal] = 0, rng.choice(1 << n, diagonal, replace=False)
        t = W.Terms(n, x, z, np.zeros(strings, np.uint8), t.coeff)
    op = PauliOperator(n, t.x, t.z, t.phase, t.coeff)
    states = 1 << (15 - n)
    assert op.apply_form(torch.complex64, states) == "strings"
    assert op.apply_form(torch.complex64, states // 2) == "rows"
    psi = W.random_state(rng, 1 << n, nstates=2)[:1].astype(np.complex64)
    p = torch.from_numpy(np.repeat(psi, states, axis=0)).to(cuda)
    y = op.apply(p).cpu().numpy()
    op.sync_check()
    ref = oracle.apply(n, t.x, t.z, oracle.make_params(t.phase, t.coeff),
                       psi[0].astype(np.complex128))
    for s in range(states):
        assert np.linalg.norm(y[s] - ref) <= 1e-6 * np.linalg.norm(ref)
