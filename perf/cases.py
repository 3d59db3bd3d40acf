"""The work a user of this package has it do, as measurable cases.

A case is a dict of plain values; ``prepare`` makes what a program holds
before the call (terms, states, the operator handle), ``run`` is one pass
through the public entry points, ``work`` what that pass cannot do without
and ``exact`` its result in 64 bits by plain torch / numpy.

Operators come in the three families the package's own workloads use:

* ``random``: letters i.i.d. I X Y Z with P = (0.55, 0.15, 0.15, 0.15) and
  N(0, 1) coefficients -- almost every term has an x mask of its own;
* ``chain``: the open TFIM + XXZ spin chain, 4 n - 3 terms;
* ``jw``: Jordan-Wigner pair terms (X or Y at i and j, Z between; four
  fifths of the terms) and products of 1-4 Z, N(0, 0.1) coefficients.
"""
import math

import numpy as np
import torch

import qrusty_gb300 as Q
from qrusty_gb300 import _lib
from qrusty_gb300.autograd import PauliTerms, pauli_apply

_DTYPE = {"c64": torch.complex64, "c128": torch.complex128}
_LR = 1e-3     # step of the training cases' coefficient update
_TOL = 1e-14   # regularisation of the preconditioner


def listed():
    return [
        # one small product: an operator of a few hundred strings on 12 qubits,
        # called once per iteration of a classical loop (latency, few blocks)
        dict(name="apply_c128_random_n12", kind="apply", family="random", n=12, terms=200,
             dtype="c128", states=1, adjoint=False),
        # a mid-sized random-letter operator on a few states at once
        dict(name="apply_c64_random_n16", kind="apply", family="random", n=16, terms=1000,
             dtype="c64", states=3, adjoint=False),
        # spin-chain products of a time evolution or Lanczos loop, both precisions
        dict(name="apply_c64_chain_n22", kind="apply", family="chain", n=22, terms=85,
             dtype="c64", states=1, adjoint=False),
        dict(name="apply_c128_chain_n22", kind="apply", family="chain", n=22, terms=85,
             dtype="c128", states=1, adjoint=False),
        # a large molecule-like Hamiltonian on one 2^26 state
        dict(name="apply_c64_jw_n26", kind="apply", family="jw", n=26, terms=10000,
             dtype="c64", states=1, adjoint=False),
        # the adjoint product of a molecule-like operator in full precision
        dict(name="apply_c128_jw_n18", kind="apply", family="jw", n=18, terms=2000,
             dtype="c128", states=3, adjoint=True),
        # many operators of uneven size on a few states each, one call
        dict(name="batch_c64_n10_18", kind="batch", ops=24, nmin=10, nmax=18, tmin=50,
             tmax=2000, states=4),
        # a variational step: product, gradients to state and coefficients, update
        dict(name="train_c64_n20", kind="train", family="random", n=20, terms=2000, dtype="c64"),
        dict(name="train_c128_n15", kind="train", family="jw", n=15, terms=500, dtype="c128"),
        # the matrix itself, left on the device
        dict(name="csr_chain_n21", kind="csr", family="chain", n=21, terms=81),
        # one step of an eigensolver on that matrix: product, residual, preconditioner
        dict(name="eigen_chain_n20", kind="eigen", family="chain", n=20, terms=77),
        # labels to a host matrix, as a small script does it
        dict(name="matrix_random_n10", kind="matrix", family="random", n=10, terms=200),
    ]


def _log(rng, lo, hi):
    """A whole number in [lo, hi], even over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _groups_bound(family, n, terms):
    """About how many distinct x masks an operator of this family has."""
    if family == "chain":
        return 2 * n
    return min(terms, n * (n - 1) // 2 + 1) if family == "jw" else terms


def draw(rng):
    kind = rng.choice(["apply"] * 6 + ["train"] * 2 + ["batch", "csr", "eigen", "matrix"])
    family = rng.choice(["random", "chain", "jw"])
    if kind == "batch":
        nmin = rng.randint(8, 12)
        return dict(kind=kind, ops=rng.randint(4, 24), nmin=nmin, nmax=rng.randint(nmin, 18),
                    tmin=rng.randint(20, 50), tmax=_log(rng, 60, 2000), states=rng.randint(1, 4))
    dtype = rng.choice(["c64", "c128"])
    # (row, x group) products allowed: never more than the largest listed case
    # of the kind, FP64 arithmetic and stored matrices a good deal less
    most = {"apply": 1e10 if dtype == "c64" else 2.5e8, "train": 2e9 if dtype == "c64" else 1e7,
            "csr": 8e7, "eigen": 4e7, "matrix": 4e5}[kind]
    lo, hi = {"apply": (8, 25), "train": (9, 20), "csr": (8, 21), "eigen": (8, 20),
              "matrix": (3, 12)}[kind]
    states = rng.choice([1, 1, 1, 2, 3, 5, 8]) if kind == "apply" else 1
    while True:
        n = rng.randint(lo, hi)
        terms = 4 * n - 3 if family == "chain" else _log(
            rng, 20, 10000 if family == "jw" and kind == "apply" else 2000)
        if _groups_bound(family, n, terms) * states * 2.0 ** n <= most:
            break
    c = dict(kind=kind, family=family, n=n, terms=terms)
    if kind in ("apply", "train"):
        c["dtype"] = dtype
    if kind == "apply":
        c["states"] = states
        c["adjoint"] = rng.random() < 0.25
    return c


# ------------------------------------------------------------------ inputs
def _terms(family, n, count, rng):
    """(x, z, phase, coeff) arrays: x, z masks with qubit 0 as bit 0, phase the
    number of Y letters mod 4, real coefficients as complex128."""
    one = np.int64(1)
    if family == "random":
        letters = rng.choice(4, size=(count, n), p=(0.55, 0.15, 0.15, 0.15))  # I X Y Z
        w = one << np.arange(n, dtype=np.int64)
        x = (((letters == 1) | (letters == 2)) * w).sum(axis=1)
        z = (((letters == 2) | (letters == 3)) * w).sum(axis=1)
        y = (letters == 2).sum(axis=1)
        c = rng.standard_normal(count)
    elif family == "chain":
        bond = (3 * one) << np.arange(n - 1, dtype=np.int64)
        site = one << np.arange(n, dtype=np.int64)
        none = np.zeros_like(bond)
        x = np.concatenate([none, bond, bond, site])
        z = np.concatenate([bond, none, bond, np.zeros_like(site)])
        y = np.concatenate([none, none, none + 2, np.zeros_like(site)])
        c = np.concatenate([rng.uniform(0.5, 1.5, 3 * (n - 1)), rng.uniform(0.0, 2.0, n)])
    else:
        pairs = count - count // 5
        i = rng.integers(0, n, pairs)
        j = (i + rng.integers(1, n, pairs)) % n
        i, j = np.minimum(i, j), np.maximum(i, j)
        a, b = rng.integers(0, 2, pairs), rng.integers(0, 2, pairs)  # X or Y at i, j
        x = (one << i) | (one << j)
        z = ((one << j) - (one << (i + 1))) | (a << i) | (b << j)
        zz = np.zeros(count - pairs, dtype=np.int64)
        for k in range(count - pairs):
            q = rng.choice(n, int(rng.integers(1, min(4, n) + 1)), replace=False)
            zz[k] = (one << q).sum()
        x = np.concatenate([x, np.zeros_like(zz)])
        z = np.concatenate([z, zz])
        y = np.concatenate([a + b, np.zeros_like(zz)])
        c = rng.normal(0.0, 0.1, count)
    return (x.astype(np.uint64), z.astype(np.uint64), (y % 4).astype(np.uint8),
            c.astype(np.complex128))


def _states(n, states, dtype, seed):
    """Unit-norm Gaussian states on the GPU, (states, 2^n), or (2^n,) for one."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    v = torch.randn(states, 1 << n, 2, generator=g, device="cuda", dtype=real)
    v /= torch.linalg.vector_norm(v, dim=(1, 2), keepdim=True)
    v = torch.view_as_complex(v)
    return v[0] if states == 1 else v


def _labels(n, x, z):
    return ["".join("IXZY"[((xk >> q) & 1) + 2 * ((zk >> q) & 1)] for q in reversed(range(n)))
            for xk, zk in zip(x.tolist(), z.tolist())]


def _case_terms(case, seed):
    """The case's operator.  Where the size of the result depends on the x
    masks (a matrix), the strings belong to the case and the seed gives the
    coefficients; elsewhere all of it comes from the seed."""
    masks = 20260 if case["kind"] in ("csr", "matrix") else seed
    x, z, phase, c = _terms(case["family"], case["n"], case["terms"],
                            np.random.default_rng(masks))
    if masks != seed:
        c = np.random.default_rng(seed).standard_normal(len(c)).astype(np.complex128)
    return x, z, phase, c


def _batch_terms(case, seed):
    """(n, terms) per operator: sizes from the case, strings from the seed."""
    size, rng = np.random.default_rng(case["ops"]), np.random.default_rng(seed)
    out = []
    for _ in range(case["ops"]):
        n = int(size.integers(case["nmin"], case["nmax"] + 1))
        count = int(size.integers(case["tmin"], case["tmax"] + 1))
        out.append((n, _terms("random", n, count, rng)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        terms = _batch_terms(case, seed)
        ops = [Q.PauliOperator(n, *t) for n, t in terms]
        psis = [_states(n, case["states"], torch.complex64, 1000 * seed + k)
                for k, (n, _) in enumerate(terms)]
        return dict(kind=kind, batch=Q.Batch(ops, [case["states"]] * len(ops)), psis=psis,
                    ys=[torch.empty_like(p) for p in psis])
    n = case["n"]
    x, z, phase, coeff = _case_terms(case, seed)
    if kind == "matrix":
        return dict(kind=kind, labels=_labels(n, x, z), coeffs=[complex(c) for c in coeff])
    if kind == "train":
        dt = _DTYPE[case["dtype"]]
        return dict(kind=kind, terms=PauliTerms(n, x, z, phase),
                    c=torch.from_numpy(coeff.real.copy()).cuda().requires_grad_(True),
                    psi=_states(n, 1, dt, seed).requires_grad_(True),
                    w=_states(n, 1, dt, seed + 500000))
    op = Q.PauliOperator(n, x, z, phase, coeff)
    s = dict(kind=kind, op=op)
    if kind == "apply":
        s["psi"] = _states(n, case["states"], _DTYPE[case["dtype"]], seed)
        s["adjoint"] = case["adjoint"]
    elif kind == "eigen":
        s["csr"] = op.csr_device()
        s["diag"] = op.diagonal()
        s["x"] = _states(n, 1, torch.complex128, seed)
        s["theta"] = -float(np.abs(coeff).sum())  # below the spectrum
    return s


def run(s):
    kind = s["kind"]
    if kind == "apply":
        return s["op"].apply(s["psi"], adjoint=s["adjoint"])
    if kind == "batch":
        return s["batch"].apply(s["psis"], s["ys"])
    if kind == "train":
        c, psi = s["c"], s["psi"]
        c.grad = psi.grad = None
        y = pauli_apply(c, psi, s["terms"])
        torch.vdot(y, s["w"]).real.backward()
        with torch.no_grad():
            c.sub_(c.grad, alpha=_LR)
        return dict(y=y, c=c, grad_c=c.grad, grad_psi=psi.grad)
    if kind == "csr":
        indptr, indices, data = s["op"].csr_device()
        return dict(indptr=indptr, indices=indices, data=data)
    if kind == "eigen":
        indptr, indices, data = s["csr"]
        x = s["x"]
        y = torch.empty_like(x)
        _lib.check(_lib.load().qr_csr_spmv(
            y.numel(), x.numel(), indptr.data_ptr(), indices.data_ptr(), data.data_ptr(),
            x.data_ptr(), y.data_ptr(), torch.cuda.current_stream().cuda_stream))
        r = Q.axpby(1.0, y, -s["theta"], x)
        return dict(r=r, t=Q.precond2(s["diag"], r, s["theta"], _TOL))
    m = Q.SparsePauliOp.from_labels(s["labels"], s["coeffs"])
    _, data, indices, indptr = m.to_matrix_mode("RowwiseUnsafeChunked/1000").export()
    return dict(indptr=indptr, indices=indices, data=data)


# ------------------------------------------------------------------ work
def _group_flops(x, z):
    """(x groups, FP operations per row): a complex multiply-add per group, of
    4 operations where the group's factor is real or imaginary throughout."""
    groups = {}
    for xk, zk in zip(x.tolist(), z.tolist()):
        groups.setdefault(xk, set()).add(bin(xk & zk).count("1") & 1)
    return len(groups), sum(4 if len(k) == 1 else 8 for k in groups.values())


def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = {"bytes": 0.0, "flops": 0.0}
        for n, (x, z, _, _) in _batch_terms(case, 0):
            w["bytes"] += 16.0 * case["states"] * 2.0 ** n + 33 * len(x)
            w["flops"] += _group_flops(x, z)[1] * 2.0 ** n * case["states"]
        return w
    n, N = case["n"], 2.0 ** case["n"]
    x, z, _, _ = _case_terms(case, 0)
    groups, per_row = _group_flops(x, z)
    nnz, table = groups * N, 33.0 * len(x)
    if kind == "apply":
        amp = 16.0 if case["dtype"] == "c128" else 8.0
        return {"bytes": 2 * amp * N * case["states"] + table,
                "flops": per_row * N * case["states"]}
    if kind == "train":
        # psi, w read, y, grad_psi written; two products, then per x group the
        # products conj(psi) w and one signed sum per string
        amp = 16.0 if case["dtype"] == "c128" else 8.0
        return {"bytes": 4 * amp * N + 3 * table, "flops": 2 * per_row * N + 8 * nnz
                + 2 * len(x) * N}
    if kind == "eigen":
        return {"bytes": 24 * nnz + 8 * N + 64 * N, "flops": per_row * N + 20 * N}
    return {"bytes": 24 * nnz + 8 * N + table, "flops": 0.0}


# ------------------------------------------------------------------ exact
class _Reference:
    """sum_k c_k P_k in 64 bits, one x group at a time: a row's factor in the
    group is a sum of signs (-1)^popc(r & z), each the product of a sign of
    the row's high bits and one of its low bits, hence one matrix product."""

    def __init__(self, n, x, z, phase, coeff):
        self.n, self.lo = n, n // 2
        self.hi = n - self.lo
        self.x, self.z = x.astype(np.int64), z.astype(np.int64)
        # (-i)^phase c, the factor of X^x Z^z in a row's entry
        unit = np.array([1, -1j, -1, 1j])[phase]
        self.unit, self.c = unit, unit * coeff
        self.groups = [(int(g), np.flatnonzero(self.x == g)) for g in np.unique(self.x)]
        self.rows = torch.arange(1 << n, device="cuda")

    def signs(self, masks, bits):
        """(count, 2^bits) matrix of (-1)^popc(r & mask)."""
        s = torch.ones(len(masks), 1, dtype=torch.float64, device="cuda")
        for q in range(bits):
            bit = torch.from_numpy(1.0 - 2.0 * ((masks >> q) & 1)).to("cuda")[:, None]
            s = torch.cat([s, s * bit], dim=1)
        return s

    def parts(self, members):
        z = self.z[members]
        return self.signs(z >> self.lo, self.hi), self.signs(z & ((1 << self.lo) - 1), self.lo)

    def factor(self, members, c):
        out = torch.zeros(1 << self.n, 2, dtype=torch.float64, device="cuda")
        for at in range(0, len(members), 256):
            k = members[at:at + 256]
            sh, sl = self.parts(k)
            for p, v in ((0, c[k].real), (1, c[k].imag)):
                if np.any(v):
                    w = torch.from_numpy(np.ascontiguousarray(v)).to("cuda")
                    out[:, p] += ((sh * w[:, None]).T @ sl).reshape(-1)
        return torch.view_as_complex(out)

    def apply(self, psi, adjoint=False):
        p = psi.to(torch.complex128).reshape(-1, 1 << self.n)
        y = torch.zeros_like(p)
        for g, members in self.groups:
            d = self.factor(members, self.c)
            if adjoint:  # entry (r, r ^ x) of the adjoint: conj of entry (r ^ x, r)
                d = d[self.rows ^ g].conj()
            y += d * (p if g == 0 else p[:, self.rows ^ g])
        return y.reshape(psi.shape)

    def term_grad(self, psi, w):
        """<P_k psi, w> per term."""
        p, v = psi.to(torch.complex128), w.to(torch.complex128)
        out = np.zeros(len(self.x), dtype=np.complex128)
        for g, members in self.groups:
            h = torch.view_as_real(p[self.rows ^ g].conj() * v)
            for at in range(0, len(members), 256):
                k = members[at:at + 256]
                sh, sl = self.parts(k)
                part = [((sh @ h[:, q].reshape(sh.shape[1], -1)) * sl).sum(dim=1).cpu().numpy()
                        for q in (0, 1)]
                out[k] = np.conj(self.unit[k]) * (part[0] + 1j * part[1])
        return out

    def csr_data(self):
        """Values of the CSR matrix, columns ascending in each row."""
        G = len(self.groups)
        val = torch.empty(1 << self.n, G, dtype=torch.complex128, device="cuda")
        col = torch.empty(1 << self.n, G, dtype=torch.int32, device="cuda")
        for k, (g, members) in enumerate(self.groups):
            val[:, k] = self.factor(members, self.c)
            col[:, k] = self.rows ^ g
        order = torch.argsort(col, dim=1)
        del col
        return torch.gather(torch.view_as_real(val).reshape(-1, G, 2), 1,
                            order[:, :, None].expand(-1, -1, 2)).contiguous()


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [_Reference(n, *t).apply(_states(n, case["states"], torch.complex64,
                                                1000 * seed + k))
                for k, (n, t) in enumerate(_batch_terms(case, seed))]
    n = case["n"]
    x, z, phase, coeff = _case_terms(case, seed)
    ref = _Reference(n, x, z, phase, coeff)
    if kind == "apply":
        return ref.apply(_states(n, case["states"], _DTYPE[case["dtype"]], seed), case["adjoint"])
    if kind == "train":
        dt = _DTYPE[case["dtype"]]
        psi, w = _states(n, 1, dt, seed), _states(n, 1, dt, seed + 500000)
        gc = torch.from_numpy(ref.term_grad(psi, w).real.copy())
        return dict(y=ref.apply(psi), c=torch.from_numpy(coeff.real.copy()) - _LR * gc, grad_c=gc,
                    grad_psi=ref.apply(w, adjoint=True))
    if kind == "eigen":
        v = _states(n, 1, torch.complex128, seed)
        theta = -float(np.abs(coeff).sum())
        r = ref.apply(v) - theta * v
        zero = np.flatnonzero(ref.x == 0)
        d = (ref.factor(zero, ref.c) if len(zero) else torch.zeros_like(v)) - theta
        return dict(r=r, t=r / torch.where(d.abs() < _TOL, torch.full_like(d, _TOL), d))
    data = torch.view_as_complex(ref.csr_data()).reshape(-1)
    return dict(indptr=None, indices=None, data=data if kind == "csr" else data.cpu().numpy())
