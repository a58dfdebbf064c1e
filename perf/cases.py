"""The work that is timed: calls of the library's public entry points at the sizes of the named
configurations (ttdft_public_gb300/system.py, tests/, bench.py).

Every case is one layer of a Kohn-Sham self-consistent-field iteration -- the Chebyshev filter, the
orthonormalisation, Rayleigh-Ritz, the density, the Hartree term, the Tucker compression, the new
Hamiltonian values, the pointwise grid work -- or one whole pass of the subspace iteration, called as
ttdft_public_gb300/scf.py calls it: operators and blocks stay on the device, and so do the fields.

A Hamiltonian has `rank`^3 basis functions, the 64-atom system's density of atoms and its 0.8 bohr of
box per basis function; the atoms, the block and the fields come from the seed.
"""
import ctypes
import dataclasses
import math

import numpy as np
import torch

from ttdft_public_gb300 import _lib, api, system
from ttdft_public_gb300._lib import check, ptr
from ttdft_public_gb300.kernel_expansion import coulomb_expansion


def listed():
    return [
        # the smallest call: a few FP32 degrees on the 4-atom test system, whose block of 24 states
        # is no multiple of the tensor cores' 16 (latency and launches)
        dict(name="filter_small", kind="filter", rank=12, k=24, degree=8, low="", n_low=0),
        # 64 atoms, 160 states: degrees of the mixed schedule (a BF16 first quarter, FP32 after),
        # the inner loop of every SCF iteration
        dict(name="filter_mixed", kind="filter", rank=40, k=160, degree=8, low="bf16", n_low=2),
        # a block as wide as the 512-atom system's (1,200 states, five column blocks), FP32
        dict(name="filter_wide", kind="filter", rank=32, k=1200, degree=4, low="", n_low=0),
        # the whole plain FP64 pass of the 8-atom configuration (N = 8,000, 16 states, degree 20):
        # filter, Cholesky-QR, Rayleigh-Ritz, rotation
        dict(name="pass_fp64", kind="pass", rank=20, k=16, degree=20),
        # Rayleigh-Ritz of the 64-atom block: H X, X^T H X, the eigensolver, X Q
        dict(name="rayleigh_ritz", kind="rr", rank=40, k=160),
        # Cholesky-QR of the 512-atom block: 512,000 x 1,200 in FP64, the largest dense call
        dict(name="orth_large", kind="orth", n=512000, k=1200),
        # X^T Y (MultTM::mult) of a narrow block of odd width and length
        dict(name="gram_odd", kind="gram", n=9261, k=57),
        # Tucker compression of V_eff at 64 atoms (360 points a direction, rank 72) and back
        dict(name="tucker", kind="tucker", n0=360, n1=360, n2=360, rank=72, eps=0.0),
        # the Hartree potential of the 64-atom density, all 35 expansion terms
        dict(name="hartree", kind="hartree", rank=60, elements=120, terms=35),
        # the 64-atom density on its 241^3 nodes from 160 states
        dict(name="density", kind="density", rank=40, k=160, elements=120),
        # new values of the 64-atom Hamiltonian for a new V_eff, and one product with them
        dict(name="h_update", kind="update", rank=40, pot_rank=72, k=160),
        # pointwise work of one iteration on 360^3 points: V_eff, exchange-correlation, the energy
        # integrals, the mixing of six densities
        dict(name="grid", kind="grid", n0=360, n1=360, n2=360, history=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["filter", "filter", "filter", "pass", "rr", "orth", "gram", "tucker", "hartree",
                       "density", "update", "grid"])
    if kind == "filter":
        # widths of 16, as the configurations have them, and ragged ones of 4 and 8
        rank = rng.randint(10, 40)
        step = rng.choice([16, 16, 16, 8, 4])
        k = max(step, _log(rng, 8, 1200 if rank <= 32 else 400) // step * step)
        k = k if step == 16 else min(k, 240)
        low = rng.choice(["", "bf16"]) if k % 8 == 0 else ""
        degree = rng.randint(4, 8)
        return dict(kind=kind, rank=rank, k=k, degree=degree, low=low, n_low=degree // 4 if low else 0)
    if kind == "pass":
        return dict(kind=kind, rank=rng.randint(10, 22), k=rng.randint(8, 40), degree=rng.randint(8, 20))
    if kind == "rr":
        rank = rng.randint(12, 40)
        return dict(kind=kind, rank=rank, k=min(_log(rng, 12, 400), rank ** 3 // 8))
    if kind == "orth":
        n = _log(rng, 8000, 512000)
        return dict(kind=kind, n=n, k=_log(rng, 16, 1200 if n > 64000 else 400))
    if kind == "gram":
        return dict(kind=kind, n=_log(rng, 1000, 200000), k=_log(rng, 12, 300))
    if kind == "tucker":
        dims = [_log(rng, 40, 360) for _ in range(3)]
        return dict(kind=kind, n0=dims[0], n1=dims[1], n2=dims[2], rank=max(6, min(min(dims) // 4, 80)),
                    eps=rng.choice([0.0, 1e-4]))
    if kind == "hartree":
        return dict(kind=kind, rank=rng.randint(12, 60), elements=_log(rng, 20, 120), terms=35)
    if kind == "density":
        rank = rng.randint(10, 40)
        return dict(kind=kind, rank=rank, k=_log(rng, 8, 160), elements=rng.randint(rank, 3 * rank))
    if kind == "update":
        return dict(kind=kind, rank=rng.randint(12, 40), pot_rank=rng.randint(12, 72),
                    k=rng.choice([16, 24, 48, 160]))
    dims = [_log(rng, 40, 360) for _ in range(3)]
    return dict(kind=kind, n0=dims[0], n1=dims[1], n2=dims[2], history=rng.randint(2, 6))


# ---------------------------------------------------------------- inputs

def _p(t):
    return ctypes.c_void_p(t.data_ptr())


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(seed, *shape):
    return torch.randn(*shape, dtype=torch.float64, device="cuda", generator=_gen(seed))


def _spec(rank, seed, elements=None):
    """The 64-atom configuration cut to `rank` basis functions a direction."""
    box = 0.8 * rank
    atoms = max(1, round(64 * (rank / 40) ** 3))
    return dataclasses.replace(system.CONFIGS["atoms64"], name="r%d" % rank, n_atoms=atoms, box=box,
                               n_el=elements or 3 * rank, rank=rank, seed=seed, min_sep=2.5, margin=2.0)


def _operator(s, k):
    return api.Operator(api.ProjectHamiltonianSparse.from_system(s), max(k, 8))


def _plain_operator(n, k, ranks=None):
    """A unit Hamiltonian, for calls that use an operator's stream and workspaces only."""
    H = system.Csr(n, n, np.arange(n + 1, dtype=np.int64), np.arange(n, dtype=np.int32), np.ones(n))
    return api.Operator(api.ProjectHamiltonianSparse(H, ranks=ranks), max(k, 8))


def _block(op, k, columns):
    """A device block from its states, one contiguous row of `columns` each."""
    X = api.Mat(op, k)
    check(_lib.ttg().ttg_block_set_device(X.h, _p(columns), op.n), "ttg_block_set_device")
    return X


def _columns(X, out):
    check(_lib.ttg().ttg_block_get_device(X.h, _p(out), X.op.n), "ttg_block_get_device")
    return out


def _orbitals(atoms, box, rank, k, seed):
    """k orthonormal states such as a converged block holds: Gaussians of s and p shape around the
    atoms, with a small rough part (k x N, a state a row)."""
    x = torch.arange(rank, dtype=torch.float64, device="cuda") * (box / rank) + 0.5 * box / rank
    R, rows = torch.from_numpy(atoms).cuda(), []
    for i in range(k):
        a, shape, width = i % len(atoms), (i // len(atoms)) % 4, 1.2 + 0.4 * (i // (4 * len(atoms)))
        f = [torch.exp(-(x - R[a, d]) ** 2 / (2 * width ** 2)) for d in range(3)]
        if shape:
            f[shape - 1] = f[shape - 1] * (x - R[a, shape - 1])
        rows.append((f[2][:, None, None] * f[1][None, :, None] * f[0][None, None, :]).reshape(-1))
    Y = torch.stack(rows)
    Y = Y / Y.norm(dim=1, keepdim=True)
    Y = Y + 0.05 * _randn(seed, k, rank ** 3) / math.sqrt(rank ** 3)
    S = Y @ Y.T
    return torch.linalg.solve_triangular(torch.linalg.cholesky(S), Y, upper=False).contiguous()


def _filter_bounds(s):
    """The interval a filter call is given: [0, upper] unwanted, the lowest state below it."""
    return 0.0, 36.0, -0.6


def _schedule(c):
    return api.sched("fp32", low=c["low"] or None, n_low=c["n_low"])


def _grid_fields(dims, seed, box):
    """A density of Gaussian atoms and a local potential on dims points (x fastest: z, y, x)."""
    rng = np.random.default_rng(seed)
    atoms = max(2, min(64, round(64 * np.prod(dims) / 360.0 ** 3)))
    R = rng.uniform(0.1, 0.9, (atoms, 3)) * box
    g, w = [], []
    for d in range(3):
        x = (np.arange(dims[d]) + 0.5) * box / dims[d]
        g.append(_dev(np.exp(-(x[None] - R[:, d][:, None]) ** 2)))
        w.append(_dev(np.exp(-(x[None] - R[:, d][:, None]) ** 2 / (2 * 0.6 ** 2))))
    z = _dev(rng.uniform(0.8, 1.2, atoms) * 3.0)
    rho = torch.einsum("az,ayx->zyx", z[:, None] * g[2] / math.pi ** 1.5, g[1][:, :, None] * g[0][:, None, :])
    v = -torch.einsum("az,ayx->zyx", z[:, None] * w[2], w[1][:, :, None] * w[0][:, None, :])
    return rho.contiguous(), v.contiguous()


class _Stream:
    """A stream of the caller's own for the grid calls, as the SCF driver has its operator's."""

    def __init__(self):
        self.stream = torch.cuda.Stream()
        self.h = ctypes.c_void_p(self.stream.cuda_stream)


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = {"case": c}
    if kind in ("filter", "pass", "rr", "update"):
        s = system.build_system(_spec(c["rank"], seed))
        k = c["k"]
        op = st["op"] = _operator(s, k)
        if kind == "update":
            _prepare_update(st, s, seed)
            return st
        if kind == "rr":
            cols = _orbitals(s.atoms, s.spec.box, c["rank"], k, seed)
        else:
            cols = _randn(seed, k, s.N)
        st["X0"], st["X"] = _block(op, k, cols), api.Mat(op, k)
        st["out"] = torch.empty(k, s.N, dtype=torch.float64, device="cuda")
        st["bounds"] = _filter_bounds(s)
        st["ax"] = api.AX(1, k)
        st["ax"].op = op
        op.sync()
    elif kind in ("orth", "gram"):
        n, k = c["n"], c["k"]
        op = st["op"] = _plain_operator(n, k)
        cols = _filtered_columns(n, k, seed)
        st["X0"] = _block(op, k, cols)
        if kind == "orth":
            st["X"], st["out"] = api.Mat(op, k), cols      # the upload has been read: see sync below
        else:
            st["Y"] = _block(op, k, _filtered_columns(n, k, seed + 7919))
        op.sync()
    elif kind == "tucker":
        dims = [c["n0"], c["n1"], c["n2"]]
        st["op"] = _plain_operator(64, 8)
        st["field"] = _veff(dims, seed).reshape(-1)
        st["dims"] = np.array(dims, np.int32)
        caps = st["caps"] = np.array([min(c["rank"], d) for d in dims], np.int32)
        st["core"] = torch.zeros(int(np.prod(caps)), dtype=torch.float64, device="cuda")
        st["U"] = [torch.zeros(dims[d] * int(caps[d]), dtype=torch.float64, device="cuda") for d in range(3)]
        st["out"] = torch.empty(int(np.prod(dims)), dtype=torch.float64, device="cuda")
    elif kind == "hartree":
        st["op"] = _plain_operator(64, 8)
        alpha, omega, G, quad, U, grids = _hartree_inputs(c, seed)
        st["n"] = np.array([g.size for g in grids], np.int32)
        st["r"] = np.array(G.shape[::-1], np.int32)
        st["alpha"], st["omega"], st["G"] = _dev(alpha), _dev(omega), _dev(G)
        st["xq"] = [_dev(q[0]) for q in quad]
        st["wq"] = [_dev(q[1]) for q in quad]
        st["U"] = [_dev(u.T) for u in U]
        st["out"] = torch.empty(int(np.prod(st["n"].astype(np.int64))), dtype=torch.float64, device="cuda")
    elif kind == "density":
        rank, k = c["rank"], c["k"]
        spec = _spec(rank, seed, c["elements"])
        op = st["op"] = _plain_operator(rank ** 3, k, (rank, rank, rank))
        atoms = np.random.default_rng(seed).uniform(0.1, 0.9, (spec.n_atoms, 3)) * spec.box
        st["X"] = _block(op, k, _orbitals(atoms, spec.box, rank, k, seed))
        U = system.make_basis_1d(system.Fem1D(spec.n_el, 0.0, spec.box), rank).nodal
        st["U"] = _dev(U.T)
        st["r"], st["n"] = np.array([rank] * 3, np.int32), np.array([U.shape[0]] * 3, np.int32)
        st["occ"] = _occupations(k)
        st["out"] = torch.empty(U.shape[0] ** 3, dtype=torch.float64, device="cuda")
        op.sync()
    else:
        dims = [c["n0"], c["n1"], c["n2"]]
        st["dims"], box = np.array(dims, np.int32), 32.0 * max(dims) / 360.0
        st["stream"] = _Stream()
        rho, vloc = _grid_fields(dims, seed, box)
        st["rho"], st["vloc"] = rho.reshape(-1), vloc.reshape(-1)
        st["vh"] = (rho * 0.7 + 0.3 * rho.mean()).reshape(-1)
        st["w"] = [_dev(np.full(d, box / d)) for d in dims]
        # a history of densities: rho_in and rho_out of earlier iterations
        st["hist"] = [st["rho"]] + [st["rho"] * (1.0 + 0.02 * j) + 1e-6 * j for j in range(1, c["history"])]
        st["coef"] = _mixing(c["history"], seed)
        for name in ("veff", "exc", "mixed"):
            st[name] = torch.empty(rho.numel(), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return st


def _filtered_columns(n, k, seed):
    """A block as the filter leaves it: columns of sizes over three decades, correlated with their
    neighbours."""
    Y = _randn(seed, k, n)
    Y[1:] += 0.3 * Y[:-1].clone()
    order = torch.randperm(k, device="cuda", generator=_gen(seed + 1))
    Y *= torch.logspace(0, -3, k, dtype=torch.float64, device="cuda")[order][:, None]
    return Y


def _occupations(k):
    return 1.0 / (1.0 + np.exp((np.arange(k) - 0.6 * k) / max(1.0, 0.03 * k)))


def _veff(dims, seed):
    rho, v = _grid_fields(dims, seed, 32.0 * max(dims) / 360.0)
    return (v - 0.9 * rho ** (1.0 / 3.0)).contiguous()


def _mixing(h, seed):
    return np.random.default_rng(seed).uniform(0.1, 0.9, h) / h


def _hartree_inputs(c, seed):
    a, o, G, quad, U, grids = system.hartree_blob_case(rank=c["rank"], seed=seed, n_el=c["elements"],
                                                       box=32.0)
    a, o = coulomb_expansion()
    return a[: c["terms"]], o[: c["terms"]], G, quad, U, grids


def _potential(c, s, seed):
    """V_eff in Tucker form: smooth factors at the quadrature points with a decaying core; the
    potential matrices of scf.potential_matrices, (ranks, r, r) a direction."""
    rng, m = np.random.default_rng(seed), c["pot_rank"]
    decay = np.exp(-0.12 * np.arange(m))
    G = rng.standard_normal((m, m, m)) * decay[:, None, None] * decay[None, :, None] * decay[None, None, :]
    P = []
    for d in range(3):
        b = s.basis[d]
        x = (b.fem.xq - b.fem.x0) / (b.fem.x1 - b.fem.x0)
        U = np.cos(np.pi * np.outer(x, np.arange(m)) + 0.3 * d)
        M = _dev((b.quad * b.fem.wJ[:, None])[:, :, None] * b.quad[:, None, :]).reshape(b.fem.nq, -1)
        P.append((_dev(U).T @ M).contiguous())
    return _dev(G), P


def _prepare_update(st, s, seed):
    c, op = st["case"], st["op"]
    mats = [np.ascontiguousarray(b.stiffness()) for b in s.basis]
    mats += [np.ascontiguousarray(b.overlap()) for b in s.basis]
    check(_lib.ttg().ttg_op_set_kinetic(op.h, *[ptr(m) for m in mats]), "ttg_op_set_kinetic")
    st["G"], st["P"] = _potential(c, s, seed)
    st["ranks"] = np.array([c["pot_rank"]] * 3, np.int32)
    # an SCF's operator has done a Rayleigh-Ritz step before its values change
    w = _block(op, c["k"], _randn(seed, c["k"], s.N))
    api.rayleigh_ritz(op, w, rotate=False)
    w.close()
    st["x"], st["y"] = _block(op, 1, _randn(seed + 1, 1, s.N)), api.Mat(op, 1)
    st["out"] = torch.empty(1, s.N, dtype=torch.float64, device="cuda")
    st["ax"] = api.AX(1, 1)
    st["ax"].op = op
    op.sync()


# ---------------------------------------------------------------- one pass

def run(st):
    c, lib = st["case"], _lib.ttg()
    kind = c["kind"]
    if kind == "filter":
        check(lib.ttg_block_copy(st["X"].h, st["X0"].h), "ttg_block_copy")
        a, b, a0 = st["bounds"]
        api.ChebyShevFilter(_schedule(c)).computeFilteredSubspace(None, st["ax"], st["X"], st["op"].n,
                                                                  c["degree"], a, b, a0)
        # the last degrees run in FP32: the block holds FP32 values
        return _columns(st["X"], st["out"]).to(torch.float32)
    if kind == "pass":
        check(lib.ttg_block_copy(st["X"].h, st["X0"].h), "ttg_block_copy")
        a, b, a0 = st["bounds"]
        w = api.chfsi_pass(st["op"], st["X"], c["degree"], a, b, a0, api.sched("fp64"), rotate=True)
        return {"w": w, "x": _columns(st["X"], st["out"])}
    if kind == "rr":
        check(lib.ttg_block_copy(st["X"].h, st["X0"].h), "ttg_block_copy")
        w = api.rayleigh_ritz(st["op"], st["X"], rotate=True)
        return {"w": w, "x": _columns(st["X"], st["out"])}
    if kind == "orth":
        check(lib.ttg_block_copy(st["X"].h, st["X0"].h), "ttg_block_copy")
        api.MultTM().orth(st["X"])
        return _columns(st["X"], st["out"])
    if kind == "gram":
        return api.MultTM().mult(st["X0"], st["Y"])
    if kind == "tucker":
        op, ranks = st["op"], np.zeros(3, np.int32)
        check(lib.ttg_tucker_sthosvd(op.h, _p(st["field"]), ptr(st["dims"]), c["eps"], ptr(st["caps"]),
                                     ptr(ranks), _p(st["core"]), *[_p(u) for u in st["U"]]),
              "ttg_tucker_sthosvd")
        check(lib.ttg_tucker_reconstruct(_p(st["core"]), ptr(ranks), *[_p(u) for u in st["U"]],
                                         ptr(st["dims"]), _p(st["out"]), ctypes.c_void_p(op.stream())),
              "ttg_tucker_reconstruct")
        return {"ranks": ranks, "field": st["out"]}
    if kind == "hartree":
        three = lambda ts: (ctypes.c_void_p * 3)(*[t.data_ptr() for t in ts])  # noqa: E731
        check(lib.ttg_hartree_device(st["op"].h, c["terms"], _p(st["alpha"]), _p(st["omega"]), ptr(st["r"]),
                                     _p(st["G"]), ptr(st["n"]), three(st["xq"]), three(st["wq"]),
                                     three(st["U"]), ptr(st["n"]), three(st["xq"]), _p(st["out"])),
              "ttg_hartree_device")
        return st["out"]
    if kind == "density":
        check(lib.ttg_density_device(st["op"].h, st["X"].h, ptr(st["occ"]), ptr(st["r"]), ptr(st["n"]),
                                     _p(st["U"]), _p(st["U"]), _p(st["U"]), _p(st["out"]), 0),
              "ttg_density_device")
        return st["out"]
    if kind == "update":
        check(lib.ttg_op_update_potential_device(st["op"].h, ptr(st["ranks"]), _p(st["G"]),
                                                 *[_p(p) for p in st["P"]]),
              "ttg_op_update_potential_device")
        st["ax"].perform_ax(st["x"], st["y"])
        return _columns(st["y"], st["out"])
    return _run_grid(st, lib)


def _run_grid(st, lib):
    h, n = st["stream"].h, st["rho"].numel()

    def lincomb(fields, coef, out, take_abs):
        f = (ctypes.c_void_p * len(fields))(*[t.data_ptr() for t in fields])
        k = np.ascontiguousarray(coef, dtype=np.float64)
        check(lib.ttg_grid_lincomb(len(fields), f, ptr(k), n, _p(out), take_abs, h), "ttg_grid_lincomb")

    def integrate(f, g):
        v = ctypes.c_double()
        check(lib.ttg_grid_integrate(_p(f), None if g is None else _p(g), ptr(st["dims"]),
                                     *[_p(w) for w in st["w"]], ctypes.byref(v), h), "ttg_grid_integrate")
        return v.value

    rho, veff, exc = st["rho"], st["veff"], st["exc"]
    lincomb(st["hist"], st["coef"], st["mixed"], 1)
    lincomb([st["vh"], st["vloc"]], [1.0, 1.0], veff, 0)
    check(lib.ttg_grid_lda(_p(rho), n, _p(veff), None, 1, h), "ttg_grid_lda")
    check(lib.ttg_grid_lda(_p(rho), n, None, _p(exc), 0, h), "ttg_grid_lda")
    e = [integrate(exc, None), integrate(rho, veff), integrate(rho, st["vloc"]), integrate(rho, None)]
    return {"mixed": st["mixed"], "veff": veff, "exc": exc, "energies": e}


# ---------------------------------------------------------------- what a pass cannot do without

def _nnz(rank):
    """Nonzeros of such a Hamiltonian with its projectors: about 1,500 a row at 20 functions a
    direction, 1,900 at 40 (the boundary cuts the rest)."""
    n = rank ** 3
    return n * min(n, 2300.0 * max(0.2, 1.0 - 2.6 / rank) ** 3)


def work(case):
    c, kind = case, case["kind"]
    if kind == "filter":
        n, k, z = c["rank"] ** 3, c["k"], _nnz(c["rank"])
        lo, hi = c["n_low"], c["degree"] - c["n_low"]
        return {"bytes": lo * (z * 6 + 3 * n * k * 2) + hi * (z * 8 + 3 * n * k * 4),
                "flops": 2.0 * z * k * c["degree"]}
    if kind == "pass":
        n, k, z = c["rank"] ** 3, c["k"], _nnz(c["rank"])
        return {"bytes": (c["degree"] + 1) * (z * 12 + 3 * n * k * 8) + 6 * n * k * 8,
                "flops": 2.0 * z * k * (c["degree"] + 1) + 8.0 * n * k * k}
    if kind == "rr":
        n, k, z = c["rank"] ** 3, c["k"], _nnz(c["rank"])
        return {"bytes": z * 12 + 6 * n * k * 8, "flops": 2.0 * z * k + 4.0 * n * k * k + 9.0 * k ** 3}
    if kind == "orth":
        n, k = c["n"], c["k"]
        return {"bytes": 3.0 * n * k * 8, "flops": 2.0 * n * k * k}
    if kind == "gram":
        return {"bytes": 2.0 * c["n"] * c["k"] * 8 + c["k"] ** 2 * 8, "flops": 2.0 * c["n"] * c["k"] ** 2}
    if kind == "tucker":
        n, r = [c["n0"], c["n1"], c["n2"]], c["rank"]
        t = n[0] * n[1] * n[2]
        f = t * n[0] + 2.0 * t * r + r * n[1] * n[2] * n[1] + 2.0 * r * n[1] * n[2] * r + r * r * n[2] * n[2]
        return {"bytes": 3.0 * t * 8, "flops": f + 2.0 * t * r}
    if kind == "hartree":
        q, r, t = 3 * c["elements"], c["rank"], c["terms"]
        return {"bytes": 8.0 * (q ** 3 + r ** 3), "flops": 2.0 * t * (q * r ** 3 + q * q * r * r + q ** 3 * r)}
    if kind == "density":
        n, r, k = 2 * c["elements"] + 1, c["rank"], c["k"]
        return {"bytes": 8.0 * (n ** 3 + k * r ** 3), "flops": 2.0 * k * (n * r ** 3 + n * n * r * r + n ** 3 * r)}
    if kind == "update":
        z, m = _nnz(c["rank"]), c["pot_rank"]
        pairs = c["rank"] * min(c["rank"], 25)
        # pattern read, new values in FP64, as FP32 pairs, and in the filter's 16-bit terms; one product
        return {"bytes": z * (4 + 8 + 8 + 6) + z * 12, "flops": 2.0 * pairs * pairs * m * m + 2.0 * z * m}
    n, h = c["n0"] * c["n1"] * c["n2"], c["history"]
    return {"bytes": 8.0 * n * (h + 1 + 2 + 2 + 1 + 5), "flops": 60.0 * n}


# ---------------------------------------------------------------- the same in plain 64 bits

def _dense_csr(M, rows, cols):
    return torch.sparse_csr_tensor(torch.from_numpy(np.asarray(M.row_ptr)).cuda(),
                                   torch.from_numpy(M.col.astype(np.int64)).cuda(),
                                   torch.from_numpy(M.val).cuda(), size=(rows, cols))


def _hamiltonian(s):
    H = _dense_csr(s.H, s.N, s.N)
    C, D = _dense_csr(s.C, s.C.n_rows, s.N).to_dense(), torch.from_numpy(s.D).cuda()[:, None]
    return lambda Y: H @ Y + C.T @ (D * (C @ Y))


def _exact_filter(apply, X, degree, a, b, a0):
    e, mid = (b - a) / 2, (b + a) / 2
    sigma = e / (a0 - mid)
    gamma = 2 / sigma
    Y = (apply(X) - mid * X) * (sigma / e)
    for _ in range(2, degree + 1):
        sigma2 = 1 / (gamma - sigma)
        X, Y = Y, (apply(Y) - mid * Y) * (2 * sigma2 / e) - sigma * sigma2 * X
        sigma = sigma2
    return Y


def _exact_ritz(apply, X):
    """w and X Q; each eigenvector's largest component is positive."""
    w, Q = torch.linalg.eigh(X.T @ apply(X))
    at = Q.abs().argmax(dim=0)
    Q = Q * torch.sign(Q[at, torch.arange(Q.shape[1], device=Q.device)])[None]
    return {"w": w, "x": (X @ Q).T.contiguous()}


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("filter", "pass", "rr"):
        s = system.build_system(_spec(c["rank"], seed))
        apply, k = _hamiltonian(s), c["k"]
        if kind == "rr":
            return _exact_ritz(apply, _orbitals(s.atoms, s.spec.box, c["rank"], k, seed).T.contiguous())
        X = _randn(seed, k, s.N).T.contiguous()
        Y = _exact_filter(apply, X, c["degree"], *_filter_bounds(s))
        if kind == "filter":
            return Y.T.contiguous()
        L = torch.linalg.cholesky(Y.T @ Y)
        return _exact_ritz(apply, torch.linalg.solve_triangular(L, Y.T, upper=False).T.contiguous())
    if kind == "orth":
        Y = _filtered_columns(c["n"], c["k"], seed)
        return torch.linalg.solve_triangular(torch.linalg.cholesky(Y @ Y.T), Y, upper=False)
    if kind == "gram":
        return _filtered_columns(c["n"], c["k"], seed) @ _filtered_columns(c["n"], c["k"], seed + 7919).T
    if kind == "tucker":
        return _exact_tucker(c, seed)
    if kind == "hartree":
        a, o, G, quad, U, grids = _hartree_inputs(c, seed)
        F = []
        for d in range(3):
            x, w, u = _dev(grids[d]), _dev(quad[d][1]), _dev(U[d])
            E = torch.exp(-_dev(a)[:, None, None] * (x[:, None] - _dev(quad[d][0])[None]) ** 2)
            F.append((E * w) @ u)
        g = _dev(G)
        V = torch.zeros([f.shape[1] for f in F[::-1]], dtype=torch.float64, device="cuda")
        for t in range(len(a)):
            p = torch.tensordot(torch.tensordot(g, F[0][t], ([2], [1])), F[1][t], ([1], [1]))
            V += float(o[t]) * torch.tensordot(F[2][t], p, ([1], [0])).permute(0, 2, 1)
        return V.reshape(-1)
    if kind == "density":
        rank, k = c["rank"], c["k"]
        spec = _spec(rank, seed, c["elements"])
        atoms = np.random.default_rng(seed).uniform(0.1, 0.9, (spec.n_atoms, 3)) * spec.box
        X = _orbitals(atoms, spec.box, rank, k, seed).reshape(k, rank, rank, rank)
        U = _dev(system.make_basis_1d(system.Fem1D(spec.n_el, 0.0, spec.box), rank).nodal)
        rho = torch.zeros([U.shape[0]] * 3, dtype=torch.float64, device="cuda")
        for i, f in enumerate(_occupations(k)):
            psi = torch.einsum("cba,xa,yb,zc->zyx", X[i], U, U, U)
            rho += 2.0 * float(f) * psi ** 2
        return rho.reshape(-1)
    if kind == "update":
        return _exact_update(c, seed)
    return _exact_grid(c, seed)


def _exact_tucker(c, seed):
    T = _veff([c["n0"], c["n1"], c["n2"]], seed).permute(2, 1, 0).contiguous()     # x, y, z
    thr, U, ranks = c["eps"] ** 2 * float((T * T).sum()) / 3.0, [], []
    A = T
    for d in range(3):
        M = A.movedim(d, 0).reshape(A.shape[d], -1)
        w, V = torch.linalg.eigh(M @ M.T)
        w, V = w.flip(0), V.flip(1)
        cap = min(c["rank"], A.shape[d])
        kept = torch.cumsum(w[:cap].clamp(min=0), 0)
        r = cap
        if thr > 0:
            ok = (w.sum() - kept <= thr).nonzero()
            r = int(ok[0]) + 1 if len(ok) else cap
        U.append(V[:, :r])
        ranks.append(r)
        A = torch.tensordot(U[d].T, A, ([1], [d])).movedim(0, d)
    for d in range(3):
        A = torch.tensordot(U[d], A, ([1], [d])).movedim(0, d)
    return {"ranks": np.array(ranks, np.int32), "field": A.permute(2, 1, 0).reshape(-1)}


def _exact_update(c, seed):
    s, r = system.build_system(_spec(c["rank"], seed)), c["rank"]
    G, P = _potential(c, s, seed)
    m = c["pot_rank"]
    P = [p.reshape(m, r * r) for p in P]
    K = [(_dev(b.stiffness()), _dev(b.overlap())) for b in s.basis]
    # sum over the x and y ranks once: (yy, xx, c); core as (z, y, x) ranks
    T1 = torch.einsum("cba,ap->cbp", G, P[0])
    T2 = torch.einsum("cbp,bq->qpc", T1, P[1]).reshape(r * r * r * r, m)
    PZ = P[2].T.contiguous()
    x = _randn(seed + 1, 1, s.N)[0]
    y = torch.zeros(s.N, dtype=torch.float64, device="cuda")
    ptr_, col = torch.from_numpy(s.H.row_ptr).cuda(), torch.from_numpy(s.H.col).cuda().long()
    row = torch.repeat_interleave(torch.arange(s.N, device="cuda"), ptr_[1:] - ptr_[:-1])
    for lo in range(0, len(col), 1 << 22):
        I, J = row[lo: lo + (1 << 22)], col[lo: lo + (1 << 22)]
        ij = [(I % r, J % r), (I // r % r, J // r % r), (I // (r * r), J // (r * r))]
        q = [i * r + j for i, j in ij]
        (dx, mx), (dy, my), (dz, mz) = [(K[d][0].reshape(-1)[q[d]], K[d][1].reshape(-1)[q[d]]) for d in range(3)]
        v = 0.5 * (dx * my * mz + mx * dy * mz + mx * my * dz)
        v += (T2[q[1] * (r * r) + q[0]] * PZ[q[2]]).sum(dim=1)
        y.index_add_(0, I, v * x[J])
    C, D = _dense_csr(s.C, s.C.n_rows, s.N).to_dense(), torch.from_numpy(s.D).cuda()
    return (y + C.T @ (D * (C @ x)))[None]


def _exact_grid(c, seed):
    dims = [c["n0"], c["n1"], c["n2"]]
    box = 32.0 * max(dims) / 360.0
    rho, vloc = _grid_fields(dims, seed, box)
    vh = rho * 0.7 + 0.3 * rho.mean()
    hist = [rho] + [rho * (1.0 + 0.02 * j) + 1e-6 * j for j in range(1, c["history"])]
    mixed = sum(float(a) * f for a, f in zip(_mixing(c["history"], seed), hist)).abs()
    # exchange and correlation after Perdew and Zunger, with the constants of the method
    g, b1, b2, A, B, Cc, Dd = -0.1423, 1.0529, 0.3334, 0.0311, -0.048, 0.002, -0.0116
    cx = -(3.0 / 4.0) * (3.0 / math.pi) ** (1.0 / 3.0)
    cr = rho ** (1.0 / 3.0)
    rs = (3.0 / (4.0 * math.pi * rho)) ** (1.0 / 3.0)
    sq, lr = rs.sqrt(), rs.log()
    den = 1.0 + b1 * sq + b2 * rs
    low = g * (1.0 + (7.0 / 6.0) * b1 * sq + (4.0 / 3.0) * b2 * rs) / (den * den)
    high = A * lr + (B - A / 3.0) + (2.0 / 3.0) * Cc * rs * lr + (2.0 * Dd - Cc) * rs / 33.0
    veff = vh + vloc + (4.0 / 3.0) * cx * cr + torch.where(rs >= 1.0, low, high)
    rs = (3.0 / (4.0 * math.pi)) ** (1.0 / 3.0) / (cr + 1e-12)
    lr = rs.log()
    ec = torch.where(rs >= 1.0, g / (1.0 + b1 * rs.sqrt() + b2 * rs), A * lr + B + Cc * rs * lr + Dd * rs)
    exc = cx * rho * cr + ec * rho
    w = np.prod([box / d for d in dims])
    e = [float(f.sum() * w) for f in (exc, rho * veff, rho * vloc, rho)]
    return {"mixed": mixed.reshape(-1), "veff": veff.reshape(-1), "exc": exc.reshape(-1), "energies": e}
