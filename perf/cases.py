"""Performance cases of the symmetry-reduced Hamiltonian application, through the public `edgpu` API.

Every case is one call (or one short sequence of calls) that a program of this framework makes in
earnest: the product `mul_` as a caller gets it from `represent` alone ("plain") and with the tables
that a solver builds once for many products ("tables"), on device vectors and on host buffers; all
momentum sectors in one batch; the differentiable product with its gradients; a whole Lanczos run;
vectors between the parent and the reduced space; and the enumeration of a sector's basis.  Sizes are
those of the benchmark's configurations and of the tests (chains of 16 to 32 sites, the triangular 6x5
torus) and tori in between.

`exact` restates the same results in plain torch at 64 bits: representatives are orbit minima under
the translations whose stabiliser has trivial character; the row formula of the reduced product is
y_r = sum amp chi(g) sqrt(|O_r| / |O_c|) x_c over the targets q of row r, with g q = c the
representative of q.
"""
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG_DIR = os.path.join(ROOT, "exactdiagonalization.jl_gb300")
if PKG_DIR not in sys.path:
    sys.path.insert(0, PKG_DIR)

SLAB_BYTES = 112 << 20      # column slabs of the benchmark
LANCZOS_STEPS = 100
LOOKUPS = 10000


# ---- the cases -----------------------------------------------------------------------------------
def _case(kind, model, L1, L2=1, q=0, k1=0, k2=0, prec="fp64", tables=False, reduced=True, name=None):
    c = {"kind": kind, "model": model, "L1": L1, "L2": L2, "q": q, "k1": k1, "k2": k2, "prec": prec,
         "tables": tables, "reduced": reduced}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the unreduced 12,870-state sector: the smallest products, where a call's latency counts
        _case("mul", "chain", 16, reduced=False, name="mul_chain16_full_c128"),
        # a product as `represent` alone gives it, on an odd chain, off 2Sz = 0, with complex characters
        _case("mul", "chain", 25, q=1, k1=3, name="mul_chain25_k3_c128"),
        # the 112,720-row sector with a solver's tables, complex64
        _case("mul", "chain", 24, prec="mixed", tables=True, name="mul_chain24_k0_c64_tables"),
        # 1.4 million rows in FP64 with tables
        _case("mul", "chain", 28, tables=True, name="mul_chain28_k0_c128_tables"),
        # one momentum sector of the triangular torus, 5.2 million rows, complex characters
        _case("mul", "triangular", 6, 5, k1=1, prec="mixed", tables=True, name="mul_tri6x5_k1_c64_tables"),
        # 18.8 million rows and 1.2e9 nonzeros: x beyond L2, several column slabs
        _case("mul", "square", 4, 8, prec="mixed", tables=True, name="mul_square4x8_k0_c64_tables"),
        # the drop-in call: ordinary (pageable) complex128 host arrays in and out
        _case("host", "chain", 24, tables=True, name="host_chain24_k0_c128"),
        # all 24 momentum sectors of a torus in one batched call, replayed from a graph
        _case("batch", "triangular", 6, 4, prec="mixed", tables=True, name="batch_tri6x4_allk_c64"),
        # forward and backward of the differentiable product with per-bond couplings
        _case("grad", "coupled", 28, tables=True, name="grad_chain28_c128"),
        # the ground state of the 112,720-row sector: 100 Lanczos steps, full reorthogonalisation
        _case("lanczos", "chain", 24, tables=True, name="lanczos_chain24_k0_c128"),
        # a reduced vector to the 10.4-million-state parent space and back
        _case("vectors", "chain", 26, k1=1, name="vectors_chain26_k1_c128"),
        # the basis of a sector and its representatives, with the tables on the host, and rows of states
        _case("basis", "chain", 26, name="basis_chain26_k0"),
    ]


_TORI = [(3, 3), (4, 3), (4, 4), (5, 4), (6, 3), (6, 4), (5, 5)]


def draw(rng):
    kind = rng.choice(["mul", "mul", "mul", "mul", "host", "batch", "grad", "lanczos", "vectors", "basis"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "mul":
        tables = rng.random() < 0.6
        if rng.random() < 0.5:
            L1, L2, model = rng.randint(10, 28 if tables else 26), 1, "chain"
        else:
            L1, L2 = rng.choice(_TORI + [(7, 4), (6, 5)] if tables else _TORI)
            model = rng.choice(["triangular", "square"])
        n = L1 * L2
        q = n % 2 + 2 * rng.choice([0, 0, 1])
        reduced = n > 18 or rng.random() < 0.7
        k1 = rng.randrange(L1) if reduced else 0
        k2 = rng.randrange(L2) if reduced else 0
        return _case(kind, model, L1, L2, q, k1, k2, prec, tables, reduced)
    if kind == "host":
        L1 = rng.randint(12, 27)
        return _case(kind, "chain", L1, 1, L1 % 2, rng.randrange(L1), 0, prec, True)
    if kind == "batch":
        L1, L2 = rng.choice([(4, 3), (4, 4), (5, 4), (6, 4), (5, 5), (12, 1), (18, 1), (21, 1), (24, 1)])
        return _case(kind, "chain" if L2 == 1 else rng.choice(["triangular", "square"]), L1, L2, (L1 * L2) % 2,
                     0, 0, "mixed", True)
    if kind == "grad":
        L1 = 2 * rng.randint(6, 14)
        return _case(kind, "coupled", L1, 1, 0, 0, 0, prec, True)
    if kind == "lanczos":
        L1 = rng.choice([16, 18, 20, 22, 24])
        return _case(kind, "chain", L1, 1, 0, 0, 0, "fp64", True)
    if kind == "vectors":
        L1 = rng.randint(10, 26)
        return _case(kind, "chain", L1, 1, L1 % 2, rng.randrange(L1), 0, prec, False)
    L1, L2 = rng.choice([(rng.randint(12, 26), 1), rng.choice(_TORI)])
    return _case(kind, "chain" if L2 == 1 else "square", L1, L2, (L1 * L2) % 2, rng.randrange(L1), 0, "fp64", False)


# ---- the model -----------------------------------------------------------------------------------
def _torus_bonds(L1, L2, vectors):
    out = []
    for dx, dy in vectors:
        for y in range(L2):
            for x in range(L1):
                out.append((x + L1 * y, (x + dx) % L1 + L1 * ((y + dy) % L2)))
    return out


def _bonds(case):
    """(bonds, jxy, jz): the Heisenberg chain (J = 1), the XXZ J1-J2 triangular torus (Jz/Jxy = 0.8,
    J2/J1 = 0.125) or the J1-J2 square torus (J2/J1 = 0.5)."""
    L1, L2 = case["L1"], case["L2"]
    if L2 == 1:
        b = [(i, (i + 1) % L1) for i in range(L1)]
        return b, [1.0] * L1, [1.0] * L1
    if case["model"] == "triangular":
        sets = (([(1, 0), (1, 1), (0, 1)], 1.0), ([(2, 1), (1, 2), (-1, 1)], 0.125))
        aniso = 0.8
    else:
        sets = (([(1, 0), (0, 1)], 1.0), ([(1, 1), (1, -1)], 0.5))
        aniso = 1.0
    bonds, jxy, jz = [], [], []
    for vecs, j in sets:
        bs = [b for b in _torus_bonds(L1, L2, vecs) if b[0] != b[1]]
        bonds += bs
        jxy += [j] * len(bs)
        jz += [j * aniso] * len(bs)
    return bonds, jxy, jz


def _rows(case):
    """Rows of the sector (to the accuracy of a work estimate: orbits are nearly all of full length)."""
    n = case["L1"] * case["L2"]
    full = math.comb(n, (n - case["q"]) // 2)
    return full if not case["reduced"] else max(1, full // n)


def _nonzeros(case):
    n = case["L1"] * case["L2"]
    k = (n - case["q"]) // 2
    return int(_rows(case) * len(_bonds(case)[0]) * 2.0 * k * (n - k) / (n * (n - 1)))


def work(case):
    N, nnz = _rows(case), _nonzeros(case)
    n = case["L1"] * case["L2"]
    s = 16 if case["prec"] == "fp64" else 8
    full = math.comb(n, (n - case["q"]) // 2)
    kind = case["kind"]
    # a product: the row states, x and y; a complex multiply-add per nonzero
    mul = {"bytes": N * (8 + 2 * s), "flops": 8.0 * nnz}
    if kind in ("mul", "host"):
        return mul
    if kind == "batch":
        return {"bytes": n * mul["bytes"], "flops": n * mul["flops"]}
    if kind == "grad":
        # x, gy in, y and dL/dx out; forward, adjoint and the per-coupling inner products
        return {"bytes": N * (8 + 4 * s), "flops": 24.0 * nnz}
    if kind == "lanczos":
        # products; two Gram-Schmidt passes over the stored basis (each vector read for its dot and
        # its subtraction, 8 + 8 flops an entry)
        m = min(LANCZOS_STEPS, N)
        return {"bytes": m * mul["bytes"] + 16.0 * N * m, "flops": m * mul["flops"] + 2 * 16.0 * N * m * (m + 1) / 2}
    if kind == "vectors":
        # the small vector and the row states in and out; the parent vector written, and read again
        return {"bytes": 2 * (N * (8 + s) + full * s), "flops": 8.0 * full}
    # representatives and orbit sizes out; keys in, two rows out each
    return {"bytes": 12.0 * N + 24.0 * LOOKUPS, "flops": 0.0}


# ---- what a program has in hand before the call ----------------------------------------------------
def _sector(case, lazy=True):
    import edgpu
    hs, _ = edgpu.spin_half_system(case["L1"] * case["L2"])
    return hs, edgpu.represent(edgpu.HilbertSpaceSector(hs, case["q"]), lazy=lazy and case["reduced"])


def _space(case, k=None):
    import edgpu
    hs, hsr = _sector(case)
    if not case["reduced"]:
        return hs, hsr
    k = (case["k1"], case["k2"]) if k is None else k
    return hs, edgpu.symmetry_reduce(hsr, edgpu.translation_symops((case["L1"], case["L2"]), k))


def _build_tables(opr, prec, autotune=True):
    """A solver's set-up, as the benchmark does it: parent-state map, target table, column slabs."""
    if hasattr(opr.space, "build_map"):
        opr.space.build_map()
    if opr.build_targets():
        if hasattr(opr.space, "free_map"):
            opr.space.free_map()
        opr.build_slabs(slab_bytes=SLAB_BYTES)
    if autotune:
        opr.autotune(prec)


def _vector(n, seed, prec):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    v = torch.randn(n, dtype=torch.complex128, device="cuda", generator=g)
    v /= torch.linalg.vector_norm(v)
    return v if prec == "fp64" else v.to(torch.complex64)


def _couplings(case, seed):
    """Per-bond couplings 0.5 + U[0, 1) drawn from the seed."""
    g = torch.Generator().manual_seed(int(seed) + 7)
    return 0.5 + torch.rand(case["L1"], dtype=torch.float64, generator=g)


def prepare(case, seed):
    import edgpu
    from edgpu import lattice
    kind, prec = case["kind"], case["prec"]
    s = {"kind": kind, "prec": prec}
    if kind == "basis":
        s["hs"], _ = edgpu.spin_half_system(case["L1"] * case["L2"])
        s["q"] = case["q"]
        s["symops"] = edgpu.translation_symops((case["L1"], case["L2"]), (case["k1"], case["k2"]))
        # states whose rows the program asks for: random words of the sector
        n = case["L1"] * case["L2"]
        g = torch.Generator().manual_seed(int(seed))
        order = torch.rand((LOOKUPS, n), generator=g).argsort(1)[:, :(n - case["q"]) // 2]
        s["keys"] = (1 << order).sum(1).numpy().astype(np.uint64)
        return s
    if kind == "batch":
        hs, hsr = _sector(case)
        H = lattice.xxz_hamiltonian(hs, *_bonds(case))
        s["oprs"] = []
        for m2 in range(case["L2"]):
            for m1 in range(case["L1"]):
                sp = edgpu.symmetry_reduce(hsr, edgpu.translation_symops((case["L1"], case["L2"]), (m1, m2)))
                opr = edgpu.represent(sp, H)
                _build_tables(opr, prec)
                s["oprs"].append(opr)
        s["batch"] = edgpu.Batch(s["oprs"])
        s["batch"].autotune(prec)
        s["x"] = [_vector(o.dimension, seed * 100 + i, prec) for i, o in enumerate(s["oprs"])]
        s["y"] = [torch.empty_like(x) for x in s["x"]]
        return s
    hs, space = _space(case)
    s["space"] = space
    n = space.dimension
    if kind == "vectors":
        s["x"] = _vector(n, seed, prec)
        return s
    if kind == "grad":
        J = _couplings(case, seed)
        m, r, c, a, ids = lattice.heisenberg_coupled(hs, _bonds(case)[0])
        opr = edgpu.OperatorRepresentation.from_terms(space, m, r, c, a, coupling_ids=ids, couplings=J.numpy())
        _build_tables(opr, prec)
        opr.build_adjoint_targets()
        s["opr"] = opr
        s["x"] = _vector(n, seed, prec).requires_grad_(True)
        s["J"] = J.requires_grad_(True)
        s["gy"] = _vector(n, seed + 1000003, prec)
        return s
    opr = edgpu.represent(space, lattice.xxz_hamiltonian(hs, *_bonds(case)))
    s["opr"] = opr
    if case["tables"]:
        _build_tables(opr, prec)
    x = _vector(n, seed, "fp64" if kind in ("host", "lanczos") else prec)
    if kind == "host":
        s["x"] = x.cpu().numpy()
        s["y"] = np.empty_like(s["x"])
    elif kind == "lanczos":
        s["v0"] = x.cpu().numpy()
    else:
        s["x"] = x
        s["y"] = torch.empty_like(x)
    return s


def run(s):
    import edgpu
    kind = s["kind"]
    if kind in ("mul", "host"):
        return edgpu.mul_(s["y"], s["opr"], s["x"], precision=s["prec"])
    if kind == "batch":
        return s["batch"].mul_(s["y"], s["x"], precision=s["prec"])
    if kind == "grad":
        s["x"].grad = s["J"].grad = None
        y = edgpu.apply_hamiltonian(s["opr"], s["x"], s["J"])
        y.backward(s["gy"])
        return {"y": y.detach(), "gx": s["x"].grad, "gJ": s["J"].grad}
    if kind == "lanczos":
        r = edgpu.lanczos(s["opr"], LANCZOS_STEPS, precision=s["prec"], reorth=True, v0=s["v0"], tol=0.0,
                          want_vector=True)
        return {"e0": np.array([r.e0]), "ground_state": r.ground_state}
    if kind == "vectors":
        large = edgpu.symmetry_unreduce(s["space"], s["x"])
        return {"large": large, "small": edgpu.symmetry_reduce(s["space"], large)}
    hsr = edgpu.represent(edgpu.HilbertSpaceSector(s["hs"], s["q"]))
    rhsr = edgpu.symmetry_reduce(hsr, s["symops"])
    return {"basis": rhsr.basis_list, "orbits": rhsr.orbit_sizes(), "rows": hsr.lookup(s["keys"]),
            "reduced_rows": rhsr.lookup(s["keys"])}


# ---- the same results in plain torch, 64 bits ------------------------------------------------------
_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_CHUNK = 1 << 22


def _popcount(v):
    v = v - ((v >> 1) & 0x5555555555555555)
    v = (v & 0x3333333333333333) + ((v >> 2) & 0x3333333333333333)
    v = (v + (v >> 4)) & 0x0F0F0F0F0F0F0F0F
    return (v * 0x0101010101010101) >> 56


def _states(n, k):
    """The words of n bits with k bits set, ascending."""
    out = []
    step = 1 << 26
    for lo in range(0, 1 << n, step):
        v = torch.arange(lo, min(lo + step, 1 << n), dtype=torch.int64, device=_DEV)
        out.append(v[_popcount(v) == k])
    return torch.cat(out)


def _shift_x(s, L1, L2):
    row = sum(1 << (L1 * y) for y in range(L2))
    low = row * ((1 << (L1 - 1)) - 1)
    return ((s & low) << 1) | ((s >> (L1 - 1)) & row)


def _shift_y(s, L1, L2):
    n = L1 * L2
    return ((s << L1) | (s >> (n - L1))) & ((1 << n) - 1)


class _Sector:
    """Representatives and stabiliser sizes of a momentum sector, and canonicalisation in it."""

    def __init__(self, case, k=None):
        self.L1, self.L2 = case["L1"], case["L2"]
        self.n = self.L1 * self.L2
        self.reduced = case["reduced"]
        self.k = (case["k1"], case["k2"]) if k is None else k
        self.parent = _states(self.n, (self.n - case["q"]) // 2)
        if not self.reduced:
            self.reps = self.parent
            return
        keep, stab = [], []
        for part in self.parent.split(_CHUNK):
            low, g, st, ok = self.canon(part, True)
            hit = (low == part) & ok
            keep.append(part[hit])
            stab.append(st[hit])
        self.reps = torch.cat(keep)
        self.stab = torch.cat(stab)

    def phase_of(self, a, b):
        return -2.0 * math.pi * ((self.k[0] * a / self.L1 + self.k[1] * b / self.L2) % 1.0)

    def canon(self, q, full=False):
        """(smallest translate, index a + L1 b of an element reaching it); full: also the stabiliser's
        size and whether the character is 1 on all of it."""
        low, g, t = q.clone(), torch.zeros_like(q), q
        st = torch.zeros_like(q) if full else None
        ok = torch.ones_like(q, dtype=torch.bool) if full else None
        for b in range(self.L2):
            for a in range(self.L1):
                if a or b:
                    less = t < low
                    low = torch.where(less, t, low)
                    g = torch.where(less, a + self.L1 * b, g)
                if full:
                    same = t == q
                    st += same
                    if (self.k[0] * a * self.L2 + self.k[1] * b * self.L1) % (self.L1 * self.L2):
                        ok &= ~same
                t = _shift_x(t, self.L1, self.L2)
            t = _shift_y(t, self.L1, self.L2)
        return (low, g, st, ok) if full else (low, g)

    def locate(self, q):
        """(row of q's representative or -1, chi(g) with g q the representative)."""
        if not self.reduced:
            c = torch.searchsorted(self.reps, q).clamp(max=self.reps.numel() - 1)
            return torch.where(self.reps[c] == q, c, -1), None
        low, g = self.canon(q)
        c = torch.searchsorted(self.reps, low).clamp(max=self.reps.numel() - 1)
        c = torch.where(self.reps[c] == low, c, -1)
        ang = torch.tensor([self.phase_of(a, b) for b in range(self.L2) for a in range(self.L1)],
                           dtype=torch.float64, device=_DEV)
        return c, torch.polar(torch.ones_like(ang), ang)[g]


def _bond_product(sec, bonds, jxy, jz, x, per_bond=None):
    """y = H x row by row; per_bond: a callback (bond, rows, element, columns, diagonal) instead."""
    y = torch.zeros_like(x)
    N = sec.reps.numel()
    step = max(1, _CHUNK)
    for r0 in range(0, N, step):
        b = sec.reps[r0:r0 + step]
        rows = torch.arange(r0, r0 + b.numel(), device=_DEV)
        for e, (i, j) in enumerate(bonds):
            anti = (((b >> i) ^ (b >> j)) & 1).bool()
            diag = torch.where(anti, -0.25, 0.25).to(torch.float64) * jz[e]
            sel = rows[anti]
            c, chi = sec.locate(b[anti] ^ ((1 << i) | (1 << j)))
            hit = c >= 0
            sel, c = sel[hit], c[hit]
            el = torch.full((sel.numel(),), 0.5 * jxy[e], dtype=torch.complex128, device=_DEV)
            if chi is not None:
                el = el * chi[hit] * torch.sqrt(sec.stab[c].double() / sec.stab[sel].double())
            if per_bond is not None:
                per_bond(e, rows, diag, sel, el, c)
            else:
                y[rows] += diag * x[rows]
                y.index_add_(0, sel, el * x[c])
    return y


def _exact_mul(case, x, k=None, sec=None):
    bonds, jxy, jz = _bonds(case)
    sec = sec or _Sector(case, k)
    return _bond_product(sec, bonds, jxy, jz, x.to(_DEV, torch.complex128))


def _lowest(A, B):
    T = np.diag(A) + np.diag(B, 1) + np.diag(B, -1)
    w, v = np.linalg.eigh(T)
    return w[0], v[:, 0]


def _exact_lanczos(case, v0):
    """The lowest eigenpair in the Krylov space of v0, phase as sum_j s_j v_j with s_0 > 0."""
    sec = _Sector(case)
    bonds, jxy, jz = _bonds(case)
    N = sec.reps.numel()
    r, c, v = [], [], []

    def add(e, rows, diag, sel, el, cols):
        r.extend((rows, sel))
        c.extend((rows, cols))
        v.extend((diag.to(torch.complex128), el))

    _bond_product(sec, bonds, jxy, jz, torch.zeros(1, dtype=torch.complex128, device=_DEV).expand(N), add)
    H = torch.sparse_coo_tensor(torch.stack((torch.cat(r), torch.cat(c))), torch.cat(v), (N, N)).coalesce()
    m = min(LANCZOS_STEPS, N)
    V = torch.zeros((m, N), dtype=torch.complex128, device=_DEV)
    V[0] = torch.from_numpy(v0).to(_DEV)
    V[0] /= torch.linalg.vector_norm(V[0])
    A, B = [], []
    for j in range(m):
        w = torch.mv(H, V[j])
        A.append(float(torch.vdot(V[j], w).real))
        for _ in range(2):
            w = w - V[:j + 1].T @ (V[:j + 1].conj() @ w)
        beta = float(torch.linalg.vector_norm(w))
        if j == m - 1 or beta <= 1e-12 * max(1.0, abs(A[-1])):
            break
        B.append(beta)
        V[j + 1] = w / beta
    e, s = _lowest(A, B)
    s = s * (1.0 if s[0] >= 0 else -1.0)
    g = V[:len(A)].T @ torch.from_numpy(s).to(_DEV, torch.complex128)
    return {"e0": np.array([e]), "ground_state": (g / torch.linalg.vector_norm(g)).cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "basis":
        return None     # whole numbers: they stay equal
    if kind == "batch":
        out = []
        for i in range(case["L1"] * case["L2"]):
            k = (i % case["L1"], i // case["L1"])
            sec = _Sector(case, k)
            x = _vector(sec.reps.numel(), seed * 100 + i, case["prec"])
            out.append(_exact_mul(case, x, sec=sec))
        return out
    sec = _Sector(case)
    N = sec.reps.numel()
    if kind == "lanczos":
        return _exact_lanczos(case, _vector(N, seed, "fp64").cpu().numpy())
    x = _vector(N, seed, "fp64" if kind == "host" else case["prec"])
    if kind == "mul":
        return _exact_mul(case, x, sec=sec)
    if kind == "host":
        return _exact_mul(case, x, sec=sec).cpu().numpy()
    if kind == "vectors":
        c, chi = sec.locate(sec.parent)
        size = sec.n // sec.stab
        hit = c >= 0
        cc = c.clamp(min=0)
        large = torch.where(hit, chi / torch.sqrt(size[cc].double()) * x.to(torch.complex128)[cc], 0)
        return {"large": large, "small": x.to(torch.complex128)}
    # grad: y = H x, dL/dx = H^dagger gy, dL/dJ_b = Re <gy | H_b x>
    J = _couplings(case, seed)
    gy = _vector(N, seed + 1000003, case["prec"]).to(torch.complex128)
    xx = x.to(torch.complex128)
    bonds = _bonds(case)[0]
    y, gx = torch.zeros_like(xx), torch.zeros_like(xx)
    gJ = torch.zeros(len(bonds), dtype=torch.float64)

    def add(e, rows, diag, sel, el, cols):
        hb = torch.zeros_like(xx)
        hb[rows] += diag * xx[rows]
        hb.index_add_(0, sel, el * xx[cols])
        y.add_(hb, alpha=float(J[e]))
        gx[rows] += float(J[e]) * diag * gy[rows]
        gx.index_add_(0, cols, float(J[e]) * el.conj() * gy[sel])
        gJ[e] += float(torch.vdot(gy, hb).real)

    one = [1.0] * len(bonds)
    _bond_product(sec, bonds, one, one, xx, add)
    return {"y": y, "gx": gx, "gJ": gJ}
