"""The Lanczos step with a stored basis: one projection on the basis per step, taken off in single precision
while the projections are at the level of rounding errors, in FP64 otherwise, and a second projection where
the first took most of the vector away.  Against dense eigenvalues (1e-10 relative, as the solver's other
tests) at sizes around the kernels' blocks, with more steps than rows, and from start vectors whose Krylov
space is (nearly) invariant.  The vector's residual |H v - E v| is checked (1e-7) where the run goes on for
all its steps; a run that stops when the eigenvalue has settled says nothing about it."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _operator(E, L, q, k):
    from edgpu import lattice
    hs, _ = E.spin_half_system(L)
    hsr = E.represent(E.HilbertSpaceSector(hs, q))
    bonds = lattice.chain_bonds(L) + [(i, (i + 2) % L) for i in range(L)]
    H = lattice.xxz_hamiltonian(hs, bonds, [1.0] * L + [0.3] * L, [0.9] * L + [0.2] * L)
    return E.represent(E.symmetry_reduce(hsr, E.translation_symops(L, k)), H)


def _check(r, w):
    assert abs(r.e0 - w[0]) < 1e-10 * max(1.0, abs(w[0]))
    assert abs(np.linalg.norm(r.ground_state) - 1.0) < 1e-10


@pytest.mark.parametrize("L,q,k", [(4, 2, 0), (5, 1, 1), (8, 0, 0), (12, 0, 0), (14, 0, 3), (14, 2, 0), (16, 0, 1)])
@pytest.mark.parametrize("precision,refine", [("fp64", False), ("mixed", True)])
def test_e0_matches_dense(L, q, k, precision, refine):
    import edgpu as E
    opr = _operator(E, L, q, k)
    w = np.linalg.eigvalsh(opr.todense())
    steps = min(opr.dimension + 5, 160)
    r = E.lanczos(opr, steps, precision=precision, reorth=True, seed=3, refine=refine, tol=1e-12, want_vector=True)
    _check(r, w)
    if precision == "fp64":
        r2 = E.lanczos(opr, steps, precision=precision, reorth=True, seed=3, tol=1e-12, want_vector=True)
        assert r2.e0 == r.e0 and np.array_equal(r2.ground_state, r.ground_state)


@pytest.mark.parametrize("noise", [0.0, 1e-13, 1e-10, 1e-6, 1e-3])
def test_nearly_invariant_start(noise):
    """Three eigenvectors and a little of all others: after three steps what is left of the recurrence is as
    small as the noise, and the projections on the basis are not small beside it."""
    import edgpu as E
    opr = _operator(E, 14, 0, 0)
    M = opr.todense()
    w, U = np.linalg.eigh(M)
    rng = np.random.default_rng(2)
    v0 = U[:, [0, 5, 40]] @ np.array([0.7, 0.5, 0.5]) + 0j
    v0 = v0 + noise * (rng.standard_normal(len(w)) + 1j * rng.standard_normal(len(w)))
    r = E.lanczos(opr, 120, precision="fp64", reorth=True, v0=v0, tol=0.0, want_vector=True)
    _check(r, w)
    assert np.linalg.norm(M @ r.ground_state - r.e0 * r.ground_state) < 1e-7


def test_more_vectors_than_blocks():
    """More groups of 16 basis vectors than row blocks that fit on the GPU: each group has one row block, in
    every step from there on.  The lowest Ritz values of the full-length run are eigenvalues, each once
    (1e-9 of a sparse eigensolver's; copies would show a lost orthogonality); a run that stops early too."""
    import scipy.linalg
    import scipy.sparse.linalg
    import torch
    import edgpu as E
    from edgpu import lattice
    hs, _ = E.spin_half_system(15)
    hsr = E.represent(E.HilbertSpaceSector(hs, 1))
    rng = np.random.default_rng(4)
    H = lattice.xxz_hamiltonian(hs, lattice.chain_bonds(15), 0.5 + rng.random(15), 0.5 + rng.random(15))
    opr = E.represent(hsr, H)
    steps = 32 * torch.cuda.get_device_properties(0).multi_processor_count + 5
    assert steps < opr.dimension
    basis = O.hs_get_basis_list(O.spin_half_sites(15), [(1,)])
    terms = [(t.bitmask, t.bitrow, t.bitcol, t.amplitude) for t in H.terms]
    A = scipy.sparse.linalg.LinearOperator((len(basis),) * 2, dtype=complex,
                                           matvec=lambda v: O.apply_rows(basis, terms, np.ravel(v)))
    w = np.sort(scipy.sparse.linalg.eigsh(A, k=8, which="SA", tol=1e-12, return_eigenvectors=False))
    r = E.lanczos(opr, steps, precision="fp64", reorth=True, seed=3, tol=1e-12)
    assert r.steps < 400 and abs(r.e0 - w[0]) < 1e-9 * abs(w[0])
    r = E.lanczos(opr, steps, precision="fp64", reorth=True, seed=3, tol=0.0)
    assert r.steps == steps
    t = scipy.linalg.eigvalsh_tridiagonal(r.alphas, r.betas[:-1], select="i", select_range=(0, 7))
    assert np.abs(t - w).max() < 1e-9 * np.abs(w).max()


@pytest.mark.parametrize("L,q", [(10, 0), (11, 1)])   # 252 and 462 rows: steps on both sides of 256 vectors
def test_full_spectrum(L, q):
    """As many steps as rows: the tridiagonal matrix has the operator's eigenvalues (1e-10), which it has only
    while the basis stays orthogonal."""
    import scipy.linalg
    import edgpu as E
    from edgpu import lattice
    hs, _ = E.spin_half_system(L)
    rng = np.random.default_rng(L)
    H = lattice.xxz_hamiltonian(hs, lattice.chain_bonds(L), 0.5 + rng.random(L), 0.5 + rng.random(L))
    opr = E.represent(E.represent(E.HilbertSpaceSector(hs, q)), H)
    w = np.linalg.eigvalsh(opr.todense())
    r = E.lanczos(opr, opr.dimension, precision="fp64", reorth=True, seed=5, tol=0.0)
    assert r.steps == opr.dimension
    t = scipy.linalg.eigvalsh_tridiagonal(r.alphas, r.betas[:-1])
    assert np.abs(t - w).max() < 1e-10 * np.abs(w).max()


@pytest.mark.parametrize("refine", [False, True])
def test_complex64_basis(refine):
    """A mixed-precision run whose basis fits as complex64 only, reorthogonalised."""
    import edgpu as E
    opr = _operator(E, 16, 0, 1)
    w = np.linalg.eigvalsh(opr.todense())
    steps = 300
    E.set_krylov_limit(12 * (steps + 1) * opr.dimension)
    try:
        r = E.lanczos(opr, steps, precision="mixed", reorth=True, seed=3, refine=refine, tol=1e-12 if refine else 0.0)
        assert abs(r.e0 - w[0]) < (1e-10 if refine else 1e-5) * abs(w[0])
        if not refine:
            t = np.linalg.eigvalsh(np.diag(r.alphas) + np.diag(r.betas[:-1], 1) + np.diag(r.betas[:-1], -1))
            assert np.abs(t[:4] - w[:4]).max() < 1e-5 * abs(w[0])
    finally:
        E.set_krylov_limit(0)


def test_large_sector_second_projection():
    """More than 2^20 rows (steps are then not issued ahead), from a start whose Krylov space is invariant up to
    1e-7, against the same recurrence on the host with two projections in every step."""
    import edgpu as E
    from edgpu import lattice
    L = 23
    hs, _ = E.spin_half_system(L)
    rng = np.random.default_rng(8)
    H = lattice.xxz_hamiltonian(hs, lattice.chain_bonds(L), 1e-7 * (1.0 + rng.random(L)), 1.0 + rng.random(L))
    opr = E.represent(E.represent(E.HilbertSpaceSector(hs, 1)), H)
    N = opr.dimension
    assert N > 1 << 20
    v0 = np.zeros(N, dtype=complex)
    v0[rng.integers(N, size=3)] = [0.8, 0.5, 0.3j]
    steps = 8
    r = E.lanczos(opr, steps, precision="fp64", reorth=True, v0=v0, tol=0.0)
    basis = O.hs_get_basis_list(O.spin_half_sites(L), [(1,)])
    terms = [(t.bitmask, t.bitrow, t.bitcol, t.amplitude) for t in H.terms]
    V, alphas, betas = [v0 / np.linalg.norm(v0)], [], []
    for j in range(steps):
        w = O.apply_rows(basis, terms, V[j])
        alphas.append(np.vdot(V[j], w).real)
        for _ in range(2):
            for u in V:
                w = w - np.vdot(u, w) * u
        betas.append(np.linalg.norm(w))
        V.append(w / betas[-1])
    assert betas[2] < 1e-5 < betas[1]
    assert np.abs(r.alphas - alphas).max() < 1e-6 * np.abs(alphas).max()
    assert np.abs(r.betas[:-1] / betas[:-1] - 1.0).max() < 1e-6


def test_memory_beside_the_basis():
    """A reorthogonalised run holds the basis that the Krylov limit counts, one vector more, and small
    buffers (the device's free memory watched from another thread)."""
    import threading
    import torch
    import edgpu as E
    opr = _operator(E, 27, 1, 0)
    steps, vector = 100, 16 * opr.dimension
    E.lanczos(opr, 5, precision="fp64", reorth=True, seed=3, tol=0.0)   # (the product's own tables)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    lowest, stop = [before], threading.Event()

    def watch():
        while not stop.is_set():
            lowest.append(torch.cuda.mem_get_info()[0])

    t = threading.Thread(target=watch)
    t.start()
    E.lanczos(opr, steps, precision="fp64", reorth=True, seed=3, tol=0.0)
    stop.set()
    t.join()
    used = before - min(lowest)
    assert vector * (steps + 1) < used
    assert used < vector * (steps + 1) + vector + (4 << 20)
