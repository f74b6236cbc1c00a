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
