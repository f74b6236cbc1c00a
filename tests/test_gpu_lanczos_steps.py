"""The Lanczos step with a stored basis: one projection on the basis per step, taken off in single precision
while the projections are at the level of rounding errors, in FP64 otherwise, and a second projection where
the first took most of the vector away.  Against dense eigenvalues (1e-10 relative, as the solver's other
tests) at sizes around the kernels' blocks, with more steps than rows, and from start vectors whose Krylov
space is (nearly) invariant.  The vector's residual |H v - E v| is checked (1e-7) where the run goes on for
all its steps; a run that stops when the eigenvalue has settled says nothing about it."""
import numpy as np
import pytest

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
