"""The coupling gradient in FP64: the kernel's form for one unit amplitude per pair with the pair's own
diagonal terms (three double-precision operations per target), with and without the product, and the
operators next to it that do not have that form (a field, a second anisotropy, a momentum, an amplitude
of its own, a constant), against Re <gy | H_c x> of the oracle: 1e-12 of the largest term sum."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _terms(E, hs, L, kind):
    from edgpu import lattice
    from edgpu.operators import pauli_matrix
    m, r, c, a, ids = lattice.heisenberg_coupled(hs, lattice.chain_bonds(L))
    a = a.copy()
    diag = r == c
    if kind == "xxz":
        a[diag] *= 0.7
    elif kind == "two anisotropies":
        a[diag & (ids == 1)] *= 0.7
    elif kind == "own amplitude":
        a[~diag & (ids == 2)] *= 1.5
    elif kind in ("field", "constant"):
        z = pauli_matrix(hs, 0, "z")
        extra = [(t.bitmask, t.bitrow, t.bitcol, t.amplitude) for t in z.terms] if kind == "field" else [(0, 0, 0, 0.5)]
        for t in extra:
            m, r, c = (np.append(v, np.uint64(w)) for v, w in zip((m, r, c), t[:3]))
            a, ids = np.append(a, complex(t[3])), np.append(ids, np.int32(L))
    return m, r, c, a, ids.astype(np.int32)


@pytest.mark.parametrize("kind", ["heisenberg", "xxz", "two anisotropies", "own amplitude", "field", "constant"])
@pytest.mark.parametrize("L,q,k", [(5, 1, 0), (8, 0, 0), (11, 3, 0), (12, 0, 0), (13, 1, 0), (12, 0, 5), (16, 2, 0)])
def test_gradient(L, q, k, kind):
    import torch
    import edgpu as E
    hs, _ = E.spin_half_system(L)
    rh = E.symmetry_reduce(E.represent(E.HilbertSpaceSector(hs, q)), E.translation_symops(L, k))
    m, r, c, a, ids = _terms(E, hs, L, kind)
    n_c = int(ids.max()) + 1
    J = 0.5 + np.random.default_rng(L).random(n_c)
    opr = E.OperatorRepresentation.from_terms(rh, m, r, c, a, coupling_ids=ids, couplings=J)
    sites = O.spin_half_sites(L)
    maps, amps = O.translation_symops((L, 1), (k, 0))
    red = O.symmetry_reduce(O.hs_get_basis_list(sites, [(q,)]), *O.bit_layout(sites), maps, amps)
    x, gy = O.complex_gaussian(red.dim, 1), O.complex_gaussian(red.dim, 2)
    want, y_want, scale = np.zeros(n_c), np.zeros(red.dim, dtype=complex), 0.0
    for j in range(n_c):
        t = [(int(m[i]), int(r[i]), int(c[i]), complex(a[i])) for i in range(len(m)) if ids[i] == j]
        hx = O.apply_rows(red, t, x)
        want[j] = np.vdot(gy, hx).real
        scale = max(scale, np.linalg.norm(gy) * np.linalg.norm(hx))
        y_want += J[j] * hx
    xd, gd = torch.from_numpy(x).cuda(), torch.from_numpy(gy).cuda()
    torch.cuda.synchronize()
    assert rh.build_map()
    for table in (False, True):
        if table:
            assert opr.build_targets(1 << 28)
        g = E.coupling_grad(opr, xd, gd, precision="fp64")
        assert np.max(np.abs(g - want)) < 1e-12 * max(scale, 1.0)
        y = torch.full_like(xd, float("nan"))
        g2 = E.coupling_grad(opr, xd, gd, precision="fp64", y=y)
        assert np.array_equal(g, g2)
        assert np.linalg.norm(y.cpu().numpy() - y_want) < 1e-12 * max(np.linalg.norm(y_want), 1.0)
    J2 = J[::-1].copy()
    opr.set_couplings(J2)
    assert np.array_equal(E.coupling_grad(opr, xd, gd, precision="fp64"), g)
