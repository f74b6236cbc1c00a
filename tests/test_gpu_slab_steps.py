"""The slab table's steps (tiles of 32 rows, at most one entry per row and step): padded tables (one pass)
and tables with masks (many passes of few entries), at sector sizes around the tile's edge, against the
oracle's reduced product.  Tolerances: FP64 1e-12, mixed 1e-5 (the bounds of the slab product's other
tests).  An infinite element of x reaches the rows that have a target on it and no others."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def relerr(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


def _sector(E, shape, q, k, scaling, slab_bytes):
    from edgpu import lattice
    n = shape[0] * shape[1]
    hs, _ = E.spin_half_system(n)
    if shape[1] == 1:
        bonds = lattice.chain_bonds(n)
        j = [1.0] * n
    else:
        nn = lattice.torus_bonds(*shape, lattice.TRIANGULAR_NN)
        nnn = lattice.torus_bonds(*shape, lattice.TRIANGULAR_NNN)
        bonds, j = nn + nnn, [1.0] * len(nn) + [0.3] * len(nnn)
    hsr = E.represent(E.HilbertSpaceSector(hs, q))
    opr = E.represent(E.symmetry_reduce(hsr, E.translation_symops(shape, k)), lattice.xxz_hamiltonian(hs, bonds, j, j))
    sites = O.spin_half_sites(n)
    parent = O.hs_get_basis_list(sites, [(q,)])
    maps, amps = O.translation_symops(shape, k)
    red = O.symmetry_reduce(parent, *O.bit_layout(sites), maps, amps)
    assert opr.build_targets(1 << 30)
    opr.slab_scaling(scaling)
    assert opr.build_slabs(slab_bytes=slab_bytes, max_bytes=1 << 30)
    return opr, red, O.heisenberg_terms(n, bonds, j, j)


# (shape, 2Sz, momentum): sectors of 1, 3, 32 and 33 rows (one tile, one row more), ragged ones, and
# several tiles; many passes: 1024 columns per slab
CASES = [((4, 1), 2, (0, 0)), ((6, 1), 0, (1, 0)), ((13, 1), 5, (3, 0)), ((11, 1), 3, (2, 0)), ((12, 1), 0, (0, 0)),
         ((4, 3), 0, (1, 2)), ((17, 1), 1, (5, 0)), ((5, 4), 0, (0, 0)), ((20, 1), 0, (3, 0))]


@pytest.mark.parametrize("slab_bytes", [1 << 20, 8192])
@pytest.mark.parametrize("scaling", [1, 2])
@pytest.mark.parametrize("shape,q,k", CASES)
def test_steps(shape, q, k, scaling, slab_bytes):
    import torch
    import edgpu as E
    opr, red, terms = _sector(E, shape, q, k, scaling, slab_bytes)
    N = opr.dimension
    x = O.complex_gaussian(N, 3)
    want = O.apply_rows(red, terms, x)
    for prec, dt, tol in (("fp64", torch.complex128, 1e-12), ("mixed", torch.complex64, 1e-5)):
        xd = torch.from_numpy(x).to(dt).cuda()
        y = torch.full_like(xd, float("nan"))
        E.mul_(y, opr, xd, precision=prec)
        assert relerr(y.cpu().numpy(), want) < tol
        E.apply_(y, opr, xd, precision=prec)
        assert relerr(y.cpu().numpy(), 2 * want) < tol


@pytest.mark.parametrize("slab_bytes", [1 << 20, 8192])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_infinite_element(prec, slab_bytes):
    import torch
    import edgpu as E
    opr, _, _ = _sector(E, (17, 1), 1, (0, 0), 1, slab_bytes)
    dt = torch.complex128 if prec == "fp64" else torch.complex64
    x = torch.from_numpy(O.complex_gaussian(opr.dimension, 5)).to(dt).cuda()
    for col in (0, 37, opr.dimension - 1):
        xi = x.clone()
        xi[col] = complex(float("inf"), 0.0)
        y = torch.empty_like(xi)
        E.mul_(y, opr, xi, precision=prec)
        opr.slab_use(prec, False)
        y0 = torch.empty_like(xi)
        E.mul_(y0, opr, xi, precision=prec)
        opr.slab_use(prec, True)
        fin, fin0 = torch.isfinite(torch.view_as_real(y)).all(1), torch.isfinite(torch.view_as_real(y0)).all(1)
        assert torch.equal(fin, fin0) and not bool(fin0.all()) and bool(fin0.any())


# sectors of long rows in one pass, whose row masks take more than a byte a row, and of several passes
@pytest.mark.parametrize("slab_bytes", [1 << 20, 8192])
@pytest.mark.parametrize("scaling", [1, 2])
@pytest.mark.parametrize("shape,q,k", [((4, 3), 0, (0, 0)), ((4, 4), 0, (1, 0)), ((5, 4), 0, (0, 0)), ((5, 4), 2, (2, 1)),
                                       ((17, 1), 1, (5, 0)), ((20, 1), 0, (0, 0))])
def test_limit_of_counts(shape, q, k, scaling, slab_bytes):
    """A limit of 4 bytes an entry, a byte a row and pass and 4 bytes a tile and pass (and 17 bytes a row of a
    scaled table) has room for a table: neither padding nor masks fit it, the rows' counts do."""
    import torch
    import edgpu as E
    opr, red, terms = _sector(E, shape, q, k, scaling, slab_bytes)
    N = opr.dimension
    passes, _, entries = opr.slabs_info
    limit = 4 * entries + passes * (N + 4 * ((N + 31) // 32)) + (17 * N if scaling == 2 else 0)
    assert opr.build_slabs(slab_bytes=slab_bytes, max_bytes=limit)
    assert opr.slabs_info[0] == passes and opr.slabs_info[2] == entries
    x = O.complex_gaussian(N, 3)
    want = O.apply_rows(red, terms, x)
    for prec, dt, tol in (("fp64", torch.complex128, 1e-12), ("mixed", torch.complex64, 1e-5)):
        xd = torch.from_numpy(x).to(dt).cuda()
        y = torch.full_like(xd, float("nan"))
        E.mul_(y, opr, xd, precision=prec)
        assert relerr(y.cpu().numpy(), want) < tol
        E.apply_(y, opr, xd, precision=prec)
        assert relerr(y.cpu().numpy(), 2 * want) < tol
        yh = np.zeros(N, dtype=complex)
        E.mul_(yh, opr, x, precision=prec)
        assert relerr(yh, want) < tol
        # an infinite element reaches the rows that it reaches through the target table
        xi = xd.clone()
        xi[N // 3] = complex(float("inf"), 0.0)
        y0 = torch.empty_like(xi)
        E.mul_(y, opr, xi, precision=prec)
        opr.slab_use(prec, False)
        E.mul_(y0, opr, xi, precision=prec)
        opr.slab_use(prec, True)
        fin, fin0 = torch.isfinite(torch.view_as_real(y)).all(1), torch.isfinite(torch.view_as_real(y0)).all(1)
        assert torch.equal(fin, fin0) and not bool(fin0.all())


@pytest.mark.parametrize("scaling", [1, 2])
@pytest.mark.parametrize("slab_bytes", [1 << 20, 8192])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_infinite_element_with_characters(prec, slab_bytes, scaling):
    """Complex coefficients, padded and masked, unscaled and scaled tables."""
    import torch
    import edgpu as E
    opr, _, _ = _sector(E, (5, 4), 0, (1, 2), scaling, slab_bytes)
    dt = torch.complex128 if prec == "fp64" else torch.complex64
    x = torch.from_numpy(O.complex_gaussian(opr.dimension, 5)).to(dt).cuda()
    for col in (0, 1027, opr.dimension - 1):
        xi = x.clone()
        xi[col] = complex(float("inf"), 0.0)
        y, y0 = torch.empty_like(xi), torch.empty_like(xi)
        E.mul_(y, opr, xi, precision=prec)
        opr.slab_use(prec, False)
        E.mul_(y0, opr, xi, precision=prec)
        opr.slab_use(prec, True)
        fin, fin0 = torch.isfinite(torch.view_as_real(y)).all(1), torch.isfinite(torch.view_as_real(y0)).all(1)
        assert torch.equal(fin, fin0) and not bool(fin0.all()) and bool(fin0.any())
