"""symmetry_unreduce / symmetry_reduce through the ring search, the search directory and the rank tables:
chains of even and odd length (sizes with and without a specialised ring search), tori, a general group,
one-row and empty sectors, materialised and lazy parents, against the oracle's parent-table restatement
(1e-13 in complex128, 1e-6 in complex64: one rounded product per entry, sums of at most 16 terms)."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,q,k", [((4, 1), 0, (2, 0)), ((5, 1), 1, (1, 0)), ((8, 1), 8, (0, 0)), ((8, 1), 8, (1, 0)),
                                       ((12, 1), 0, (6, 0)), ((13, 1), 3, (5, 0)), ((16, 1), 2, (0, 0)),
                                       ((15, 1), 1, (4, 0)), ((3, 3), 1, (1, 2)), ((4, 4), 0, (2, 2)), ((6, 2), 2, (3, 1))])
@pytest.mark.parametrize("lazy", [False, True])
def test_against_tables(shape, q, k, lazy):
    import torch
    import edgpu as E
    n = shape[0] * shape[1]
    hs, _ = E.spin_half_system(n)
    rh = E.symmetry_reduce(E.represent(E.HilbertSpaceSector(hs, q), lazy=lazy), E.translation_symops(shape, k))
    sites = O.spin_half_sites(n)
    parent = O.hs_get_basis_list(sites, [(q,)])
    maps, amps = O.translation_symops(shape, k)
    red = O.symmetry_reduce(parent, *O.bit_layout(sites), maps, amps)
    rng = np.random.default_rng(n + q)
    small = rng.standard_normal(red.dim) + 1j * rng.standard_normal(red.dim)
    large = rng.standard_normal(parent.size) + 1j * rng.standard_normal(parent.size)
    want_l, want_s = O.unreduce(red, small), O.reduce_vector(red, large)
    for dt, tol in ((torch.complex128, 1e-13), (torch.complex64, 1e-6)):
        s, l = torch.from_numpy(small).to(dt).cuda(), torch.from_numpy(large).to(dt).cuda()
        torch.cuda.synchronize()
        for _ in range(2):   # the space's tables are built by the first call
            got = E.symmetry_unreduce(rh, s).cpu().numpy()
            assert np.max(np.abs(got - want_l), initial=0.0) < tol * max(1.0, np.max(np.abs(small), initial=0.0))
            got = E.symmetry_reduce(rh, l).cpu().numpy()
            assert np.max(np.abs(got - want_s), initial=0.0) < tol * 16 * np.max(np.abs(large))


@pytest.mark.parametrize("flip", [False, True])
def test_general_group(flip):
    """Translations times the global spin flip (and the translations alone, as site permutations listed in
    another order): the general path."""
    import torch
    import edgpu as E
    L = 10
    hs, _ = E.spin_half_system(L)
    tr = E.translation_symops(L, 0)
    ops = [(t, a) for t, a in tr] + ([(t * E.GlobalBitFlip(True), -a) for t, a in tr] if flip else [])
    if not flip:
        ops = [ops[0]] + ops[:0:-1]
    rh = E.symmetry_reduce(E.represent(E.HilbertSpaceSector(hs, 0)), ops)
    small = np.arange(1, rh.dimension + 1) * (1.0 + 0.5j)
    x = torch.from_numpy(small).cuda()
    torch.cuda.synchronize()
    large = E.symmetry_unreduce(rh, x)
    idx, amp = rh.basis_mapping_index, rh.basis_mapping_amplitude
    want = np.where(idx >= 0, amp * small[np.maximum(idx, 0)], 0)
    assert np.max(np.abs(large.cpu().numpy() - want)) < 1e-13 * np.max(np.abs(small))
    assert np.max(np.abs(E.symmetry_reduce(rh, large).cpu().numpy() - small)) < 1e-12 * np.max(np.abs(small))


@pytest.mark.parametrize("L,q", [(8, 2), (10, 2), (10, -4), (12, 0), (9, 1)])
@pytest.mark.parametrize("lazy", [False, True])
def test_flips_out_of_the_sector(L, q, lazy):
    """Translations times the spin flip on a sector that the flip leaves (all but 2Sz = 0): members of an orbit
    outside the parent have no entry of the large vector.  Against the sums written out (1e-13)."""
    import torch
    import edgpu as E
    hs, _ = E.spin_half_system(L)
    hsr = E.represent(E.HilbertSpaceSector(hs, q), lazy=lazy)
    full = (1 << L) - 1
    ops, elems = [], []
    for a, (t, chi) in enumerate(E.translation_symops(L, 1)):
        for f, par in ((False, 1), (True, -1)):
            ops.append((t * E.GlobalBitFlip(f) if f else t, chi * par))
            elems.append((list(t.map), full if f else 0, chi * par))
    rh = E.symmetry_reduce(hsr, ops)
    index = {int(b): i for i, b in enumerate(O.popcount_basis(L, (L - q) // 2))}
    large = O.complex_gaussian(len(index), 5)
    want = np.zeros(rh.dimension, dtype=complex)
    for r, rep in enumerate(int(b) for b in rh.basis_list):
        images = [(sum(((rep >> i) & 1) << m[i] for i in range(L)) ^ f, chi) for m, f, chi in elems]
        stab = sum(im == rep for im, _ in images)
        want[r] = sum(chi * large[index[im]] for im, chi in images if im in index) * np.sqrt(stab / len(elems)) / stab
    got = E.symmetry_reduce(rh, torch.from_numpy(large).cuda()).cpu().numpy()
    assert np.abs(got - want).max(initial=0.0) < 1e-13 * 2 * L * np.abs(large).max()


def test_tables_are_kept_once():
    """Sectors of one parent share its rank tables (32 MB at 44 bits), and symmetry_unreduce needs none."""
    import torch
    import edgpu as E
    L, q = 44, 40
    hs, _ = E.spin_half_system(L)
    hsr = E.represent(E.HilbertSpaceSector(hs, q))
    parent = O.popcount_basis(L, (L - q) // 2)
    sectors = [E.symmetry_reduce(hsr, E.translation_symops(L, k)) for k in range(6)]
    large = O.complex_gaussian(parent.size, 5)
    lt = torch.from_numpy(large).cuda()
    smalls = [E.random_state(s.dimension, 3, "fp64") for s in sectors]
    torch.cuda.synchronize()
    free = [torch.cuda.mem_get_info()[0]]
    for s, v in zip(sectors, smalls):
        E.symmetry_unreduce(s, v)
    free.append(torch.cuda.mem_get_info()[0])
    for k, s in enumerate(sectors):
        maps, amps = O.translation_symops((L, 1), (k, 0))
        red = O.symmetry_reduce(parent, *O.bit_layout(O.spin_half_sites(L)), maps, amps)
        got = E.symmetry_reduce(s, lt).cpu().numpy()
        assert np.abs(got - O.reduce_vector(red, large)).max() < 1e-13 * L * np.abs(large).max()
    free.append(torch.cuda.mem_get_info()[0])
    assert free[0] - free[1] < 16 << 20
    assert free[1] - free[2] < (32 << 20) + (16 << 20)
