"""Enumeration, representatives, orbit sizes and the search directory where their kernels divide the work:
tables of less than one group, of a group's last lane and of several blocks; rings with and without an
unrolled rotation search, of two-bit sites, and of lengths with one, two and no prime factor below them; tori,
a general group, materialised and lazy parents; tables with crowded, single and wide gaps between keys.
Whole numbers: everything is compared exactly."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def check_lookup(space, table, rng, nbits):
    miss = rng.integers(0, 1 << nbits, 500, dtype=np.uint64)
    q = np.concatenate([table[rng.integers(0, len(table), 500)], miss]) if len(table) else miss
    at = np.searchsorted(table, q)
    hit = at < len(table)
    hit[hit] = table[at[hit]] == q[hit]
    assert np.array_equal(space.lookup(q), np.where(hit, at, -1))


@pytest.mark.parametrize("shape,q,k", [((2, 1), 0, (0, 0)), ((3, 1), 1, (1, 0)), ((7, 1), 1, (0, 0)), ((8, 1), 0, (4, 0)),
                                       ((9, 1), 1, (3, 0)), ((12, 1), 0, (0, 0)), ((12, 1), 0, (5, 0)),
                                       ((13, 1), 13, (0, 0)), ((13, 1), 13, (1, 0)), ((16, 1), 0, (8, 0)),
                                       ((18, 1), 0, (6, 0)), ((3, 3), 1, (1, 1)), ((4, 4), 0, (0, 2)), ((6, 2), 0, (2, 1))])
@pytest.mark.parametrize("lazy", [False, True])
def test_sectors(shape, q, k, lazy):
    import edgpu as E
    n = shape[0] * shape[1]
    hs, _ = E.spin_half_system(n)
    hsr = E.represent(E.HilbertSpaceSector(hs, q), lazy=lazy)
    sites = O.spin_half_sites(n)
    parent = O.hs_get_basis_list(sites, [(q,)])
    rng = np.random.default_rng(n)
    if not lazy:
        assert np.array_equal(hsr.basis_list, parent)
        check_lookup(hsr, parent, rng, n)
    rh = E.symmetry_reduce(hsr, E.translation_symops(shape, k))
    maps, amps = O.translation_symops(shape, k)
    red = O.symmetry_reduce(parent, *O.bit_layout(sites), maps, amps)
    assert np.array_equal(rh.basis_list, red.basis_list)
    table = np.asarray(red.basis_list, dtype=np.uint64)
    check_lookup(rh, table, rng, n)
    off, bw = O.bit_layout(sites)
    orbit = [len({sum(((int(s) >> i) & 1) << int(m[i]) for i in range(n)) for m in maps}) for s in table]
    assert np.array_equal(rh.orbit_sizes(), orbit)


@pytest.mark.parametrize("n_sites,d", [(5, 3), (6, 4), (7, 3)])
def test_ring_of_wide_sites(n_sites, d):
    """Two bits per site: the ring rotates by two bits at a time."""
    import edgpu as E
    site = E.Site([E.State(f"s{i}", i) for i in range(d)])
    hs = E.HilbertSpace([site] * n_sites)
    hsr = E.represent(hs)
    for k in (0, 1):
        rh = E.symmetry_reduce(hsr, E.translation_symops(n_sites, k))
        ops = E.translation_symops(n_sites, k)
        basis = np.asarray(hsr.basis_list)
        mask = (1 << (2 * n_sites)) - 1
        rot = lambda s, a: ((s << (2 * a)) | (s >> (2 * (n_sites - a)))) & mask
        keep, size = [], []
        for s in (int(v) for v in basis):
            images = [rot(s, a) for a in range(n_sites)]
            stab = [a for a in range(n_sites) if images[a] == s]
            if min(images) == s and all(a * k % n_sites == 0 for a in stab):
                keep.append(s)
                size.append(n_sites // len(stab))
        assert np.array_equal(rh.basis_list, np.array(keep, dtype=np.uint64))
        assert np.array_equal(rh.orbit_sizes(), size)
        check_lookup(rh, np.array(keep, dtype=np.uint64), np.random.default_rng(d), 2 * n_sites)


@pytest.mark.parametrize("n_keys", [1, 2, 23, 24, 25, 192, 193, 5000, 70000])
@pytest.mark.parametrize("kind", ["dense", "spread", "clusters", "one_far"])
@pytest.mark.parametrize("n_sites", [30, 50])
def test_directory_of_given_bases(n_keys, kind, n_sites):
    """Hit and miss lookups, and the share of keys that their bucket answers (recounted from the table)."""
    import edgpu as E
    rng = np.random.default_rng(n_keys + n_sites)
    if kind == "dense":
        b = np.arange(n_keys, dtype=np.uint64)
    elif kind == "spread":
        b = np.unique(rng.integers(0, 1 << n_sites, n_keys, dtype=np.uint64))
    elif kind == "clusters":
        b = np.unique((rng.integers(0, 1 << (n_sites - 14), 1 + n_keys // 6000, dtype=np.uint64)[:, None] << np.uint64(14))
                      + np.arange(6000, dtype=np.uint64)[None, :])[:n_keys]
    else:
        b = np.concatenate([np.arange(n_keys, dtype=np.uint64), [np.uint64((1 << n_sites) - 1)]])
    hs, _ = E.spin_half_system(n_sites)
    sp = E.represent(hs, b)
    assert np.array_equal(sp.basis_list, b)
    check_lookup(sp, b, rng, n_sites)
    st = E.search_stats(sp)
    shift, K = st["shift"], st["inline_per_bucket"]
    _, inv, cnt = np.unique(b >> np.uint64(shift), return_inverse=True, return_counts=True)
    assert st["inline_fraction"] == pytest.approx(np.sum(cnt[inv] <= K) / len(b), abs=1e-12)
