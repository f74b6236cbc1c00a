"""A product captured into the caller's CUDA graph reads the coupling values of the time it is replayed:
set_couplings rewrites the operator's tables in place.  FP64 to 1e-12 and mixed precision to 1e-5 of the
oracle, as the products' other tests."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

L = 12


def _problem(E, path):
    """The space, prepared for the path, and the oracle's tables of it."""
    from edgpu import lattice
    hs, _ = E.spin_half_system(L)
    hsr = E.represent(E.HilbertSpaceSector(hs, 0))
    sites = O.spin_half_sites(L)
    parent = O.hs_get_basis_list(sites, [(0,)])
    terms = lattice.heisenberg_coupled(hs, lattice.chain_bonds(L))
    if path == "full":
        return hsr, parent, terms
    rh = E.symmetry_reduce(hsr, E.translation_symops(L, 3 if path == "momentum" else 0))
    maps, amps = O.translation_symops((L, 1), (3 if path == "momentum" else 0, 0))
    return rh, O.symmetry_reduce(parent, *O.bit_layout(sites), maps, amps), terms


def _prepare(opr, path):
    if path == "map":
        assert opr.space.build_map()
    if path in ("table", "slab"):
        assert opr.build_targets(1 << 28)
    if path == "slab":
        assert opr.build_slabs(1 << 20, 1 << 28)


def _check_replays(E, opr, ora, ids, m, r, c, a, settings, prec):
    import torch
    n = opr.dimension
    xh = O.complex_gaussian(n, 3)
    x = torch.from_numpy(xh).cuda().to(torch.complex128 if prec == "fp64" else torch.complex64)
    y = torch.empty_like(x)
    E.mul_(y, opr, x, precision=prec)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        E.mul_(y, opr, x, precision=prec)
    for J in settings:
        opr.set_couplings(J)
        y.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        t = [(int(m[i]), int(r[i]), int(c[i]), complex(a[i]) * J[ids[i]]) for i in range(len(m))]
        want = O.apply_rows(ora, t, xh)
        got = y.cpu().numpy()
        assert np.linalg.norm(got - want) <= (1e-12 if prec == "fp64" else 1e-5) * np.linalg.norm(want), J


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("per_bond", [False, True])
@pytest.mark.parametrize("path", ["full", "direct", "map", "table", "slab", "momentum"])
def test_replay_after_new_couplings(path, per_bond, prec):
    import edgpu as E
    space, ora, (m, r, c, a, ids) = _problem(E, path)
    if not per_bond:
        ids = np.zeros_like(ids)
    n_c = int(ids.max()) + 1
    opr = E.OperatorRepresentation.from_terms(space, m, r, c, a, coupling_ids=ids, couplings=np.ones(n_c))
    _prepare(opr, path)
    rng = np.random.default_rng(1)
    settings = [np.full(n_c, 0.7), 0.5 + rng.random(n_c), np.full(n_c, -1.3), np.ones(n_c)]
    _check_replays(E, opr, ora, ids, m, r, c, a, settings, prec)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("path,span", [(p, s) for p in ("full", "direct", "map", "table", "momentum") for s in (1, 2)] +
                                      [("slab", 2)])
def test_replay_after_an_imaginary_coupling(path, span, prec):
    """A Dzyaloshinskii-Moriya term (imaginary amplitudes) whose coupling is 0 at the capture, on the bonds of
    the other coupling or on bonds of its own (a slab table needs the latter)."""
    import edgpu as E
    from edgpu import lattice
    from edgpu.operators import pauli_matrix, simplify
    space, ora, (m, r, c, a, ids) = _problem(E, path)
    hs, _ = E.spin_half_system(L)
    m, r, c, a = (list(v) for v in (m, r, c, a))
    ids = [0] * len(m)
    for i, j in [(i, (i + span) % L) for i in range(L)]:
        t = simplify(0.25 * (pauli_matrix(hs, i, "x") * pauli_matrix(hs, j, "y") +
                             (-1.0) * (pauli_matrix(hs, i, "y") * pauli_matrix(hs, j, "x"))))
        for p in t.terms:
            m.append(p.bitmask), r.append(p.bitrow), c.append(p.bitcol), a.append(p.amplitude), ids.append(1)
    m, r, c = (np.array(v, dtype=np.uint64) for v in (m, r, c))
    a, ids = np.array(a, dtype=complex), np.array(ids, dtype=np.int32)
    assert np.abs(a[ids == 1].imag).min() > 0
    opr = E.OperatorRepresentation.from_terms(space, m, r, c, a, coupling_ids=ids, couplings=[1.0, 0.0])
    _prepare(opr, path)
    _check_replays(E, opr, ora, ids, m, r, c, a, np.array([[1.0, 0.4], [0.6, 0.0], [0.6, -0.8]]), prec)
