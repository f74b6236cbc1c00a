"""The slab product of sectors around the sizes up to which four warps share a tile by place (600 and 1024 tiles of
in-order tables, 400 and 16384 of others in FP64), and coefficient tables below and above the size for it.  Products
repeated back to back, against the oracle's reduced product, 1e-12 in FP64 and 1e-5 in mixed precision (the
bounds of the slab product's other tests)."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_slab_steps import _sector, relerr

pytestmark = pytest.mark.gpu


def _check(opr, red, terms):
    import torch
    import edgpu as E
    x = O.complex_gaussian(opr.dimension, 7)
    want = O.apply_rows(red, terms, x)
    want2 = O.apply_rows(red, terms, want)
    for prec, dt, tol in (("fp64", torch.complex128, 1e-12), ("mixed", torch.complex64, 1e-5)):
        xd = torch.from_numpy(x).to(dt).cuda()
        y, z = torch.full_like(xd, float("nan")), torch.full_like(xd, float("nan"))
        for _ in range(20):
            E.mul_(y, opr, xd, precision=prec)
            E.mul_(z, opr, y, precision=prec)
        assert relerr(y.cpu().numpy(), want) < tol
        assert relerr(z.cpu().numpy(), want2) < 2 * tol
        E.apply_(y, opr, xd, precision=prec)
        assert relerr(y.cpu().numpy(), 2 * want) < tol


@pytest.mark.parametrize("scaling", [1, 2])
@pytest.mark.parametrize("shape,q,k", [((3, 1), 1, (1, 0)), ((14, 1), 0, (0, 0)), ((21, 1), 1, (2, 0)), ((22, 1), 0, (3, 0)),
                                       ((22, 1), 0, (0, 0)), ((23, 1), 1, (0, 0)), ((6, 4), 0, (0, 0)), ((6, 4), 0, (1, 2))])
def test_sizes(shape, q, k, scaling):
    import edgpu as E
    _check(*_sector(E, shape, q, k, scaling, 1 << 20))


@pytest.mark.parametrize("L,k", [(14, 0), (16, 3), (20, 3)])
def test_many_coefficients(L, k):
    """A coupling per bond: 14 to 20 amplitudes by characters and pairs of orbit sizes."""
    import edgpu as E
    from edgpu import lattice
    hs, _ = E.spin_half_system(L)
    rh = E.symmetry_reduce(E.represent(E.HilbertSpaceSector(hs, 0)), E.translation_symops(L, k))
    m, r, c, a, ids = lattice.heisenberg_coupled(hs, lattice.chain_bonds(L))
    J = 0.5 + np.random.default_rng(L).random(L)
    opr = E.OperatorRepresentation.from_terms(rh, m, r, c, a, coupling_ids=ids, couplings=J)
    maps, amps = O.translation_symops((L, 1), (k, 0))
    red = O.symmetry_reduce(O.popcount_basis(L, L // 2), *O.bit_layout(O.spin_half_sites(L)), maps, amps)
    terms = [(int(m[i]), int(r[i]), int(c[i]), complex(a[i]) * J[ids[i]]) for i in range(len(m))]
    assert opr.build_targets(1 << 30)
    for scaling in (1, 2):
        opr.slab_scaling(scaling)
        if opr.build_slabs(slab_bytes=1 << 20, max_bytes=1 << 30):
            _check(opr, red, terms)
        else:
            assert scaling == 1   # (more coefficients than an unscaled table holds)
