"""The slab product of sectors on either side of the size up to which several warps share a tile of 32 rows
(400 tiles): by-bond and in-order tables, real and complex momenta, one and many passes, products repeated
back to back (each launch may start before the one before it has ended).  Against the oracle's reduced
product, 1e-12 in FP64 and 1e-5 in mixed precision (the bounds of the slab product's other tests)."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_slab_steps import _sector, relerr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slab_bytes", [1 << 20, 16384])
@pytest.mark.parametrize("shape,q,k", [((2, 1), 0, (0, 0)), ((4, 4), 0, (0, 0)), ((4, 4), 2, (1, 0)), ((5, 4), 0, (2, 1)),
                                       ((7, 3), 1, (0, 0)), ((7, 3), 1, (1, 0)), ((20, 1), 0, (0, 0)), ((21, 1), 1, (2, 0))])
def test_split(shape, q, k, slab_bytes):
    import torch
    import edgpu as E
    opr, red, terms = _sector(E, shape, q, k, 1, slab_bytes)
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
