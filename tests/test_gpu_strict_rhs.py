"""The strict variant's right-hand side: the reference's own operations on its face fluxes, two IEEE
divides and a subtraction, to the bit."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bench,split,recon,ni,nj", [(11, 101, 253, 40, 32), (2, 103, 255, 37, 29), (13, 104, 0, 24, 51),
                                                     (5, 105, 0, 60, 15)])
def test_strict_rhs_is_the_divided_flux_difference(dense, bench, split, recon, ni, nj):
    c, cons, prim, x, y = dense.init_general(dense.config_default(ni=ni, nj=nj, benchmark=bench, splitting=split,
                                                                  recon=recon, cfl=0.5, strict=1))
    out = torch.empty((4, nj, ni), dtype=torch.float64, device="cuda")
    with dense.Solver(c) as s:
        s.upload(cons, prim, x, y)
        assert s.lib.dense_rhs_device(s.h, 1, ctypes.c_void_p(out.data_ptr()), None) == 0
        torch.cuda.synchronize()
        hx, he = s.fluxes()
    want = -(hx[1:] - hx[:-1]) / c.dx - ((he[1:] - he[:-1]) / c.dy).transpose(1, 0, 2)
    np.testing.assert_array_equal(out.cpu().numpy(), want.transpose(2, 1, 0))
