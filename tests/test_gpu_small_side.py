"""The fast sweeps on the small side of a jump: a gas 1e8 times as thin beside a dense one at the same
temperature (and so of the same wave speeds), whose faces two and three cells from the jump have it in
their stencils. The right-hand side there, fast against strict, relative to the thin side: each face flux
is some fifty roundings of that size, so 1e-13."""
import importlib

import numpy as np
import pytest
import torch

import torch_step

pytestmark = pytest.mark.gpu

THIN = 1e-8


def state(c, axis, every_field=False):
    """Dense in the first half along the axis, thin in the second; smooth variations of a few percent.
    every_field: a transverse velocity that jumps too, and a fast stream far from the jumps, so that
    the domain's wave speed is none of a face's own: every characteristic field jumps by its level."""
    X, Y = np.meshgrid(np.arange(c.ni + 8) - 4 + 0.5, np.arange(c.nj + 8) - 4 + 0.5, indexing="ij")
    k = 2 * np.pi / np.array([c.ni, c.nj])
    rho = 1 + 0.05 * np.sin(k[0] * X) * np.cos(k[1] * Y)
    u, v = 0.4 + 0.1 * np.cos(k[0] * X + k[1] * Y), -0.3 + 0.1 * np.sin(2 * k[0] * X - k[1] * Y)
    p = 1 + 0.04 * np.cos(k[0] * X - k[1] * Y)
    thin = np.where((X if axis == 0 else Y) % (c.ni if axis == 0 else c.nj) < (c.ni if axis == 0 else c.nj) // 2, 1.0, THIN)
    rho, p = rho * thin, p * thin
    if every_field:
        n, Z = (c.ni, X) if axis == 0 else (c.nj, Y)
        stream = 2.0 * (np.abs(Z % n - n / 4) < 3)
        shear = np.where(thin < 1, 1.0, 0.0)
        u, v = (u + stream, v + shear) if axis == 0 else (u + shear, v + stream)
    cons = np.zeros(rho.shape + (4,), order="F")
    cons[..., 0], cons[..., 1], cons[..., 2] = rho, rho * u, rho * v
    cons[..., 3] = p / (c.gamma - 1.0) + 0.5 * rho * (u * u + v * v)
    return cons


def right_hand_sides(dense, split, recon, axis, n, every_field=False):
    """(strict, fast, configuration) in the rows two to four cells from the jumps."""
    ops = importlib.import_module("2dense_gb300.torch_ops")
    L, c = [], None
    for strict in (1, 0):
        c = dense.init_general(dense.config_default(ni=n, nj=n + 8, benchmark=11, splitting=split, recon=recon,
                                                    cfl=0.5, strict=strict))[0]
        u = ops.padded_state(state(c, axis, every_field))
        L.append(torch.ops.dense2d.rhs(u, ops.config_tensor(c)).cpu().numpy())
    m = n if axis == 0 else n + 8
    rows = [m // 2 + 1, m // 2 + 2, m // 2 + 3, m - 4, m - 3, m - 2]
    return (*(np.take(x, rows, axis=2 if axis == 0 else 1) for x in L), c)


@pytest.mark.parametrize("n", [40, 400])  # the small grids' tiles and the others
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("split,recon", [(101, 253), (101, 255), (102, 255), (103, 253), (103, 255)])
def test_thin_side(dense, split, recon, axis, n):
    strict, fast, c = right_hand_sides(dense, split, recon, axis, n)
    size = THIN * 3.0 / min(c.dx, c.dy)  # a thin-side flux over the cell's size
    assert np.abs(strict).max() < 100 * size  # (the dense side is not in these)
    assert np.abs(fast - strict).max() <= 1e-13 * size


@pytest.mark.parametrize("n", [40, 400])
@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("split", [104, 105])
def test_thin_side_characteristic(dense, split, axis, n):
    """The characteristic schemes: through the weights a share of the dense side, (ss / jump^2)^2 of it,
    reaches the thin side's fields, so the size is that of the largest value there. The fields' jumps
    are good to some fifty roundings, the share to four times that, 5e-14: 1e-12."""
    strict, fast, c = right_hand_sides(dense, split, 0, axis, n, every_field=True)
    size = max(np.abs(strict).max(), THIN * 3.0 / min(c.dx, c.dy))
    assert size < 1e-4 * 3.0 / min(c.dx, c.dy)
    assert np.abs(fast - strict).max() <= 1e-12 * size


@pytest.mark.parametrize("axis", [0, 1])
@pytest.mark.parametrize("split,recon", [(101, 253), (101, 255), (103, 255), (104, 0), (105, 0)])
def test_thin_side_adjoint(dense, split, recon, axis):
    """The transposed Jacobian for weights on thin cells three and more from the jumps, at the thin cells
    beside those, against autograd through the PyTorch step; entries there are of order one whatever
    the density, so a field's value is needed to its own digits. 1e-10 as on smooth states."""
    adjoint = importlib.import_module("2dense_gb300.adjoint")
    c = dense.init_general(dense.config_default(ni=40, nj=48, benchmark=11, splitting=split, recon=recon, cfl=0.5))[0]
    U = torch.from_numpy(np.ascontiguousarray(state(c, axis, True)[4:-4, 4:-4].transpose(2, 1, 0))).cuda()
    m, dim = (c.ni, 2) if axis == 0 else (c.nj, 1)
    rows = torch.arange(m // 2 + 2, m - 2, device="cuda")
    v = torch.zeros_like(U)
    w = torch.randn(U.shape, generator=torch.Generator().manual_seed(7), dtype=torch.float64).cuda()
    v.index_copy_(dim, rows, w.index_select(dim, rows))
    with adjoint.Adjoint(c) as adj:
        out, _ = adj.rhs_vjp(U, v)
    Ut = U.clone().requires_grad_(True)
    (ref,) = torch.autograd.grad(torch_step.rhs(Ut, c.gamma, c.dx, c.dy, recon, split, delta=c.delta), Ut, v)
    out, ref = (x.index_select(dim, rows) for x in (out, ref))
    assert float((out - ref).abs().max() / ref.abs().max()) < 1e-10
