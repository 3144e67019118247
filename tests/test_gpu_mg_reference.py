"""A V-cycle's finest level against the same steps written out with the public operator, transfers and the next
level's own V-cycle: smoothing, residual and restriction in one launch (up to 65536 elements) and in two (above),
nested and not, at tile edges, with nine viscosities an element."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

f64 = torch.float64


def build(nx, nz, etaq, precision):
    from meeuuw_b200 import _lib
    from meeuuw_b200.stokes import StokesSolver
    fix = torch.zeros(2 * nz + 1, 2 * nx + 1, 2, dtype=torch.bool, device="cuda")
    fix[:, 0, 0] = fix[:, -1, 0] = True
    fix[0, :, 1] = fix[-1, :, 1] = True
    fix[0, :, 0] = True
    S = StokesSolver(_lib.box_of(nx, nz, 1.3, 1.0), fix.reshape(-1), precisions=(precision,), cheb_degree=2)
    S.set_viscosity(etaq, etaq.mean(1).contiguous())
    return S


def diagonal(S, etaq):
    """diag(K) from the Gauss points (build_matrix_stokes.py:140), summed on the nodes."""
    from meeuuw_b200 import fe_tables
    t = {k: torch.as_tensor(v, dtype=f64, device="cuda") for k, v in fe_tables.host_tables().items()}
    b = S.box
    e = etaq * (t["weightq"] * (b.hx * b.hz / 4))
    B, Z = 2 / b.hx * t["dNdr_V"], 2 / b.hz * t["dNdt_V"]
    el = torch.stack([e @ (2 * B * B + Z * Z), e @ (2 * Z * Z + B * B)], 2).view(b.nelz, b.nelx, 9, 2)
    at = [(0, 0), (0, 2), (2, 2), (2, 0), (0, 1), (1, 2), (2, 1), (1, 0), (1, 1)]      # (dz, dx) of local node k
    d = torch.zeros(2 * b.nelz + 1, 2 * b.nelx + 1, 2, dtype=f64, device="cuda")
    for k, (dz, dx) in enumerate(at):
        d[dz:dz + 2 * b.nelz:2, dx:dx + 2 * b.nelx:2] += el[:, :, k]
    return d.reshape(-1)


def vcycle_by_steps(S, C, etaq, b, precision):
    dt = b.dtype
    K = lambda x: S.apply(x, precision=precision)[0]
    D = diagonal(S, etaq).to(dt)
    v = (1.0 + 0.5 * torch.sin(0.7 * torch.arange(S.nv, dtype=f64, device="cuda"))).to(dt)
    for _ in range(S.prm.power_iters):
        v = K((v.double() / v.double().norm()).to(dt)) / D
    lmax = float(v.double().norm()) * S.prm.cheb_safety
    lmin = lmax / S.prm.cheb_ratio
    theta, delta = (lmax + lmin) / 2, (lmax - lmin) / 2
    sigma = theta / delta
    rho = 1 / (2 * sigma - 1 / sigma)
    c = [(0.0, 1 / theta), (rho / sigma, 2 * rho / delta)]
    d = c[0][1] * b / D                                     # from zero, then one step
    x = d.clone()
    d = c[1][0] * d + c[1][1] * (b - K(x)) / D
    x = x + d
    bc = S.restrict(0, b - K(x), precision)
    x = x + S.prolong(0, C.vcycle(bc, precision), precision)
    d = c[0][1] * (b - K(x)) / D
    x = x + d
    return x + c[1][0] * d + c[1][1] * (b - K(x)) / D


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("shape", [(24, 20), (26, 28), (256, 256), (258, 256), (300, 240), (264, 250), (288, 252),
                                   (27, 21), (257, 257), (335, 197), (261, 255), (290, 227), (258, 257)])
def test_finest_level(shape, precision):
    """Within rounding: the residual's is some ten products of relative size 2^-24 (2^-53), the cycle's answer to it
    like its answer to b, and the intervals agree as far as the sums of the power iterations: 1e-4 (1e-10) of the
    largest value, where a lost halo is 1e-2 and more."""
    nx, nz = shape
    cx, cz = (nx + 1) // 2, (nz + 1) // 2
    g = torch.Generator(device="cuda").manual_seed(nx)
    if nx % 2 == 0 and nz % 2 == 0:                         # a coarse element's viscosity: the mean of its 36 values
        etaq = torch.exp(3.0 * torch.rand(nx * nz, 9, generator=g, device="cuda", dtype=f64))
        own = etaq.float().double() if precision == "f32" else etaq
        coarse = own.view(cz, 2, cx, 2, 9).mean((1, 3, 4)).reshape(-1, 1).expand(-1, 9).contiguous()
    else:
        etaq = torch.full((nx * nz, 9), 2.5, dtype=f64, device="cuda")
        coarse = torch.full((cx * cz, 9), 2.5, dtype=f64, device="cuda")
    S, C = build(nx, nz, etaq, precision), build(cx, cz, coarse, precision)
    assert S.level_shape(1, precision) == (cx, cz)
    assert [S.level_shape(l + 1, precision) for l in range(C.levels(precision))] == \
        [C.level_shape(l, precision) for l in range(C.levels(precision))]
    b = torch.randn(S.nv, generator=g, device="cuda", dtype=torch.float32 if precision == "f32" else f64)
    got, want = S.vcycle(b, precision), vcycle_by_steps(S, C, etaq, b, precision)
    bound = 1e-4 if precision == "f32" else 1e-10
    assert float((got - want).abs().max()) < bound * float(want.abs().max())
