"""The mass-matrix preconditioner node by node: after one Schur iteration from zero pressure the pressure is a
multiple of the first direction, the Chebyshev steps for M w = G^T K^-1 f less its mean, less their own mean;
those steps written out, for step counts that fill a launch, leave a remainder and take two or three launches, on
meshes at the edges of the nodes that a tile owns (22, 20 and more a side)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

f64 = torch.float64


def mass(w, x, hx, hz):
    """M_w x of the bilinear elements weighted by w (nelz, nelx); x (nelz + 1, nelx + 1)."""
    m = torch.tensor([[4, 2, 1, 2], [2, 4, 2, 1], [1, 2, 4, 2], [2, 1, 2, 4]], dtype=f64, device="cuda") * (hx * hz / 36)
    c = [x[:-1, :-1], x[:-1, 1:], x[1:, 1:], x[1:, :-1]]
    y = torch.zeros_like(x)
    for k, (a, b) in enumerate(((0, 0), (0, 1), (1, 1), (1, 0))):
        y[a:a + w.shape[0], b:b + w.shape[1]] += w * sum(m[k, j] * c[j] for j in range(4))
    return y


def chebyshev(w, r, hx, hz, steps):
    lo, hi = 0.25 / 1.02, 2.25 * 1.02
    theta, delta = (hi + lo) / 2, (hi - lo) / 2
    sigma = theta / delta
    D = torch.zeros_like(r)
    for a in (0, 1):
        for b in (0, 1):
            D[a:a + w.shape[0], b:b + w.shape[1]] += w * (4 * hx * hz / 36)
    d = r / (theta * D)
    x, rho = d.clone(), 1 / sigma
    for _ in range(steps - 1):
        new = 1 / (2 * sigma - rho)
        d = new * rho * d + 2 * new / delta * (r - mass(w, x, hx, hz)) / D
        x, rho = x + d, new
    return x


@pytest.mark.parametrize("scheme", ["cd_u_eta", "uzawa3"])
@pytest.mark.parametrize("nx,nz", [(21, 22), (22, 43), (43, 19), (20, 40), (64, 31)])
@pytest.mark.parametrize("steps", [1, 2, 5, 6, 7, 12, 13])
def test_first_direction(nx, nz, steps, scheme):
    """The inner solve is run beside it with the same iterates, so that only the roundings of some twenty steps
    and of the sums differ: 1e-10 of the largest value."""
    from meeuuw_b200 import _lib
    from meeuuw_b200.stokes import StokesSolver
    box = _lib.box_of(nx, nz, 1.3, 1.0)
    g = torch.Generator(device="cuda").manual_seed(nx + nz)
    fix = torch.zeros(2 * nz + 1, 2 * nx + 1, 2, dtype=torch.bool, device="cuda")
    fix[:, 0, 0] = fix[:, -1, 0] = True
    fix[0, :, 1] = fix[-1, :, 1] = True
    S = StokesSolver(box, fix.reshape(-1), precisions=("f64",))
    eta = torch.exp(3.0 * torch.rand(nx * nz, generator=g, device="cuda", dtype=f64))
    S.set_viscosity(eta[:, None].expand(-1, 9).contiguous(), eta)
    f = torch.randn(S.nv, generator=g, device="cuda", dtype=f64)
    f[fix.reshape(-1)] = 0.0
    h = torch.zeros(S.np, device="cuda", dtype=f64)
    _, P, _ = S.solve(f, h, scheme=scheme, precision="f64", tol=1e-14, inner_rtol=1e-12, max_inner=100, max_outer=1,
                      mass_iters=steps)
    V, _, _ = S.solve_K(f, precision="f64", rtol=1e-12, maxit=100)
    r = S.div(V)
    r = (r - r.mean()).view(nz + 1, nx + 1)
    w = (1 / eta if scheme == "cd_u_eta" else torch.ones_like(eta)).view(nz, nx)
    d = chebyshev(w, r, box.hx, box.hz, steps).reshape(-1)
    d = d - d.mean()
    alpha = float((P * d).sum() / (d * d).sum())
    assert alpha > 0
    assert float((P - alpha * d).abs().max()) < 1e-10 * float(P.abs().max())
