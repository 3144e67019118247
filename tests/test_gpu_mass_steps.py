"""The mass-matrix preconditioner of the Schur iteration (launches of at most six Chebyshev steps on tiles of
32 x 32 pressure nodes) against the cluster solve, which takes the same steps one at a time through global
memory: step counts that fill a launch, leave a remainder, take two or three launches; meshes at the edges of
the owned 22, 20 and fewer nodes a side.  Bounds as between the two solvers elsewhere: both reach the
tolerance, iteration counts within two, velocities within 1e-6 in norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(21, 22), (22, 43), (40, 24), (64, 19)])
@pytest.mark.parametrize("steps", [1, 5, 6, 7, 12, 13])
def test_mass_steps_match_cluster_solve(nx, nz, steps):
    from meeuuw_b200 import _lib
    from meeuuw_b200.stokes import StokesEnsembleSolve, StokesSolver
    box = _lib.box_of(nx, nz, 1.3, 1.0)
    g = torch.Generator(device="cuda").manual_seed(nx + nz)
    fix = torch.zeros(2 * nz + 1, 2 * nx + 1, 2, dtype=torch.bool, device="cuda")
    fix[:, 0, 0] = fix[:, -1, 0] = True
    fix[0, :, 1] = fix[-1, :, 1] = True
    S = StokesSolver(box, fix.reshape(-1))
    etaq = torch.exp(3.0 * torch.rand(nx * nz, 1, generator=g, device="cuda", dtype=torch.float64)).expand(-1, 9).contiguous()
    S.set_viscosity(etaq, etaq[:, 0].contiguous())
    f = torch.randn(S.nv, generator=g, device="cuda", dtype=torch.float64)
    f[fix.reshape(-1)] = 0.0
    h = torch.zeros(S.np, device="cuda", dtype=torch.float64)
    kw = dict(scheme="cd_u_eta", tol=1e-8, mass_iters=steps, inner_rtol=1e-2, max_outer=200)
    V, P, info = S.solve(f, h, precision="mixed", **kw)
    assert info["converged"] == 1
    Vc, Pc = torch.zeros_like(V), torch.zeros_like(P)
    S.prepare("mixed")
    StokesEnsembleSolve([S], [f], [h], [Vc], [Pc]).solve(use_guess=False, **kw)
    torch.cuda.synchronize()
    other = S.device_info(1e-8)
    assert other["converged"] == 1
    assert abs(info["outer_iters"] - other["outer_iters"]) <= 2
    assert float((V - Vc).norm() / V.norm()) < 1e-6
