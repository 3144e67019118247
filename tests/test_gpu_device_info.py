"""The outcome of the last solve, read from the device, outlives the calls that are no solve: a residual of
another vector, a solve with K, the Schur residual of another pressure."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def other_calls(S, f, h):
    g = torch.Generator(device="cuda").manual_seed(3)
    V = torch.randn(S.nv, generator=g, device="cuda", dtype=torch.float64)
    P = torch.randn(S.np, generator=g, device="cuda", dtype=torch.float64)
    prec = "f64" if S.prm.precisions & 1 else "f32"
    yield lambda: S.residual(V, P, f, h)
    yield lambda: S.solve_K(V, precision=prec, rtol=1e-3, maxit=20)
    yield lambda: S.uzawa_residual(f, h, P, precision=prec)


@pytest.mark.parametrize("stokes", ["mixed", "f64"])
def test_recorded_step(stokes):
    from meeuuw_b200 import configs
    from meeuuw_b200.timestep import GPUModel
    m = GPUModel(configs.fk_convection(32, seed=5, Ra=1e5), stokes=stokes)
    m.step()
    m.capture_step()
    m.step()
    info = m.solver.device_info(m.tol)
    assert info["converged"] == 1 and info["outer_iters"] > 0 and info["inner_iters"] > 0
    for call in other_calls(m.solver, m.rhs_f, m.rhs_h):
        call()
        assert m.solver.device_info(m.tol) == info


@pytest.mark.parametrize("host_loops", [0, 1])
def test_solve(host_loops):
    from test_gpu_mg_level import solver
    S, g = solver(24, 18, "f32")
    f = torch.randn(S.nv, generator=g, device="cuda", dtype=torch.float64)
    f[S.fix.bool()] = 0.0
    h = torch.zeros(S.np, device="cuda", dtype=torch.float64)
    _, _, out = S.solve(f, h, precision="mixed", tol=1e-8, inner_rtol=2e-2, host_loops=host_loops)
    info = S.device_info(1e-8)
    assert info["converged"] == 1
    for k in ("outer_iters", "inner_iters", "refinements", "rel_residual", "initial_rel_residual"):
        assert info[k] == out[k], k
    for call in other_calls(S, f, h):
        call()
        assert S.device_info(1e-8) == info
