"""The multigrid level launches (mg_level.cu) against the cluster tail, which runs the same cycle
phase by phase from level 1 down: V-cycles equal bit for bit at the sizes where tiles end (tiles own
10, 12 or 14 cells a side; the last one may own one more), and multigrid-PCG on level 0's viscosity
planes converges as fast as at other sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def solver(nx, nz, precision, seed=0, **kw):
    from meeuuw_b200 import _lib
    from meeuuw_b200.stokes import StokesSolver
    box = _lib.box_of(nx, nz, 1.3, 1.0)
    g = torch.Generator(device="cuda").manual_seed(seed)
    fix = torch.zeros(2 * nz + 1, 2 * nx + 1, 2, dtype=torch.bool, device="cuda")
    fix[:, 0, 0] = fix[:, -1, 0] = True
    fix[0, :, 1] = fix[-1, :, 1] = True
    fix[0, :, 0] = True
    S = StokesSolver(box, fix.reshape(-1), precisions=(precision,), **kw)
    etaq = torch.exp(3.0 * torch.rand(nx * nz, 9, generator=g, device="cuda", dtype=torch.float64))
    S.set_viscosity(etaq, etaq.mean(1).contiguous())
    return S, g


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("degree", [1, 2])
@pytest.mark.parametrize("level1", [(3, 5), (9, 11), (10, 12), (13, 14), (20, 10), (21, 29), (26, 28), (30, 24)])
def test_vcycle_equals_cluster_tail(level1, degree, precision):
    nx, nz = 2 * level1[0], 2 * level1[1]
    out = []
    for tail in (0, 10 ** 6):
        S, g = solver(nx, nz, precision, cheb_degree=degree, tail_nel=tail)
        b = torch.randn(S.nv, generator=g, device="cuda", dtype=torch.float32 if precision == "f32" else torch.float64)
        out.append(S.vcycle(b, precision))
    assert torch.equal(out[0], out[1])


@pytest.mark.parametrize("precision,degree", [("f32", 2), ("f64", 1)])
@pytest.mark.parametrize("shape", [(2, 2), (9, 11), (10, 12), (14, 28), (25, 13), (48, 70)])
def test_solve_K_converges(shape, precision, degree):
    S, g = solver(*shape, precision, cheb_degree=degree)
    b = torch.randn(S.nv, generator=g, device="cuda", dtype=torch.float64)
    rtol = 1e-10 if precision == "f64" else 1e-4
    x, it, rr = S.solve_K(b, precision=precision, rtol=rtol, maxit=60)
    assert rr <= rtol and it < 60
    if precision == "f64":
        y, _ = S.apply(x)
        assert float((y - b).norm() / b.norm()) < 10 * rtol


@pytest.mark.parametrize("shape", [(2, 2), (3, 3), (4, 4), (3, 5), (2, 7), (2, 8)])
def test_coarsest_inverse(shape):
    """A hierarchy of one level is its dense inverse (50 ... 170 unknowns): K V(b) = b to FP64 rounding
    times the condition number (about 1e4 here)."""
    S, g = solver(*shape, "f64")
    assert S.levels("f64") == 1
    b = torch.randn(S.nv, generator=g, device="cuda", dtype=torch.float64)
    y, _ = S.apply(S.vcycle(b, "f64"))
    assert float((y - b).norm() / b.norm()) < 1e-10
