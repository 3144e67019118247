"""The coarse levels in one launch (mg_tail.cu) against the cluster tail, which runs the same cycle phase by
phase: equal bit for bit where the first level just fits a CTA's 384 threads (21 x 18 cells) and where it just
does not, on chains that are and are not nested, with a coarsest inverse that fits shared memory beside the
levels and one that does not."""
import pytest
import torch

from test_gpu_mg_level import solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("degree", [1, 2])
@pytest.mark.parametrize("level1,kw", [((16, 16), {}), ((20, 17), {}), ((20, 18), {}), ((47, 7), {}), ((48, 7), {}),
                                       ((13, 19), {}), ((8, 8), {}), ((4, 5), {}), ((12, 12), dict(coarse_dense_max=0)),
                                       ((40, 36), {}), ((75, 49), {})])
def test_vcycle_equals_cluster_tail(level1, kw, degree, precision):
    out = []
    for tail in (0, 10 ** 6):
        S, g = solver(2 * level1[0], 2 * level1[1], precision, cheb_degree=degree, tail_nel=tail, **kw)
        b = torch.randn(S.nv, generator=g, device="cuda", dtype=torch.float32 if precision == "f32" else torch.float64)
        out.append([S.vcycle(b, precision) for _ in range(2)])
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
