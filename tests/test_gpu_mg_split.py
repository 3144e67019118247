"""Large multigrid levels (above 65536 elements), whose downward half runs as two launches, against the cluster
tail running the same cycle from level 1 down: equal bit for bit, nested and not, at tile edges."""
import pytest
import torch

from test_gpu_mg_level import solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("level1", [(300, 240), (257, 257), (336, 196), (338, 195)])
def test_vcycle_equals_cluster_tail(level1, precision):
    out = []
    for tail in (0, 10 ** 6):
        S, g = solver(2 * level1[0], 2 * level1[1], precision, cheb_degree=2, tail_nel=tail)
        b = torch.randn(S.nv, generator=g, device="cuda", dtype=torch.float32 if precision == "f32" else torch.float64)
        out.append(S.vcycle(b, precision))
    assert torch.equal(out[0], out[1])
