"""A solver's workspace is written in the order of the stream that uses it: created on a side stream over a
block that queued work still overwrites, or first used while a graph is recorded, it works as one created in
peace."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(38, 25), (32, 16)]                  # transfer tables, and none


def problem(nx, nz, precision):
    from test_gpu_mg_level import solver
    S, g = solver(nx, nz, precision)
    etaq = S._eta
    b = torch.randn(S.nv, generator=g, device="cuda", dtype=torch.float32 if precision == "f32" else torch.float64)
    return S, etaq, b


def use(S, etaq, b, precision):
    S.set_viscosity(etaq, etaq.mean(1).contiguous())
    x = S.vcycle(b, precision)
    y, it, rr = S.solve_K(b.double(), precision=precision, rtol=1e-4, maxit=60)
    return x, y, it


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("shape", SHAPES)
def test_recycled_block_with_queued_writes(shape, precision):
    from meeuuw_b200.stokes import StokesSolver
    A, etaq, b = problem(*shape, precision)
    want = use(A, etaq, b, precision)
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        block = torch.empty(A.work.numel(), dtype=torch.uint8, device="cuda")
        at = block.data_ptr()
        torch.cuda._sleep(20_000_000)            # some 10 ms, the block's write behind it
        block.fill_(0x7f)
        del block
        B = StokesSolver(A.box, A.fix, precisions=(precision,))
        assert B.work.data_ptr() == at
        got = use(B, etaq, b, precision)
        torch.cuda.synchronize()
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and got[2] == want[2]


@pytest.mark.parametrize("shape", SHAPES)
def test_first_use_recorded(shape):
    """A first use in a recording runs with the recording, as often as it is replayed."""
    from meeuuw_b200.stokes import StokesSolver
    A, etaq, b = problem(*shape, "f32")
    eta_e = etaq.mean(1).contiguous()
    want = A.vcycle(b, "f32")
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        B = StokesSolver(A.box, A.fix, precisions=("f32",))
        B.work.fill_(0x7f)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            B.set_viscosity(etaq, eta_e)
            x = B.vcycle(b, "f32")
        for _ in range(2):
            g.replay()
            s.synchronize()
            assert torch.equal(x, want)
