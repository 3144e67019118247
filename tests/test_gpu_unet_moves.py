"""The network's data-movement kernels on the shapes they branch on -- channel counts that are not a
multiple of a vector, images narrower and wider than a tile, padded and unaligned leading dimensions --
against plain torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
bf16 = torch.bfloat16


def entry(name, *args):
    import meeuuw_b200.unet  # noqa: F401  (registers the entry points)
    from meeuuw_b200._lib import call, ptr, stream_ptr
    call(name, *[ptr(a) if isinstance(a, torch.Tensor) else a for a in args], stream_ptr())


def at(shape, dtype, offset):
    n = 1
    for k in shape:
        n *= k
    return torch.zeros(n + offset, dtype=dtype, device="cuda")[offset:].view(shape)


def patches(X, Kp):
    B, H, W, C = X.shape
    P = torch.zeros(B, H + 2, W + 2, C, dtype=X.dtype, device="cuda")
    P[:, 1:-1, 1:-1] = X
    cols = [P[:, 1 + dy:1 + dy + H, 1 + dx:1 + dx + W].reshape(-1, C) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    out = torch.zeros(B * H * W, Kp, dtype=X.dtype, device="cuda")
    out[:, :9 * C] = torch.cat(cols, 1)
    return out


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("B,H,W,C", [(1, 8, 8, 2), (2, 24, 40, 5), (3, 16, 8, 32), (1, 5, 7, 33), (1, 8, 136, 96)])
def test_im2col(B, H, W, C, offset):
    Kp, M = -(-9 * C // 64) * 64, B * H * W
    g = torch.Generator(device="cuda").manual_seed(1)
    X = at((B, H, W, C), bf16, offset)
    X.copy_(torch.randn(B, H, W, C, generator=g, device="cuda"))
    want = patches(X, Kp)
    col = at((M, Kp), bf16, offset)
    entry("mw_unet_im2col", B, H, W, C, Kp, 0, 0, X, col)
    assert torch.equal(col, want)
    for ldT in (M, -(-M // 64) * 64 + 64, M + 3):
        colT = at((Kp, ldT), bf16, offset)
        colT.fill_(7.0)
        entry("mw_unet_im2col", B, H, W, C, Kp, 1, ldT, X, colT)
        assert torch.equal(colT[:, :M].T, want) and bool((colT[:, M:] == 0).all())


@pytest.mark.parametrize("M,C,relu", [(1, 1, 1), (100, 5, 0), (4099, 32, 1), (130, 96, 1), (640, 40, 1)])
def test_relu_grad_and_column_sums(M, C, relu):
    g = torch.Generator(device="cuda").manual_seed(2)
    dA = torch.randn(M, C, generator=g, device="cuda")
    A = torch.randn(M, C, generator=g, device="cuda").to(bf16)
    ldT = M + 5
    dZ, dZT, dZ32 = at((M, C), bf16, 0), at((C, ldT), bf16, 0), at((M, C), torch.float32, 0)
    dZT.fill_(3.0)
    entry("mw_unet_relu_grad", M, C, relu, ldT, dA, A, dZ, dZT, dZ32)
    want = torch.where(A.float() > 0, dA, torch.zeros_like(dA)) if relu else dA
    assert torch.equal(dZ32, want) and torch.equal(dZ, want.to(bf16))
    assert torch.equal(dZT[:, :M].T, want.to(bf16)) and bool((dZT[:, M:] == 3.0).all())
    s = torch.empty(C, device="cuda")
    entry("mw_unet_colsum", M, C, dZ32, s)
    exact = dZ32.double().sum(0)
    assert float((s.double() - exact).abs().max()) <= 2.0 ** -23 * float(exact.abs().max()) + 1e-30


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("C,Ctot,c0", [(32, 96, 64), (8, 24, 16), (5, 13, 6), (4, 12, 8)])
def test_pool_upsample_slices(C, Ctot, c0, offset):
    B, h, w = 2, 6, 10
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=g, device="cuda")
    X = at((B, h, w, C), bf16, offset)
    X.copy_(rnd(B, h, w, C))
    Y = at((B, 2 * h, 2 * w, Ctot), bf16, offset)
    entry("mw_unet_upsample2_into", B, h, w, C, Ctot, c0, X, Y)
    assert torch.equal(Y[..., c0:c0 + C], X.repeat_interleave(2, 1).repeat_interleave(2, 2))
    Y.zero_()
    entry("mw_unet_copy_channels", B * h * w, C, Ctot, c0, X, Y)
    assert torch.equal(Y.reshape(-1, Ctot)[:B * h * w, c0:c0 + C], X.reshape(-1, C))
    P = at((B, h // 2, w // 2, C), bf16, offset)
    entry("mw_unet_avgpool2", B, h, w, C, X, P)
    x = X.float()
    assert torch.equal(P, (0.25 * (x[:, ::2, ::2] + x[:, ::2, 1::2] + x[:, 1::2, ::2] + x[:, 1::2, 1::2])).to(bf16))
    dY = at((B, 2 * h, 2 * w, Ctot), torch.float32, offset)
    dY.copy_(rnd(B, 2 * h, 2 * w, Ctot))
    dX = at((B, h, w, C), torch.float32, offset)
    entry("mw_unet_upsample2_bwd", B, h, w, C, Ctot, c0, dY, dX)
    d = dY[..., c0:c0 + C]
    assert torch.equal(dX, d[:, ::2, ::2] + d[:, ::2, 1::2] + d[:, 1::2, ::2] + d[:, 1::2, 1::2])
    base = rnd(B * 4 * h * w, C)
    for acc in (0, 1):
        S = at((B * 4 * h * w, C), torch.float32, offset)
        S.copy_(base)
        entry("mw_unet_slice_grad", B * 4 * h * w, C, Ctot, c0, dY, S, acc)
        assert torch.equal(S, d.reshape(-1, C) + (base if acc else 0))
        G = at((B, 2 * h, 2 * w, C), torch.float32, offset)
        G.copy_(base.view(B, 2 * h, 2 * w, C))
        entry("mw_unet_avgpool2_bwd", B, 2 * h, 2 * w, C, dX, G, acc)
        up = 0.25 * dX.repeat_interleave(2, 1).repeat_interleave(2, 2)
        assert torch.equal(G, up + (base.view_as(G) if acc else 0))
