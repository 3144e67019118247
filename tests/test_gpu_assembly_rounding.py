"""The rounding of the assembled viscous block (nine rounded additions an entry, one a Gauss point) and its range
in FP32."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def assemble(nx, nz, Lx, etaq, precision):
    from meeuuw_b200 import _lib, fe_tables, ops
    box = _lib.box_of(nx, nz, Lx, Lx * nz / nx)
    nel = nx * nz
    D = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()
    one = torch.ones(nel, 9, dtype=torch.float64, device="cuda")
    q = dict(rhoq=one, etaq=D(etaq), gxq=0 * one, gzq=-one, eta_e=D(etaq.mean(1)),
             **fe_tables.uniform_geometry(nel, box.hx, box.hz))
    nv = 2 * (2 * nx + 1) * (2 * nz + 1)
    fix = torch.zeros(nv, dtype=torch.bool, device="cuda")
    val = torch.zeros(nv, dtype=torch.float64, device="cuda")
    out = ops.assemble_stokes(box, True, precision, q, fe_tables.device_tables(), fix, val, 1.0, 1.0)
    return box, out["VV_K"].cpu().numpy().reshape(nel, 9, 2, 9, 2)


def test_rounding_of_the_own_component():
    """Against exact sums, the root mean square error is that of nine additions of rounded products (computed
    here on the same numbers), within 4 %: the same data in eighteen additions are 8 to 15 % further off."""
    from meeuuw_b200 import fe_tables
    nx, nz = 37, 53
    etaq = np.exp(np.random.default_rng(0).uniform(-6, 6, (nx * nz, 9)))
    box, K = assemble(nx, nz, 1.3, etaq, 0)
    t = {k: np.asarray(v, dtype=np.float64) for k, v in fe_tables.host_tables().items()}
    W = box.hx * box.hz / 4 * t["weightq"]
    D = ((2 / box.hx) * t["dNdr_V"], (2 / box.hz) * t["dNdt_V"])
    wide = np.longdouble
    fma = lambda a, b, c: (wide(a) * wide(b) + wide(c)).astype(np.float64)
    got = nine = 0.0
    for c in (0, 1):
        o, s = D[c], D[1 - c]
        for i in range(9):
            exact, model = np.zeros((nx * nz, 9), dtype=wide), np.zeros((nx * nz, 9))
            for q in range(9):
                for j in range(9):
                    exact[:, j] += wide(etaq[:, q]) * wide(W[q]) * (2 * wide(o[q, i]) * wide(o[q, j])
                                                                      + wide(s[q, i]) * wide(s[q, j]))
                    a = fma(np.float64(2 * o[q, i]), np.float64(o[q, j]), np.float64(s[q, i] * s[q, j]))
                    model[:, j] = fma(a * etaq[:, q], np.float64(W[q]), model[:, j])
            scale = np.abs(exact[:, i:i + 1])
            got += float((((K[:, i, c, :, c] - exact) / scale) ** 2).mean())
            nine += float((((model - exact) / scale) ** 2).mean())
    assert got ** 0.5 <= 1.04 * nine ** 0.5, (got ** 0.5, nine ** 0.5)


def test_fp32_range():
    """Entries of some 1e28 from a viscosity whose product with JxW (4e38) is past FP32's largest number; FP32
    rounds each of about ten operations an entry, of terms up to ten times the entry: 1e-5 of the largest."""
    etaq = np.exp(np.random.default_rng(1).uniform(-0.1, 0.1, (12, 9))) * 1e28
    _, K = assemble(4, 3, 3e6, etaq, 0)
    _, K32 = assemble(4, 3, 3e6, etaq, 1)
    assert np.isfinite(K32).all()
    assert np.abs(K32 - K).max() <= 1e-5 * np.abs(K).max()
