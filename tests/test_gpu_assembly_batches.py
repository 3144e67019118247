"""Stokes element assembly at the edges of its batches, against a plain PyTorch FP64 form of the same sums.

Sizes: one element, a batch (16 elements), one element more, more batches than the CTAs of a launch; fixed
degrees of freedom inside and on the boundary with non-zero values; outputs on and off a 16-byte boundary
(bulk copies or plain stores).  Tolerances relative to the largest entry: 9 products summed and at most 18
eliminated terms, 1e-13 in FP64 and 1e-5 in FP32 (eps 6e-8 times about 9 * 9 roundings).
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

f64 = torch.float64


def _reference(box, q, tb, fix, val, scale):
    nel = box.nelx * box.nelz
    nnx = 2 * box.nelx + 1
    e = torch.arange(nel, device="cuda")
    ex, ez = e % box.nelx, e // box.nelx
    dx = torch.tensor([0, 2, 2, 0, 1, 2, 1, 0, 1], device="cuda")
    dz = torch.tensor([0, 0, 2, 2, 0, 1, 2, 1, 1], device="cuda")
    node = (2 * ez[:, None] + dz) * nnx + 2 * ex[:, None] + dx
    dof = torch.stack([2 * node, 2 * node + 1], -1).reshape(nel, 18)
    NV, NP = tb["N_V"].reshape(9, 9), tb["N_P"].reshape(9, 4)
    x = lambda a, b, s: q[a][..., None] * tb["dNdr_" + s].reshape(9, -1) + q[b][..., None] * tb["dNdt_" + s].reshape(9, -1)
    gx, gz = x("jcbi00q", "jcbi01q", "V"), x("jcbi10q", "jcbi11q", "V")
    px, pz = x("jcbi00q", "jcbi01q", "P"), x("jcbi10q", "jcbi11q", "P")
    J = q["JxWq"]
    B = torch.zeros(nel, 9, 3, 18, dtype=f64, device="cuda")
    B[:, :, 0, 0::2], B[:, :, 1, 1::2], B[:, :, 2, 0::2], B[:, :, 2, 1::2] = gx, gz, gz, gx
    C = torch.tensor([2.0, 2.0, 1.0], dtype=f64, device="cuda")
    K = torch.einsum("eqai,a,eqaj,eq->eij", B, C, B, q["etaq"] * J)
    f = torch.zeros(nel, 18, dtype=f64, device="cuda")
    f[:, 0::2] = torch.einsum("qi,eq->ei", NV, J * q["rhoq"] * q["gxq"])
    f[:, 1::2] = torch.einsum("qi,eq->ei", NV, J * q["rhoq"] * q["gzq"])
    d = torch.stack([gx, gz], -1).reshape(nel, 9, 18)
    G = -torch.einsum("eqi,qk,eq->eik", d, NP, J) * scale
    H = torch.zeros(nel, 4, 18, dtype=f64, device="cuda")
    H[:, :, 0::2] = torch.einsum("eqk,qi,eq->eki", px, NV, J)
    H[:, :, 1::2] = torch.einsum("eqk,qi,eq->eki", pz, NV, J)
    M = torch.einsum("qk,ql,eq->ekl", NP, NP, J)
    fx, v = fix[dof], torch.where(fix[dof], val[dof], torch.zeros((), dtype=f64, device="cuda"))
    kd = torch.diagonal(K, dim1=1, dim2=2).clone()
    f = torch.where(fx, kd * v, f - torch.einsum("eij,ej->ei", K, v))
    h = -torch.einsum("eik,ei->ek", G, v)
    K = K.masked_fill(fx[:, :, None] | fx[:, None, :], 0.0) + torch.diag_embed(torch.where(fx, kd, torch.zeros_like(kd)))
    G = G.masked_fill(fx[:, :, None], 0.0)
    rf = torch.zeros(2 * nnx * (2 * box.nelz + 1), dtype=f64, device="cuda").index_add_(0, dof.reshape(-1), f.reshape(-1))
    ncx = box.nelx + 1
    pn = torch.stack([ez * ncx + ex, ez * ncx + ex + 1, (ez + 1) * ncx + ex + 1, (ez + 1) * ncx + ex], 1)
    rh = torch.zeros(ncx * (box.nelz + 1), dtype=f64, device="cuda").index_add_(0, pn.reshape(-1), h.reshape(-1))
    full = torch.cat([K, G.repeat_interleave(2, 2)], 2)
    return dict(VV_Stokes=full, VV_K=K, VV_G=G, VV_GT=G.transpose(1, 2), VV_M=M, VV_M_eta=M / q["eta_e"][:, None, None],
                VV_H=H, rhs_f=rf, rhs_h=rh)


@pytest.mark.parametrize("nelx,nelz", [(1, 1), (4, 4), (17, 1), (5, 7), (130, 61)])
@pytest.mark.parametrize("blocks", [False, True])
@pytest.mark.parametrize("precision,shift", [(0, 0), (0, 1), (1, 0), (1, 1)])
def test_assembly_batches(nelx, nelz, blocks, precision, shift):
    from meeuuw_b200 import _lib, fe_tables, ops
    box = _lib.box_of(nelx, nelz, 1.3, 0.9)
    nel, nv = nelx * nelz, 2 * (2 * nelx + 1) * (2 * nelz + 1)
    gen = torch.Generator("cuda").manual_seed(nelx * 7 + nelz)
    R = lambda *s, lo=0.5, hi=1.5: lo + (hi - lo) * torch.rand(*s, dtype=f64, device="cuda", generator=gen)
    q = {k: R(nel, 9) for k in ("rhoq", "etaq", "gxq", "gzq", "JxWq", "jcbi00q", "jcbi11q")}
    q.update(jcbi01q=R(nel, 9, lo=-0.3, hi=0.3), jcbi10q=R(nel, 9, lo=-0.3, hi=0.3), eta_e=R(nel))
    tb = fe_tables.device_tables()
    fix, val = R(nv, lo=0.0, hi=1.0) < 0.15, R(nv, lo=-1.0, hi=1.0)
    ref = _reference(box, q, tb, fix, val, 3.0 / 1.5)
    dt = torch.float32 if precision else f64
    out = {k: torch.zeros(ref[k].numel() + 4, dtype=dt, device="cuda")[shift:shift + ref[k].numel()]
           for k in (("VV_K", "VV_G", "VV_GT", "VV_M", "VV_M_eta", "VV_H") if blocks else ("VV_Stokes",))}
    out.update(rhs_f=torch.zeros(nv, dtype=f64, device="cuda"),
               rhs_h=torch.zeros((nelx + 1) * (nelz + 1), dtype=f64, device="cuda"))
    ops.assemble_stokes(box, blocks, precision, q, tb, fix, val, 3.0, 1.5, out=out)
    for k, v in out.items():
        r = ref[k].reshape(-1)
        assert float((v.to(f64) - r).abs().max()) <= (1e-5 if precision else 1e-13) * max(float(r.abs().max()), 1e-3), k
