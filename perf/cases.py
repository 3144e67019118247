"""Workloads that stand for this framework's use, for timing and for comparing results.

A case is a dict of plain values; `prepare` makes what a program has in hand before the call,
`run` is one pass through the public entry points, `exact` the same numbers from plain torch in
64 bits where that is quick, `work` the bytes and operations a pass cannot do without.

Kinds of work:
  step      one recorded time step of a model (`GPUModel.capture_step`, then `step`), from the same
            state every pass: the particles, fields and Stokes guess are put back first
  cold      a Stokes solve from zero for a new viscosity (`StokesSolver.set_viscosity`, `solve`)
  apply     the matrix-free Stokes operator on a velocity and a pressure (`StokesSolver.apply`)
  pic       the particle half of a step (`ops`: interpolation and material, binning, projections,
            advection, locate)
  assemble  the element matrices and right-hand side of Stokes (`ops.assemble_stokes`)
  energy    the temperature equation of a step (`ops.energy_op_setup`, `ops.energy_op_solve`)
  train     one training step of the warm-start network (`UNet.forward`, `mse`, `backward`, `step`)
"""
import math

import numpy as np
import torch

from meeuuw_b200 import _lib, configs, fe_tables, ops
from meeuuw_b200.stokes import StokesSolver
from meeuuw_b200.timestep import GPUModel
from meeuuw_b200.unet import NOUT, UNet

f64 = torch.float64


def listed():
    return [
        # the smallest member of an ensemble of convection models: a step is a chain of short launches
        dict(name="step_fk_64", kind="step", model="fk", nelx=64, nelz=64, precision="mixed"),
        # a box whose element counts are not multiples of anything, as ensembles and aspect ratios give
        dict(name="step_fk_150x97", kind="step", model="fk", nelx=150, nelz=97, precision="mixed"),
        # two materials, no slip, 25 particles per element, no temperature
        dict(name="step_rt_256", kind="step", model="rt", nelx=256, nelz=256, precision="mixed"),
        # the headline model: 512^2 elements, 4.2 million particles
        dict(name="step_fk_512", kind="step", model="fk", nelx=512, nelz=512, precision="mixed"),
        # the plain FP64 solver, which parity runs and comparisons use
        dict(name="step_fk_128_f64", kind="step", model="fk", nelx=128, nelz=128, precision="f64"),
        # the first step of a model, or a restart: no previous solution to start from
        dict(name="cold_fk_384x256", kind="cold", nelx=384, nelz=256, contrast=1e4),
        # the operator alone, as a caller with an iteration of its own uses it
        dict(name="apply_f32_512", kind="apply", nelx=512, nelz=512, precision="f32"),
        # the particle half of a step, the headline model's and a small two-material one
        dict(name="pic_fk_512", kind="pic", model="fk", nelx=512, nelz=512, ppd=4, rk=4),
        dict(name="pic_rt_40x33", kind="pic", model="rt", nelx=40, nelz=33, ppd=5, rk=2),
        # assembled matrices, for programs that keep their own sparse solver
        dict(name="assemble_256", kind="assemble", nelx=256, nelz=256, blocks=False, precision="f64"),
        # the temperature equation of a medium box with shear heating
        dict(name="energy_eba_300x200", kind="energy", nelx=300, nelz=200, formulation="EBA"),
        # training of the warm-start network on 128^2 snapshots
        dict(name="train_128_b16", kind="train", n=128, batch=16),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "cold", "apply", "pic", "pic", "assemble", "energy", "train"])
    n = lambda lo, hi: int(round(_log(rng, lo, hi)))
    if kind == "step":
        precision = rng.choice(["mixed", "mixed", "mixed", "f64"])
        top = 400 if precision == "mixed" else 160
        return dict(kind=kind, model=rng.choice(["fk", "fk", "rt"]), nelx=n(48, top), nelz=n(48, top),
                    precision=precision)
    if kind == "cold":
        return dict(kind=kind, nelx=n(48, 384), nelz=n(48, 384), contrast=round(_log(rng, 1.0, 1e5), 3))
    if kind == "apply":
        return dict(kind=kind, nelx=n(32, 512), nelz=n(32, 512), precision=rng.choice(["f32", "f64"]))
    if kind == "pic":
        return dict(kind=kind, model=rng.choice(["fk", "rt"]), nelx=n(24, 512), nelz=n(24, 400),
                    ppd=rng.choice([3, 4, 5]), rk=rng.choice([1, 2, 4]))
    if kind == "assemble":
        return dict(kind=kind, nelx=n(32, 256), nelz=n(32, 256), blocks=rng.random() < 0.5,
                    precision=rng.choice(["f32", "f64"]))
    if kind == "energy":
        return dict(kind=kind, nelx=n(32, 512), nelz=n(32, 512), formulation=rng.choice(["BA", "EBA"]))
    return dict(kind=kind, n=rng.choice([32, 64, 128]), batch=rng.randint(1, 16))


# ------------------------------------------------------------------------------------- set-up
def _config(case, seed):
    base = configs.fk_convection(case["nelx"]) if case["model"] == "fk" else configs.rayleigh_taylor(case["nelx"])
    kw = dict(nelx=case["nelx"], nelz=case["nelz"], seed=int(seed))
    if "ppd" in case:
        kw["nparticle_per_dim"] = case["ppd"]
    return configs.replace(base, **kw)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _lattice(box):
    """x, z of the Q2 lattice, flat, x fastest."""
    x = torch.arange(2 * box.nelx + 1, dtype=f64, device="cuda") * (box.hx / 2)
    z = torch.arange(2 * box.nelz + 1, dtype=f64, device="cuda") * (box.hz / 2)
    return x.repeat(2 * box.nelz + 1), z.repeat_interleave(2 * box.nelx + 1)


def _temperature(box, g):
    """A convecting temperature: the conductive profile, a few smooth modes, a little noise."""
    x, z = _lattice(box)
    T = 1.0 - z
    for k, l in ((1, 1), (2, 1), (3, 2), (1, 3)):
        a, ph = torch.rand(2, generator=g, device="cuda", dtype=f64)
        T = T + (0.25 * (a - 0.5) / l) * torch.cos(math.pi * k * x + 6.283 * ph) * torch.sin(math.pi * l * z)
    T = T + 1e-3 * torch.randn(T.shape, generator=g, device="cuda", dtype=f64)
    T = T.clamp(0.0, 1.0)
    T[z < 1e-12] = 1.0
    T[z > 1 - 1e-12] = 0.0
    return T


def _cell_velocity(box, g, amplitude=100.0):
    """A velocity of a few convection cells with zero normal flow on the sides."""
    x, z = _lattice(box)
    u, w = torch.zeros_like(x), torch.zeros_like(x)
    for k, l in ((1, 1), (2, 1), (1, 2)):
        a = amplitude * torch.randn(1, generator=g, device="cuda", dtype=f64)
        kx, kz = math.pi * k / box.Lx, math.pi * l / box.Lz
        u += a * kz * torch.sin(kx * x) * torch.cos(kz * z)
        w -= a * kx * torch.cos(kx * x) * torch.sin(kz * z)
    return u, w


def _free_slip(box):
    nnx, nnz = 2 * box.nelx + 1, 2 * box.nelz + 1
    fix = torch.zeros(nnz, nnx, 2, dtype=torch.bool, device="cuda")
    fix[:, 0, 0] = fix[:, -1, 0] = True
    fix[0, :, 1] = fix[-1, :, 1] = True
    return fix.reshape(-1)


def _elements(box):
    """(nel, 9) Q2 and (nel, 4) Q1 node numbers."""
    ez, ex = torch.meshgrid(torch.arange(box.nelz, device="cuda"), torch.arange(box.nelx, device="cuda"),
                            indexing="ij")
    ex, ez, nnx = ex.reshape(-1), ez.reshape(-1), 2 * box.nelx + 1
    b = 2 * ex + 2 * ez * nnx
    v = torch.stack([b, b + 2, b + 2 + 2 * nnx, b + 2 * nnx, b + 1, b + 2 + nnx, b + 1 + 2 * nnx, b + nnx,
                     b + 1 + nnx], 1)
    p = ex + ez * (box.nelx + 1)
    return v, torch.stack([p, p + 1, p + box.nelx + 2, p + box.nelx + 1], 1)


def _box(case, Lx=None, Lz=1.0):
    return _lib.box_of(case["nelx"], case["nelz"], case["nelx"] / case["nelz"] if Lx is None else Lx, Lz)


_STATE = ("x", "z", "active", "r", "t", "iel", "T", "exx_n", "ezz_n", "exz_n", "q", "u", "w", "p", "solV", "solP",
          "dt_state")


def _prepare_step(case, seed):
    cfg = _config(case, seed)
    m = GPUModel(cfg, configs.build_host_model(cfg), stokes=case["precision"])
    m.step()                                      # the cold start
    m.capture_step()
    live = [getattr(m, k) for k in _STATE]
    return dict(model=m, live=live, kept=[a.clone() for a in live])


def _prepare_stokes(case, seed):
    g = _generator(seed)
    box = _box(case)
    nel = box.nelx * box.nelz
    tables = fe_tables.device_tables()
    geo = fe_tables.uniform_geometry(nel, box.hx, box.hz)
    icon, _ = _elements(box)
    T = _temperature(box, g)
    eta_e = torch.exp(-math.log(case.get("contrast", 1e4)) * T[icon].mean(1))
    rho_e = 1.0 - 1e-2 * T[icon].mean(1)
    wide = lambda a: a[:, None].expand(-1, 9).contiguous()
    s = dict(box=box, tables=tables, geo=geo, fix=_free_slip(box), eta_e=eta_e, etaq=wide(eta_e), rhoq=wide(rho_e),
             gxq=torch.zeros(nel, 9, dtype=f64, device="cuda"),
             gzq=torch.full((nel, 9), -1e6 / 1e-2, dtype=f64, device="cuda"))
    return s, g


def _prepare_cold(case, seed):
    s, _ = _prepare_stokes(case, seed)
    box = s["box"]
    nn, npp = (2 * box.nelx + 1) * (2 * box.nelz + 1), (box.nelx + 1) * (box.nelz + 1)
    s["f"], s["h"] = torch.empty(2 * nn, dtype=f64, device="cuda"), torch.empty(npp, dtype=f64, device="cuda")
    ops.stokes_rhs_body(box, s["rhoq"], s["gxq"], s["gzq"], s["geo"]["JxWq"], s["tables"]["N_V"], s["fix"], s["f"],
                        s["h"])
    s["solver"] = StokesSolver(box, s["fix"], eta_ref=1.0, L_ref=0.5 * (box.Lx + box.Lz), precisions=("f32",),
                               cheb_degree=2, power_iters_warm=6)
    return s


def _prepare_apply(case, seed):
    s, g = _prepare_stokes(case, seed)
    box = s["box"]
    s["solver"] = StokesSolver(box, s["fix"], eta_ref=1.0, L_ref=0.5 * (box.Lx + box.Lz),
                               precisions=(case["precision"],))
    s["solver"].set_viscosity(s["etaq"], s["eta_e"])
    dt = torch.float32 if case["precision"] == "f32" else f64
    u, w = _cell_velocity(box, g)
    npp = (box.nelx + 1) * (box.nelz + 1)
    s["u"] = torch.stack([u, w], 1).reshape(-1).to(dt)
    s["u"] += torch.randn(s["u"].shape, generator=g, device="cuda", dtype=dt)
    s["p"] = (1e4 * torch.randn(npp, generator=g, device="cuda", dtype=f64)).to(dt)
    return s


def _prepare_pic(case, seed):
    cfg = _config(case, 0)
    g = _generator(seed)
    box = _lib.box_of(cfg.nelx, cfg.nelz, cfg.Lx, cfg.Lz)
    nel, ppe = cfg.nel, cfg.nparticle_per_dim ** 2
    n = nel * ppe
    # the swarm as the set-up makes it, element by element at random places, carried on a little
    e = torch.arange(nel, device="cuda").repeat_interleave(ppe)
    rnd = lambda: torch.rand(n, generator=g, device="cuda", dtype=f64)
    x = ((e % cfg.nelx) + 0.002 + 0.996 * rnd()) * box.hx
    z = ((e // cfg.nelx) + 0.002 + 0.996 * rnd()) * box.hz
    s = dict(cfg=cfg, box=box, x0=x, z0=z, act0=torch.ones(n, dtype=torch.bool, device="cuda"),
             mat=(z >= 0.2 + 0.02 * torch.cos(x * math.pi / 0.9142)).to(torch.int8),
             material=ops.material_struct(cfg))
    u, w = _cell_velocity(box, g)
    s["u"], s["w"] = u, w
    speed = float(torch.maximum(u.abs().max(), w.abs().max()))
    s["dt"] = 0.25 * min(box.hx, box.hz) / speed
    T = _temperature(box, g)
    s["nodal"] = dict(exx=torch.randn(T.shape, generator=g, device="cuda", dtype=f64), ezz=w / 7, exz=u / 3,
                      q=1e3 * T, T=T)
    E = lambda dt=f64: torch.empty(n, dtype=dt, device="cuda")
    s["x"], s["z"], s["act"] = x.clone(), z.clone(), s["act0"].clone()
    s["r"], s["t"], s["iel"] = E(), E(), E(torch.int32)
    s["err"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    ops.locate(box, s["act"], s["x"], s["z"], s["r"], s["t"], s["iel"], s["err"])
    s["r0"], s["t0"], s["iel0"] = s["r"].clone(), s["t"].clone(), s["iel"].clone()
    s["props"] = {k: E() for k in ("exx", "ezz", "exz", "p", "T", "rho", "eta", "hcond", "hcapa", "hprod", "alpha")}
    s["up"], s["wp"] = E(), E()
    s["counts"], s["offsets"] = (torch.empty(nel + k, dtype=torch.int32, device="cuda") for k in (0, 1))
    s["order"] = E(torch.int32)
    s["rho_e"], s["eta_e"] = (torch.empty(nel, dtype=f64, device="cuda") for _ in range(2))
    s["rho_n"], s["eta_n"] = torch.empty_like(T), torch.empty_like(T)
    return s


def _prepare_energy(case, seed):
    s, g = _prepare_stokes(case, seed)
    box = s["box"]
    nel = box.nelx * box.nelz
    T = _temperature(box, g)
    _, z = _lattice(box)
    s["fixT"] = (z < 1e-12) | (z > 1 - 1e-12)
    s["valT"] = torch.where(z < 0.5, 1.0, 0.0).to(f64) * s["fixT"]
    u, w = _cell_velocity(box, g)
    NV = s["tables"]["N_V"]
    s["dt"] = 0.25 * min(box.hx, box.hz) / float(torch.maximum(u.abs().max(), w.abs().max()))
    q = lambda a: ops.nodal_to_qpoints(box, _lib.SPACE_Q2, NV, a)
    full = lambda v: torch.full((nel, 9), v, dtype=f64, device="cuda")
    s["q"] = dict(rhoq=s["rhoq"], etaq=s["etaq"], Tq=q(T), uq=q(u), wq=q(w), hcondq=full(1.0), hcapaq=full(1.0),
                  alphaq=full(1e-2), hprodq=full(0.0), exxq=q(u), ezzq=q(w), exzq=q(0.5 * (u - w)), **s["geo"])
    for k in ("exxq", "ezzq", "exzq"):
        s["q"][k] *= 1e-2
    s["T"] = T
    s["op"] = torch.empty(_lib.lib().mw_energy_op_bytes(box), dtype=torch.uint8, device="cuda")
    s["rhs"], s["sol"] = torch.empty_like(T), torch.empty_like(T)
    return s


def _prepare_train(case, seed):
    g = _generator(seed)
    n, b = case["n"], case["batch"]
    net = UNet(base=32, levels=4, seed=int(seed))
    X = torch.randn(b, n // 8, n // 8, 2, generator=g, device="cuda").repeat_interleave(8, 1).repeat_interleave(8, 2)
    X = X + 0.1 * torch.randn(b, n, n, 2, generator=g, device="cuda")
    Y = torch.randn(b * n * n, NOUT, generator=g, device="cuda")
    return dict(net=net, X=X.to(torch.bfloat16), Y=Y, b=b, n=n)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        s = _prepare_step(case, seed)
    elif kind == "cold":
        s = _prepare_cold(case, seed)
    elif kind == "apply":
        s = _prepare_apply(case, seed)
    elif kind == "pic":
        s = _prepare_pic(case, seed)
    elif kind == "assemble":
        s, _ = _prepare_stokes(case, seed)
        s["val"] = torch.zeros(s["fix"].shape, dtype=f64, device="cuda")
    elif kind == "energy":
        s = _prepare_energy(case, seed)
    else:
        s = _prepare_train(case, seed)
    s["case"] = case
    return s


# ---------------------------------------------------------------------------------------- run
def _run_step(s):
    m = s["model"]
    torch._foreach_copy_(s["live"], s["kept"])
    m.step()
    out = {k: getattr(m, k) for k in ("u", "w", "p", "x", "z", "active", "iel", "gq_out", "dt_out")}
    if m.cfg.solve_T:
        out.update(T=m.T, nu_out=m.nu_out)
    return out


def _run_cold(s):
    s["solver"].set_viscosity(s["etaq"], s["eta_e"])
    V, P, _ = s["solver"].solve(s["f"], s["h"], scheme="cd_u_eta", precision="mixed", tol=1e-8, inner_rtol=2e-2,
                                mass_iters=6, sweep_target=0.1)
    return dict(V=V, P=P)


def _run_pic(s):
    cfg, box, P = s["cfg"], s["box"], s["props"]
    torch._foreach_copy_([s[k] for k in ("x", "z", "act", "r", "t", "iel")],
                         [s[k + "0"] for k in ("x", "z", "act", "r", "t", "iel")])
    nel = cfg.nel
    ops.interp_material(box, s["act"], s["r"], s["t"], s["iel"], s["mat"], s["nodal"], s["material"], P)
    ops.bin_particles(nel, s["act"], s["iel"], s["counts"], s["offsets"], s["order"], s["err"])
    ops.project_elements(nel, s["offsets"], s["order"], P["rho"], P["eta"], cfg.averaging, s["rho_e"], s["eta_e"],
                         s["err"])
    ops.project_nodes(box, cfg.nodal_projection_type, [(P["rho"], "arithmetic"), (P["eta"], cfg.averaging)],
                      s["offsets"], s["order"], s["r"], s["t"], [s["rho_n"], s["eta_n"]])
    ops.advect(box, s["case"]["rk"], s["dt"], s["x"], s["z"], s["act"], s["u"], s["w"], s["up"], s["wp"], s["err"])
    ops.locate(box, s["act"], s["x"], s["z"], s["r"], s["t"], s["iel"], s["err"])
    out = {k: s[k] for k in ("counts", "offsets", "order", "rho_e", "eta_e", "rho_n", "eta_n", "x", "z", "act", "up",
                             "wp", "r", "t", "iel")}
    out.update({"p_" + k: P[k] for k in ("exx", "ezz", "exz", "p", "T", "rho", "eta")})
    return out


def _run_energy(s):
    box, c = s["box"], s["case"]
    ops.energy_op_setup(box, s["T"], s["q"], s["tables"], s["fixT"], s["valT"], s["dt"], 1.0, c["formulation"],
                        s["op"], s["rhs"])
    s["sol"].copy_(s["T"])
    ops.energy_op_solve(box, s["op"], s["rhs"], s["sol"], rtol=1e-10, maxit=300)
    return dict(rhs=s["rhs"], T=s["sol"])


def _run_train(s):
    net = s["net"]
    y = net.forward(s["X"], s["b"], s["n"], s["n"])
    dy, part = net.mse(y, s["Y"])
    net.backward(dy)
    net.step(lr=1e-4)
    out = dict(y=y, loss=part)
    for i, l in enumerate(net.layers()):
        out.update({f"gw{i}": l.gw, f"gb{i}": l.gb, f"w{i}": l.w, f"b{i}": l.b})
    return out


def run(state):
    kind = state["case"]["kind"]
    if kind == "step":
        return _run_step(state)
    if kind == "cold":
        return _run_cold(state)
    if kind == "apply":
        yV, yP = state["solver"].apply(state["u"], state["p"], precision=state["case"]["precision"])
        return dict(yV=yV, yP=yP)
    if kind == "pic":
        return _run_pic(state)
    if kind == "assemble":
        c = state["case"]
        q = dict(rhoq=state["rhoq"], etaq=state["etaq"], gxq=state["gxq"], gzq=state["gzq"], eta_e=state["eta_e"],
                 **state["geo"])
        return ops.assemble_stokes(state["box"], c["blocks"], 1 if c["precision"] == "f32" else 0, q,
                                   state["tables"], state["fix"], state["val"], 1.0,
                                   0.5 * (state["box"].Lx + state["box"].Lz))
    if kind == "energy":
        return _run_energy(state)
    return _run_train(state)


# ---------------------------------------------------------------------------------------- exact
def _host_tables():
    return {k: torch.as_tensor(v, dtype=f64, device="cuda") for k, v in fe_tables.host_tables().items()}


def _exact_apply(case, seed):
    s = _prepare_apply(case, seed)
    box, t = s["box"], _host_tables()
    iv, ip = _elements(box)
    scale = 1.0 / (0.5 * (box.Lx + box.Lz))
    sx, sz, jac = 2 / box.hx, 2 / box.hz, box.hx * box.hz / 4
    fix = s["fix"].view(-1, 2)
    u = s["u"].to(f64).view(-1, 2)
    um = torch.where(fix, 0.0, u)
    # the operator sees the viscosity in its own type
    etaq = s["etaq"].to(s["u"].dtype).to(f64)
    yV, yP = torch.zeros_like(u), torch.zeros((box.nelx + 1) * (box.nelz + 1), dtype=f64, device="cuda")
    dk = torch.zeros_like(u)
    B, Z, W = sx * t["dNdr_V"], sz * t["dNdt_V"], jac * t["weightq"]
    for a in range(0, iv.shape[0], 65536):
        v, p, e = iv[a:a + 65536], ip[a:a + 65536], etaq[a:a + 65536] * W
        ue = um[v]
        dx, dz = torch.einsum("qk,ekc->eqc", B, ue), torch.einsum("qk,ekc->eqc", Z, ue)
        pq = scale * W * (s["p"].to(f64)[p] @ t["N_P"].T)
        sxx, szz, sxz = 2 * e * dx[..., 0] - pq, 2 * e * dz[..., 1] - pq, e * (dz[..., 0] + dx[..., 1])
        yu = sxx @ B + sxz @ Z
        yw = szz @ Z + sxz @ B
        yV.index_add_(0, v.reshape(-1), torch.stack([yu, yw], 2).reshape(-1, 2))
        yP.index_add_(0, p.reshape(-1), (-scale * W * (dx[..., 0] + dz[..., 1]) @ t["N_P"]).reshape(-1))
        dd = torch.stack([e @ (2 * B * B + Z * Z), e @ (2 * Z * Z + B * B)], 2)
        dk.index_add_(0, v.reshape(-1), dd.reshape(-1, 2))
    yV = torch.where(fix, dk * u, yV)
    return dict(yV=yV.reshape(-1), yP=yP)


def _q2(r, t):
    lr = (0.5 * r * (r - 1), (1 - r) * (1 + r), 0.5 * r * (r + 1))
    lt = (0.5 * t * (t - 1), (1 - t) * (1 + t), 0.5 * t * (t + 1))
    return torch.stack([lr[i] * lt[j] for i, j in ((0, 0), (2, 0), (2, 2), (0, 2), (1, 0), (2, 1), (1, 2), (0, 1),
                                                   (1, 1))], 1)


def _exact_pic(case, seed):
    s = _prepare_pic(case, seed)
    cfg, box = s["cfg"], s["box"]
    iv, _ = _elements(box)
    nel = iv.shape[0]
    r, t, e = s["r0"], s["t0"], s["iel0"].long()
    N = _q2(r, t)
    at = lambda a: (N * a[iv[e]]).sum(1)
    out = {"p_" + k: at(s["nodal"][j]) for k, j in (("exx", "exx"), ("ezz", "ezz"), ("exz", "exz"), ("p", "q"),
                                                    ("T", "T"))}
    if case["model"] == "fk":
        rho, eta = cfg.rho0 * (1 - cfg.alphaT * out["p_T"]), torch.exp(-cfg.fk_gamma * out["p_T"])
    else:
        pick = lambda v: torch.tensor(v, dtype=f64, device="cuda")[s["mat"].long()]
        rho, eta = pick(cfg.mat_rho), pick(cfg.mat_eta)
    out.update(p_rho=rho, p_eta=eta)
    fwd, inv = {"geometric": (torch.log10, lambda a: 10.0 ** a), "harmonic": (lambda a: 1 / a, lambda a: 1 / a),
                "arithmetic": (lambda a: a, lambda a: a)}[cfg.averaging]
    add = lambda n, i, v: torch.zeros(n, dtype=f64, device="cuda").index_add_(0, i, v)
    cnt = add(nel, e, torch.ones_like(rho))
    out.update(rho_e=add(nel, e, rho) / cnt, eta_e=inv(add(nel, e, fwd(eta)) / cnt))
    W = torch.stack([(1 - r) * (1 - t), (1 + r) * (1 - t), (1 + r) * (1 + t), (1 - r) * (1 + t)], 1) / 4
    nnx, nnz = 2 * box.nelx + 1, 2 * box.nelz + 1
    node = iv[e][:, :4].reshape(-1)
    nodal = lambda v: add(nnx * nnz, node, (W * v[:, None]).reshape(-1))
    den = nodal(torch.ones_like(rho))
    for k, v in (("rho_n", nodal(rho) / den), ("eta_n", inv(nodal(fwd(eta)) / den))):
        c = v.view(nnz, nnx)[::2, ::2]
        f = torch.empty(nnz, nnx, dtype=f64, device="cuda")
        f[::2, ::2] = c
        f[::2, 1::2] = (c[:, :-1] + c[:, 1:]) / 2
        f[1::2, ::2] = (c[:-1] + c[1:]) / 2
        f[1::2, 1::2] = (c[:-1, :-1] + c[:-1, 1:] + c[1:, 1:] + c[1:, :-1]) / 4
        out[k] = f.reshape(-1)

    def velocity(x, z):
        ex, ez = (x / box.hx).long().clamp(0, box.nelx - 1), (z / box.hz).long().clamp(0, box.nelz - 1)
        M = _q2(2 * (x / box.hx - ex) - 1, 2 * (z / box.hz - ez) - 1)
        v = iv[ez * box.nelx + ex]
        return (M * s["u"][v]).sum(1), (M * s["w"][v]).sum(1)

    x, z, dt = s["x0"], s["z0"], s["dt"]
    ua, wa = velocity(x, z)
    if case["rk"] > 1:
        ub, wb = velocity(x + ua * dt / 2, z + wa * dt / 2)
        if case["rk"] == 2:
            ua, wa = ub, wb
        else:
            uc, wc = velocity(x + ub * dt / 2, z + wb * dt / 2)
            ud, wd = velocity(x + uc * dt, z + wc * dt)
            ua, wa = (ua + 2 * ub + 2 * uc + ud) / 6, (wa + 2 * wb + 2 * wc + wd) / 6
    xn, zn = x + ua * dt, z + wa * dt
    if bool(((xn < 0) | (xn > box.Lx) | (zn < 0) | (zn > box.Lz)).any()):
        return out                                # particles leave: where they go is the code's rule
    out.update(up=ua, wp=wa, x=xn, z=zn)
    return out


def _exact_assemble(case, seed):
    s = _prepare_stokes(case, seed)[0]
    box, t = s["box"], _host_tables()
    iv, ip = _elements(box)
    nel = iv.shape[0]
    scale = 1.0 / (0.5 * (box.Lx + box.Lz))
    B, Z = 2 / box.hx * t["dNdr_V"], 2 / box.hz * t["dNdt_V"]
    W = box.hx * box.hz / 4 * t["weightq"]
    e = s["etaq"] * W
    pair = lambda a, b: torch.einsum("qi,qj->qij", a, b).reshape(9, 81)
    K = torch.empty(nel, 9, 2, 9, 2, dtype=f64, device="cuda")
    K[:, :, 0, :, 0] = (e @ (2 * pair(B, B) + pair(Z, Z))).view(nel, 9, 9)
    K[:, :, 1, :, 1] = (e @ (2 * pair(Z, Z) + pair(B, B))).view(nel, 9, 9)
    K[:, :, 0, :, 1] = (e @ pair(Z, B)).view(nel, 9, 9)
    K[:, :, 1, :, 0] = (e @ pair(B, Z)).view(nel, 9, 9)
    K = K.view(nel, 18, 18)
    G = torch.empty(9, 2, 4, dtype=f64, device="cuda")
    G[:, 0], G[:, 1] = (-scale * torch.einsum("q,qk,qj->kj", W, D, t["N_P"]) for D in (B, Z))
    fixed = torch.stack([s["fix"][2 * iv], s["fix"][2 * iv + 1]], 2).view(nel, 18)
    keep = ~fixed
    eye = torch.eye(18, dtype=torch.bool, device="cuda")
    K = torch.where((keep[:, :, None] & keep[:, None, :]) | eye, K, 0.0)
    G = torch.where(keep[:, :, None], G.view(18, 4)[None], 0.0)
    load = torch.einsum("eq,qk->ek", s["rhoq"] * W * s["gzq"], t["N_V"])
    f = torch.zeros(2 * (2 * box.nelx + 1) * (2 * box.nelz + 1), dtype=f64, device="cuda")
    f.index_add_(0, (2 * iv + 1).reshape(-1), load.reshape(-1))
    f = torch.where(s["fix"], 0.0, f)
    out = dict(rhs_f=f)
    if case["blocks"]:
        M = torch.einsum("q,qi,qj->ij", W, t["N_P"], t["N_P"])
        out.update(VV_K=K.reshape(-1), VV_M=M.expand(nel, 4, 4).reshape(-1),
                   VV_M_eta=(M[None] / s["eta_e"][:, None, None]).reshape(-1))
        # G and its transpose are laid out row by row, G_j of row i
        out.update(VV_G=G.reshape(-1))
    else:
        both = torch.stack([G, G], 3).reshape(nel, 18, 8)     # each entry, and its transpose's
        out["VV_Stokes"] = torch.cat([K, both], 2).reshape(-1)
    return out


def _exact_energy(case, seed):
    s = _prepare_energy(case, seed)
    box, t, q, dt = s["box"], _host_tables(), s["q"], s["dt"]
    iv, _ = _elements(box)
    N, B, Z = t["N_V"], 2 / box.hx * t["dNdr_V"], 2 / box.hz * t["dNdt_V"]
    W = box.hx * box.hz / 4 * t["weightq"]
    pair = lambda a, b: torch.einsum("qi,qj->qij", a, b).reshape(9, 81)
    cap = q["hcapaq"] * W                         # the reference density is 1
    mass = (cap @ pair(N, N)).view(-1, 9, 9)
    K = ((cap * q["uq"]) @ pair(N, B) + (cap * q["wq"]) @ pair(N, Z)
         + (q["hcondq"] * W) @ (pair(B, B) + pair(Z, Z))).view(-1, 9, 9)
    src = q["hprodq"] * W
    if case["formulation"] == "EBA":              # shear heating and adiabatic heating
        xx, zz, xz = q["exxq"], q["ezzq"], q["exzq"]
        src = src + 2 * q["etaq"] * (2 / 3 * (xx * xx + zz * zz - xx * zz) + 2 * xz * xz) * W
        src = src - 10.0 * q["alphaq"] * q["Tq"] * q["wq"] * W
    A, R = mass + dt / 2 * K, mass - dt / 2 * K
    nn = s["T"].shape[0]
    flat = iv.reshape(-1)
    spread = lambda be: torch.zeros(nn, dtype=f64, device="cuda").index_add_(0, flat, be.reshape(-1))
    mul = lambda M, v: spread(torch.einsum("eij,ej->ei", M, v[iv]))
    fix, val = s["fixT"], s["valT"]
    free = lambda v: torch.where(fix, 0.0, v)
    diag = spread(torch.diagonal(A, dim1=1, dim2=2))
    b = free(mul(R, s["T"]) + spread(dt * src @ N) - mul(A, val))
    op = lambda v: free(mul(A, v)) / diag
    x = free(s["T"])                              # BiCGSTAB on the free nodes, to rounding
    res = b / diag - op(x)
    r0, p, rho = res.clone(), res.clone(), torch.dot(res, res)
    goal = 1e-15 * float(x.norm())
    for _ in range(100):
        if float(res.norm()) <= goal:
            break
        v = op(p)
        alpha = rho / torch.dot(r0, v)
        h = res - alpha * v
        th = op(h)
        om = torch.dot(th, h) / torch.dot(th, th)
        x = x + alpha * p + om * h
        res = h - om * th
        rho2 = torch.dot(r0, res)
        p = res + rho2 / rho * (alpha / om) * (p - om * v)
        rho = rho2
    return dict(T=x + val, rhs=torch.where(fix, diag * val, b))


def _exact_train(case, seed):
    s = _prepare_train(case, seed)
    b, n, net = s["b"], s["n"], s["net"]
    conv = torch.nn.functional.conv2d

    def layer(l, x, relu=True):
        w = l.w16[:, :9 * l.cin].to(f64).view(l.cout, 3, 3, l.cin).permute(0, 3, 1, 2)
        y = conv(x, w, l.b.to(f64), padding=1)
        return y.relu() if relu else y

    x = s["X"].to(f64).permute(0, 3, 1, 2)
    skips = []
    for i, (c1, c2) in enumerate(net.enc):
        x = layer(c2, layer(c1, x))
        if i < len(net.enc) - 1:
            skips.append(x)
            x = torch.nn.functional.avg_pool2d(x, 2)
    for (c1, c2), skip in zip(net.dec, reversed(skips)):
        x = torch.cat([x.repeat_interleave(2, 2).repeat_interleave(2, 3), skip], 1)
        x = layer(c2, layer(c1, x))
    y = layer(net.head, x, relu=False)
    return dict(y=y.permute(0, 2, 3, 1).reshape(b * n * n, NOUT))


def exact(case, seed):
    """The outputs in 64 bits by plain torch; None for solves and whole steps, which it would take a
    direct factorisation to give."""
    f = dict(apply=_exact_apply, pic=_exact_pic, assemble=_exact_assemble, energy=_exact_energy,
             train=_exact_train).get(case["kind"])
    return f(case, seed) if f else None


# ---------------------------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "train":
        m, b, fl = case["n"], case["batch"], 0.0
        for level, layers in enumerate(([(2, 32), (32, 32), (96, 32), (32, 32), (32, NOUT)],
                                        [(32, 64), (64, 64), (192, 64), (64, 64)],
                                        [(64, 128), (128, 128), (384, 128), (128, 128)], [(128, 256), (256, 256)])):
            fl += sum(2.0 * 9 * a * c for a, c in layers) * b * (m >> level) ** 2
        weights = 1.93e6
        return {"bytes": b * m * m * (2 * 2 + 2 * 4 * NOUT) + weights * 4 * 7, "flops": 3 * fl}
    nel = case["nelx"] * case["nelz"]
    nn = (2 * case["nelx"] + 1) * (2 * case["nelz"] + 1)
    npp = (case["nelx"] + 1) * (case["nelz"] + 1)
    if kind == "step":
        part = nel * (16 if case["model"] == "fk" else 25)
        # positions, flags, reduced coordinates and element numbers in and out; the nodal fields in and out
        return {"bytes": 2 * (part * 37 + nn * 8 * 8 + (2 * nn + npp) * 8), "flops": 0}
    if kind == "cold":
        return {"bytes": nel * 80 + 2 * 8 * (2 * nn + npp), "flops": 0}
    if kind == "apply":
        size = 4 if case["precision"] == "f32" else 8
        return {"bytes": size * (2 * (2 * nn + npp) + 9 * nel), "flops": nel * 2 * 2 * (2 * 108 + 60)}
    if kind == "pic":
        n = nel * case["ppd"] ** 2
        return {"bytes": n * (21 + 11 * 8 + 4 + 17 + 17 + 16 + 20) + nn * 8 * (5 + 2 + 2) + nel * 24,
                "flops": n * (5 * 18 + 40 + 36 * case["rk"] * 2)}
    if kind == "assemble":
        size = 4 if case["precision"] == "f32" else 8
        return {"bytes": nel * (9 * 9 * 8 + 8 + (324 + 3 * 72 + 2 * 16 if case["blocks"] else 468) * size) + nn * 2 * 17
                + npp * 8, "flops": nel * 9 * (4 * 81 * 2 + 18 * 4)}
    fields = 14 if case["formulation"] == "EBA" else 9
    return {"bytes": nel * 9 * 8 * (fields + 3) + nn * (4 * 8 + 9), "flops": nel * 9 * 200}
