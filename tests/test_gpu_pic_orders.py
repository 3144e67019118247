"""Particle kernels on orders, counts and alignments they branch on: bins in any memory order, longer
than a lane group and than the sorted length, inactive particles, arrays that start off a vector's
boundary, and element counts on both sides of the element projection's block size."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def swarm(nelx, nelz, n, order, seed=0, inactive=0.1):
    rng = np.random.default_rng(seed)
    nel = nelx * nelz
    iel = np.sort(rng.integers(0, nel, n)).astype(np.int32)
    if order == "crowded":                       # most particles in bins of about 80
        iel[: (4 * n) // 5] = rng.integers(0, min(nel, max(1, n // 100)), (4 * n) // 5)
        iel = np.sort(iel)
    if order in ("shuffled", "crowded"):
        iel = rng.permutation(iel)
    active = rng.random(n) >= inactive
    r, t = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    return iel.astype(np.int32), active, r, t, np.exp(rng.normal(0, 3, n)), rng.uniform(0.9, 1.1, n)


def dev(a, offset=0):
    """`a` on the device, starting `offset` entries into its allocation."""
    t = torch.as_tensor(a)
    buf = torch.empty(len(a) + offset, dtype=t.dtype, device="cuda")
    buf[offset:] = t.cuda()
    return buf[offset:]


@pytest.mark.parametrize("offset", [0, 1, 3])
@pytest.mark.parametrize("order", ["sorted", "shuffled", "crowded"])
@pytest.mark.parametrize("nelx,nelz,n", [(1, 1, 1), (3, 2, 101), (33, 31, 16385), (40, 30, 30000)])
def test_bins(nelx, nelz, n, order, offset):
    from meeuuw_b200 import ops
    iel, active, *_ = swarm(nelx, nelz, n, order)
    nel = nelx * nelz
    counts, offsets, perm = ops.bin_particles(nel, dev(active, offset), dev(iel, offset))
    want = np.bincount(iel[active], minlength=nel)
    assert np.array_equal(counts.cpu().numpy(), want)
    assert np.array_equal(offsets.cpu().numpy(), np.concatenate([[0], np.cumsum(want)]))
    idx = np.flatnonzero(active)
    assert np.array_equal(perm.cpu().numpy()[: len(idx)], idx[np.argsort(iel[idx], kind="stable")])


@pytest.mark.parametrize("averaging", ["arithmetic", "geometric", "harmonic"])
@pytest.mark.parametrize("order", ["sorted", "crowded"])
@pytest.mark.parametrize("nelx,nelz,n", [(7, 5, 900), (300, 260, 400000)])
def test_element_and_node_projections(nelx, nelz, n, order, averaging):
    """Element means as the sequential sums (bit for bit for the arithmetic one); nodal projections of all
    flavours against the exact-order path, to the rounding of reordered sums (1e-13)."""
    from meeuuw_b200 import _lib, ops
    iel, active, r, t, eta, rho = swarm(nelx, nelz, n, order)
    nel = nelx * nelz
    iel[: min(n, nel)] = np.arange(min(n, nel))             # no element empty
    active[: min(n, nel)] = True
    counts, offsets, perm = ops.bin_particles(nel, dev(active), dev(iel))
    rho_e, eta_e = ops.project_elements(nel, offsets, perm, dev(rho), dev(eta), averaging)
    s = np.zeros(nel)
    np.add.at(s, iel[active], rho[active])
    assert np.array_equal(rho_e.cpu().numpy(), s / np.bincount(iel[active], minlength=nel))
    fwd = {"arithmetic": lambda a: a, "geometric": np.log10, "harmonic": lambda a: 1 / a}[averaging]
    inv = {"arithmetic": lambda a: a, "geometric": lambda a: 10.0 ** a, "harmonic": lambda a: 1 / a}[averaging]
    m = np.zeros(nel)
    np.add.at(m, iel[active], fwd(eta[active]))
    want = inv(m / np.bincount(iel[active], minlength=nel))
    assert np.max(np.abs(eta_e.cpu().numpy() / want - 1)) < 1e-13
    box = _lib.box_of(nelx, nelz, 1.0, 1.0)
    for flavour in (1, 2):
        fields = [(dev(rho), "arithmetic"), (dev(eta), averaging), (dev(r), "arithmetic")]
        a = ops.project_nodes(box, flavour, fields, offsets, perm, dev(r), dev(t))
        b = ops.project_nodes(box, flavour, fields, offsets, perm, dev(r), dev(t), exact_order=True)
        for x, y in zip(a, b):
            assert float((x - y).abs().max() / y.abs().max()) < 1e-13


def test_interp_material_pairs_equal_single():
    """The paired form (aligned arrays, even count) against the single one (arrays off a pair's boundary)."""
    from meeuuw_b200 import _lib, configs, ops
    nelx, nelz, n = 21, 17, 5000
    iel, active, r, t, *_ = swarm(nelx, nelz, n, "shuffled")
    box = _lib.box_of(nelx, nelz, 1.0, 1.0)
    nodal = {k: torch.rand((2 * nelx + 1) * (2 * nelz + 1), dtype=torch.float64, device="cuda")
             for k in ("exx", "ezz", "exz", "q", "T")}
    mat = np.random.default_rng(1).integers(0, 2, n).astype(np.int8)
    for cfg in (configs.fk_convection(8), configs.rayleigh_taylor(8)):
        res = []
        for off in (0, 1):
            out = {k: dev(np.zeros(n), off) for k in ("exx", "ezz", "exz", "p", "T", "rho", "eta", "hcond", "hcapa",
                                                      "hprod", "alpha")}
            ops.interp_material(box, dev(active, off), dev(r, off), dev(t, off), dev(iel, off), dev(mat, off), nodal,
                                ops.material_struct(cfg), out)
            res.append(out)
        for k in res[0]:
            assert torch.equal(res[0][k], res[1][k]), k
