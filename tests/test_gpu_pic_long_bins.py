"""Bins around and past the lengths the particle kernels branch on: the sort by rank, by merge exchange, the rounds
of 16 and of 1024 particles of the projections, all nodal flavours, all capacities for fields."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def lengths(kind, nel, rng):
    if kind == "mixed":                          # one bin empty, some short, some at the edges, one very long
        m = rng.choice([1, 3, 15, 16, 17, 63, 64, 65, 128, 129, 300], nel)
        m[nel // 2] = 3000
        m[0] = 0 if nel > 1 else m[0]
        return m
    return np.full(nel, int(kind))


def swarm(kind, nel, order, seed=0):
    rng = np.random.default_rng(seed)
    iel = np.repeat(np.arange(nel), lengths(kind, nel, rng)).astype(np.int32)
    if order == "shuffled":
        iel = rng.permutation(iel)
    if order == "reversed":
        iel = iel[::-1].copy()
    n = len(iel)
    return iel, rng.uniform(-1, 1, n), rng.uniform(-1, 1, n), np.exp(rng.normal(0, 3, n)), rng.uniform(0.9, 1.1, n)


def bins(iel, nel):
    from meeuuw_b200 import ops
    active = torch.ones(len(iel), dtype=torch.bool, device="cuda")
    return ops.bin_particles(nel, active, torch.as_tensor(iel).cuda())


@pytest.mark.parametrize("order", ["sorted", "shuffled", "reversed"])
@pytest.mark.parametrize("kind", ["64", "65", "100", "257", "mixed"])
def test_bins_are_sorted(kind, order):
    nel = 33 * 7
    iel = swarm(kind, nel, order)[0]
    counts, offsets, perm = bins(iel, nel)
    want = np.bincount(iel, minlength=nel)
    assert np.array_equal(counts.cpu().numpy(), want)
    assert np.array_equal(offsets.cpu().numpy(), np.concatenate([[0], np.cumsum(want)]))
    assert np.array_equal(perm.cpu().numpy()[: len(iel)], np.argsort(iel, kind="stable"))


@pytest.mark.parametrize("nel", [1, 63, 64, 65, 40 * 33, 300 * 260])
@pytest.mark.parametrize("kind", ["1", "4", "16", "25", "100", "mixed"])
def test_element_means(kind, nel):
    """The arithmetic mean is the sequential sum's, bit for bit; the geometric one to 1e-13 (its transform)."""
    from meeuuw_b200 import ops
    if nel > 10000 and kind in ("100", "mixed"):
        nel = 70 * 70
    iel, _, _, eta, rho = swarm(kind, nel, "shuffled")
    counts, offsets, perm = bins(iel, nel)
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rho_e, eta_e = ops.project_elements(nel, offsets, perm, torch.as_tensor(rho).cuda(), torch.as_tensor(eta).cuda(),
                                        "geometric", err=err)
    cnt = np.bincount(iel, minlength=nel)
    s, l = np.zeros(nel), np.zeros(nel)
    np.add.at(s, iel, rho)
    np.add.at(l, iel, np.log10(eta))
    full = cnt > 0
    assert np.array_equal(rho_e.cpu().numpy()[full], s[full] / cnt[full])
    assert np.max(np.abs(eta_e.cpu().numpy()[full] / 10.0 ** (l[full] / cnt[full]) - 1)) < 1e-13
    assert (int(err.item()) != 0) == (not full.all())


@pytest.mark.parametrize("nfield", [1, 2, 3, 5, 8])
@pytest.mark.parametrize("flavour", [1, 2, 3, 4])
@pytest.mark.parametrize("order", ["sorted", "shuffled"])
def test_node_projections(order, flavour, nfield):
    """All flavours and field counts with several rounds a bin against the exact-order path, to the rounding of
    reordered sums (1e-13)."""
    from meeuuw_b200 import _lib, ops
    nelx, nelz = 35, 9
    iel, r, t, eta, rho = swarm("40", nelx * nelz, order)
    counts, offsets, perm = bins(iel, nelx * nelz)
    D = lambda a: torch.as_tensor(a).cuda()
    averaging = ["arithmetic", "geometric", "harmonic"]
    fields = [(D(rho if f % 2 else eta), averaging[f % 3]) for f in range(nfield)]
    box = _lib.box_of(nelx, nelz, 1.0, 1.0)
    a = ops.project_nodes(box, flavour, fields, offsets, perm, D(r), D(t))
    b = ops.project_nodes(box, flavour, fields, offsets, perm, D(r), D(t), exact_order=True)
    for x, y in zip(a, b):
        assert float((x - y).abs().max() / y.abs().max()) < 1e-13


def test_node_projection_of_a_tall_mesh():
    """A column of more tiles than a launch has in its second dimension."""
    from meeuuw_b200 import _lib, ops
    nelx, nelz = 1, 530000
    iel, r, t, eta, rho = swarm("1", nelx * nelz, "sorted")
    counts, offsets, perm = bins(iel, nelx * nelz)
    D = lambda a: torch.as_tensor(a).cuda()
    fields = [(D(rho), "arithmetic"), (D(eta), "geometric")]
    box = _lib.box_of(nelx, nelz, 1.0, 1.0 * nelz)
    a = ops.project_nodes(box, 2, fields, offsets, perm, D(r), D(t))
    b = ops.project_nodes(box, 2, fields, offsets, perm, D(r), D(t), exact_order=True)
    for x, y in zip(a, b):
        assert float((x / y - 1).abs().max()) < 1e-12
