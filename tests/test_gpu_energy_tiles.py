"""The matrix-free energy kernels at the edges of their tiles, against the element matrices.

Sizes: one element; one below, at and one above the element tile (odd rows are padded to an even
number of coefficients); more tiles than CTAs of a launch (1184); an operator buffer on an 8-byte boundary,
which the kernels read without TMA.  Tolerances as between the two forms elsewhere: right-hand side and
products 1e-12 of the largest entry (FP64, another association), solutions at rtol 1e-12 to 1e-10.
"""
import pytest
import torch

from conftest import rel_err
from test_gpu_energy_mf import H, _random_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nelx,nelz,shift", [(1, 1, 0), (15, 6, 0), (15, 7, 0), (16, 7, 0), (16, 8, 0), (17, 9, 0), (33, 1, 0), (1, 40, 0),
                                             (17, 9, 8), (16, 8, 8)])
@pytest.mark.parametrize("formulation", ["BA", "EBA"])
def test_energy_tiles(nelx, nelz, shift, formulation):
    from meeuuw_b200 import _lib, ops
    box, args = _random_case(nelx, nelz, formulation, 3 + nelx * nelz, "z")
    nb = _lib.lib().mw_energy_op_bytes(box)
    buf = torch.full((nb + 16,), 255, dtype=torch.uint8, device="cuda")[shift:shift + nb]   # NaN in the padding
    VV, rhs0 = ops.assemble_energy(box, 0, *args)
    op, rhs1 = ops.energy_op_setup(box, *args, op=buf)
    assert rel_err(H(rhs1), H(rhs0)) < 1e-12
    x = torch.randn(rhs0.numel(), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    assert rel_err(H(ops.energy_op_apply(box, op, x)), H(ops.energy_matvec(box, VV, x))) < 1e-12
    T0, T1 = args[0].clone(), args[0].clone()
    i0, r0 = ops.energy_solve(box, VV, rhs0, T0, rtol=1e-12, maxit=300)
    i1, r1 = ops.energy_op_solve(box, op, rhs1, T1, rtol=1e-12, maxit=300)
    assert r0 <= 1e-12 and r1 <= 1e-12 and abs(i1 - i0) <= 2
    assert rel_err(H(T1), H(T0)) < 1e-10
    assert ops.energy_device_info(box, op=True) == (i1, r1)


def test_energy_more_tiles_than_ctas():
    from meeuuw_b200 import ops
    box, args = _random_case(607, 297, "EBA", 9, "xz")
    VV, rhs0 = ops.assemble_energy(box, 0, *args)
    op, rhs1 = ops.energy_op_setup(box, *args)
    assert rel_err(H(rhs1), H(rhs0)) < 1e-12
    x = torch.randn(rhs0.numel(), dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    assert rel_err(H(ops.energy_op_apply(box, op, x)), H(ops.energy_matvec(box, VV, x))) < 1e-12
