"""The apply of an operator nobody tuned: the same bits as the register gather on
both sides of the line where it takes the cell scatter (a 24 MB matrix)."""
import numpy as np
import pytest

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg
from lfric_core_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("space,n,nl,bits", [
    ("w0", 20, 19, 64), ("w0", 20, 21, 64), ("w0", 25, 33, 32), ("w2", 24, 24, 64),
    ("w2", 24, 25, 64), ("w2", 25, 45, 32)])
def test_default_apply_bits(ctx, space, n, nl, bits):
    p = (mg.w0_problem if space == "w0" else mg.w2_problem)(n, nl, seed=3)
    prec = lfx.R64 if bits == 64 else lfx.R32
    op = wl._lma(ctx, p, prec)
    x = lfx.FieldVector.from_array(ctx, mg.normal(5, p.undf), prec)
    y, z = lfx.FieldVector(ctx, [p.undf], prec), lfx.FieldVector(ctx, [p.undf], prec)
    op.apply(x, y)
    ctx.set_apply_kernel(1)
    try:
        op.apply(x, z)
    finally:
        ctx.set_apply_kernel(-1)
    assert np.array_equal(y.export_field(), z.export_field())
