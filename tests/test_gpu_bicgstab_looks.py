"""BiCGStab past the iterations after which the host looks at the state after two
graphs: the iterations and bits of a solve that looks after each (as it does when
applies are timed)."""
import numpy as np
import pytest

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg
from lfric_core_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iterations", [15, 16, 17, 20, 21, 24, 25, 33])
def test_long_bicgstab(ctx, iterations):
    p = mg.w2_problem(10, 8, seed=6)
    s = wl.device_w2(ctx, p)
    diag = lfx.DiagonalPreconditioner(ctx, s.diag)
    b, x, got = s.vector(p.rhs), s.vector(), []
    solver = lfx.BiCGStab(s.op, diag, 0.0, 0.0, iterations)
    for timed in (False, True):
        ctx.enable_apply_timing(timed)
        x.set_scalar(0.0)
        try:
            info = solver.apply(x, b)
        finally:
            ctx.enable_apply_timing(False)
        assert info.iterations == iterations
        got.append(x.export_field())
    assert np.array_equal(*got)
