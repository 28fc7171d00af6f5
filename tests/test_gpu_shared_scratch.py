"""A solver's captured graphs and the context's reduction scratch: a small
solver gives the same bits after a larger vector has made the scratch grow, and
writes nothing into memory that others have taken since."""
import numpy as np
import pytest

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg
from lfric_core_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make", [
    lambda s: lfx.GMRES(s.op, s.prec, 6, 1e-9, 0.0, 50),
    lambda s: lfx.BiCGStab(s.op, s.prec, 1e-9, 0.0, 200),
    lambda s: lfx.ConjugateGradient(s.op, s.prec, 1e-9, 0.0, 500)], ids=["gmres", "bicgstab", "cg"])
def test_graphs_survive_a_larger_scratch(make):
    ctx = lfx.Context(0)
    p = mg.w2_problem(9, 7, seed=4)
    s = wl.device_w2(ctx, p)
    solver, b, x = make(s), s.vector(p.rhs), s.vector()
    solver.apply(x, b)
    first = x.export_field()
    before = ctx.device_bytes()
    big = lfx.FieldVector(ctx, [6_000_000])  # 4 sums of 2930 chunks: past the first 8192 values
    assert ctx.device_bytes() - before > 8 * 6_000_000
    # takers of whatever memory the growth gave back (the scratch held 64 KB)
    takers = [lfx.FieldVector.from_array(ctx, np.full(8192, 7.0)) for _ in range(64)]
    for _ in range(2):
        x.set_scalar(0.0)
        solver.apply(x, b)
        assert np.array_equal(first, x.export_field())
    assert all(np.all(t.export_field() == 7.0) for t in takers)
