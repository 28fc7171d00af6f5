"""The persistent conjugate gradient launch against the launch per phase (taken
when an apply kernel is forced): the same bits, iteration counts and norms, at
the edges of its column packing (heights 8, 16 and 32 lanes, taller columns), on
one cluster and on the whole grid, from any starting point and over several
launches."""
import numpy as np
import pytest

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg
from lfric_core_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def solve(ctx, s, b, x0, kernel, **kw):
    args = dict(r_tol=1e-9 if s.precision == lfx.R64 else 1e-5, a_tol=0.0, max_iter=3000)
    args.update(kw)
    cg = lfx.ConjugateGradient(s.op, s.prec, args.pop("r_tol"), args.pop("a_tol"),
                               args.pop("max_iter"), **args)
    x = s.vector(x0)
    ctx.set_apply_kernel(kernel)
    try:
        info = cg.apply(x, b)
    finally:
        ctx.set_apply_kernel(-1)
    return x.export_field(), info.as_dict()


def check(ctx, s, p, x0=None, **kw):
    x0 = np.zeros(p.undf) if x0 is None else x0
    b = s.vector(p.rhs)
    (xa, ia), (xb, ib) = (solve(ctx, s, b, x0, k, **kw) for k in (-1, 1))
    assert repr(ia) == repr(ib)  # (as text: a NaN norm is the same NaN)
    nan = np.isnan(xa)
    assert np.array_equal(nan, np.isnan(xb))
    assert np.array_equal(xa[~nan].view(np.int64), xb[~nan].view(np.int64))
    return ia


@pytest.mark.parametrize("space,n,nl,bits", [
    ("w0", 2, 1, 64), ("w0", 4, 6, 64), ("w0", 5, 7, 32), ("w0", 6, 8, 64), ("w0", 9, 15, 64),
    ("w0", 7, 16, 32), ("w0", 12, 31, 64), ("w0", 10, 32, 64), ("w0", 6, 65, 32), ("w0", 24, 20, 64),
    ("w0", 37, 23, 32), ("w2", 3, 2, 64), ("w2", 8, 7, 32), ("w2", 11, 16, 64), ("w2", 9, 40, 64),
    ("w2", 24, 20, 64)])
def test_persistent_cg_bits(ctx, space, n, nl, bits):
    p = (mg.w0_problem if space == "w0" else mg.w2_problem)(n, nl, seed=n + nl)
    s = wl.device_w0(ctx, p, lfx.R64 if bits == 64 else lfx.R32)
    assert check(ctx, s, p)["converged"] == 1


def test_persistent_cg_start_and_stop(ctx):
    p = mg.w0_problem(8, 6, seed=5)
    s = wl.device_w0(ctx, p)
    check(ctx, s, p, x0=mg.normal(9, p.undf))
    assert check(ctx, s, p, max_iter=1)["converged"] == 0
    assert check(ctx, s, p, r_tol=0.0, a_tol=1e-3)["converged"] == 1
    # past the iterations of one launch (the residual has long reached zero)
    i = check(ctx, s, p, r_tol=0.0, max_iter=2003, monitor_convergence=False)
    assert i["iterations"] == 2003
    # zero right-hand side: done before the first iteration
    b, x = s.vector(), s.vector()
    assert lfx.ConjugateGradient(s.op, s.prec, 1e-8, 0.0, 10).apply(x, b).iterations == 0
