"""A barrier wait that runs out in a persistent CG or GMRES launch: the solve
returns LFX_TIMEOUT at the next look at its state (not after max_iter more
cycles on a barrier that is not ready), and the context goes on as before."""
import numpy as np
import pytest

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg
from lfric_core_b200 import workloads as wl

pytestmark = pytest.mark.gpu

MAX = 400
SOLVERS = {"cg": lambda s: lfx.ConjugateGradient(s.op, s.prec, 0.0, 0.0, MAX),
           "gmres": lambda s: lfx.GMRES(s.op, s.prec, 6, 0.0, 0.0, MAX)}


@pytest.mark.parametrize("name", SOLVERS)
def test_time_out_ends_the_solve(name):
    ctx = lfx.Context(0)  # its own: other tests' graphs keep their limit
    p = mg.w0_problem(24, 20, seed=3)  # past one cluster: a grid barrier
    s = wl.device_w0(ctx, p)
    b, x = s.vector(p.rhs), s.vector()
    # a limit of 0: the first poll that finds the barrier closed gives up
    ctx.set_wait_limit(0.0)
    solver = SOLVERS[name](s)
    n0 = ctx.launch_count()
    with pytest.raises(lfx.LfxError) as e:
        solver.apply(x, b)
    assert e.value.status == 6  # LFX_TIMEOUT
    # one cycle (GMRES(6): under 100 launches) or one launch, not MAX of them
    assert ctx.launch_count() - n0 < 150
    # the flag and the barrier words are ready: the next solves are as ever
    ctx.set_wait_limit(2.0)
    ctx.check_device_error()
    results = []
    for kernel in (-1, 1):
        ctx.set_apply_kernel(kernel)
        solver = type(solver)(s.op, s.prec, *((6,) if name == "gmres" else ()), 0.0, 0.0, 20)
        x.set_scalar(0.0)
        assert solver.apply(x, b).iterations == 20
        results.append(x.export_field())
    ctx.set_apply_kernel(-1)
    assert np.array_equal(*results)


def test_wait_limit_range(ctx):
    for bad in (-1.0, float("nan"), 61.0):
        with pytest.raises(lfx.LfxError):
            ctx.set_wait_limit(bad)
