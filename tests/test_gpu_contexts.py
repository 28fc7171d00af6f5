"""Solves of several contexts at once, each from a thread of its own: the bits of
a solve alone. Sizes whose grids share the device and sizes that queue for it."""
import threading

import numpy as np
import pytest

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg
from lfric_core_b200 import workloads as wl

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nl", [(8, 6), (10, 40), (12, 33), (24, 20)])
def test_cg_of_two_contexts(n, nl):
    p = mg.w0_problem(n, nl, seed=n)
    systems = [wl.device_w0(lfx.Context(0), p) for _ in range(2)]
    work = [(lfx.ConjugateGradient(s.op, s.prec, 1e-9, 0.0, 3000), s.vector(), s.vector(p.rhs))
            for s in systems]
    solver, x, b = work[0]
    systems[0].ctx.set_apply_kernel(1)  # the launch per phase
    solver.apply(x, b)
    systems[0].ctx.set_apply_kernel(-1)
    alone, got, start = x.export_field(), [[], []], threading.Barrier(2)

    def run(k):
        solver, x, b = work[k]
        start.wait()
        for _ in range(5):
            x.set_scalar(0.0)
            solver.apply(x, b)
            got[k].append(x.export_field())

    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(len(g) == 5 and all(np.array_equal(alone, v) for v in g) for g in got)
