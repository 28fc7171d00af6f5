"""GMRES with its Gram-Schmidt steps as persistent launches: bit for bit the
oracle's solve with less than one 2048-value chunk, a partial last chunk, several
chunks a block, and more chunks than a block's shared memory holds."""
import numpy as np
import pytest

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg
from lfric_core_b200 import workloads as wl
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nl,gcrk,cycles", [
    (3, 2, 1, 4), (4, 3, 10, 3), (8, 6, 3, 5), (17, 9, 24, 1), (40, 30, 6, 1), (96, 30, 3, 1)])
def test_gmres_bits(ctx, n, nl, gcrk, cycles):
    p = mg.w2_problem(n, nl, seed=n)
    s = wl.device_w0(ctx, p)  # the diagonal preconditioner, on the W2 operator
    npc, cic = p.mesh.colour_lookup()
    op = orc.LmaOperator(p.ncell_2d, nl, 6, 6, p.map, p.map, p.undf, p.undf, p.lma, npc, cic)
    x_o, i_o = orc.solve("gmres", op, orc.Preconditioner.diagonal(op.diagonal()), p.rhs,
                         r_tol=1e-12, a_tol=0.0, max_iter=cycles, gcrk=gcrk)
    x, b = s.vector(), s.vector(p.rhs)
    g = lfx.GMRES(s.op, s.prec, gcrk, 1e-12, 0.0, cycles)
    info = g.apply(x, b)
    assert info.iterations == i_o.iterations and info.converged == i_o.converged
    assert np.array_equal(x.export_field().view(np.int64), x_o.view(np.int64))
    # again, from another start, on the same graph and barrier words
    x0 = mg.normal(3, p.undf)
    x_o, _ = orc.solve("gmres", op, orc.Preconditioner.diagonal(op.diagonal()), p.rhs, x0=x0,
                       r_tol=1e-12, a_tol=0.0, max_iter=cycles, gcrk=gcrk)
    x.import_field(x0)
    g.apply(x, b)
    assert np.array_equal(x.export_field().view(np.int64), x_o.view(np.int64))
