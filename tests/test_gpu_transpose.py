"""The transpose apply of operators on faces (W2 -> W3 divergence, square W2)
against the oracle's transpose_matrix_vector, bit for bit in FP64, over column
heights around the 32 and 64 levels of a pass and odd panels; FP32 against the FP64
product within its rounding (at most 12 products of both factors rounded, u = 2^-24:
16 u |A^T| |x|)."""
import numpy as np
import pytest

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg
from oracle import oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nl", [(2, 1), (3, 31), (4, 32), (5, 63), (3, 64), (4, 70), (2, 97)])
@pytest.mark.parametrize("square", [False, True])
def test_transpose_on_faces(ctx, n, nl, square):
    p = mg.w2_problem(n, nl, seed=7, keep_parts=True)
    npc, cic = p.mesh.colour_lookup()
    if square:
        # not symmetric: the local matrices scaled row by row
        lma = (p.lma.reshape(6, 6, -1) * np.arange(1, 7)[None, :, None]).reshape(-1).copy()
        args = (6, 6, p.map, p.map, p.undf, p.undf, lma)
    else:
        lma = p.extra["div"]
        args = (1, 6, p.extra["map_w3"], p.map, p.extra["undf_w3"], p.undf, lma)
    x = mg.normal(11, args[4])
    o = orc.LmaOperator(p.ncell_2d, nl, *args, npc, cic, transpose=True)
    want = o.apply(x)
    op = lfx.LmaOperator(ctx, p.ncell_2d, nl, *args, npc, cic)
    X, Y = lfx.FieldVector.from_array(ctx, x), lfx.FieldVector(ctx, [p.undf])
    op.apply_transpose(X, Y)
    assert np.array_equal(Y.export_field().view(np.int64), want.view(np.int64))
    op32 = op.like(lma, lfx.R32)
    X = lfx.FieldVector.from_array(ctx, x, lfx.R32)
    Y = lfx.FieldVector(ctx, [p.undf], lfx.R32)
    op32.apply_transpose(X, Y)
    oa = orc.LmaOperator(p.ncell_2d, nl, *args[:6], np.abs(lma), npc, cic,
                         transpose=True)
    bound = 16 * 2.0 ** -24 * oa.apply(np.abs(x))
    assert np.all(np.abs(Y.export_field() - want) <= bound)
