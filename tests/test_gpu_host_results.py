"""Scalar results that reach the host through its mapped memory: many in a row on
changing values, several fields, a field without values, and two contexts in turn."""
import numpy as np
import pytest

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg

pytestmark = pytest.mark.gpu


def test_results_in_a_row(ctx):
    other = lfx.Context(0)
    try:
        n = [5000, 1, 0, 2049]
        vs = []
        for c in (ctx, other):
            v = lfx.FieldVector(c, n)
            for f, k in enumerate(n):
                v.import_field(np.ones(k), f + 1)
            vs.append(v)
        for i in range(300):  # sums of whole numbers: exact
            for v in vs:
                v.set_scalar(float(i))
                assert v.dot(v) == i * i * sum(n)
                assert v.field_norm(4) == np.sqrt(float(i * i * 2049))
                assert v.field_norm(3) == 0.0
    finally:
        del vs, v
        other.close()
