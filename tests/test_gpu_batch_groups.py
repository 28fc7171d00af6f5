"""A batch with enough chunks takes several of them an item: the bits of each
slot stay those of the slot alone."""
import pytest

from test_gpu_batch import run_batch, same, w0_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nl,count", [(47, 70, 32)])  # 230 chunks a slot: groups of 4, 2 left over
def test_grouped_chunks_give_the_bits_of_a_slot_alone(ctx, n, nl, count):
    big, small = w0_system(ctx, n, nl, 1), w0_system(ctx, 5, 7, 2)
    systems, tols = [big] * count + [small], [1e-6] * count + [1e-9]
    mixed = run_batch(ctx, systems, tols)
    for s, tol, got in ((big, 1e-6, mixed[:count]), (small, 1e-9, mixed[count:])):
        x, info = run_batch(ctx, [s], [tol])[0]
        for xm, im in got:
            assert same(x, xm)
            assert im["iterations"] == info["iterations"]
