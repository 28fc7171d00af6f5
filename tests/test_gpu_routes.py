"""That a call takes the form its size is meant for, by the launches it counts, and
inputs that the forms' own tests leave out."""
import numpy as np
import pytest
import torch

from lfric_core_b200 import lfx
from lfric_core_b200 import meshgen as mg
from lfric_core_b200 import workloads as wl
from test_gpu_mrhs import mrhs_apply

pytestmark = pytest.mark.gpu


def launches(ctx, call):
    call()  # a first call may build tables
    n0 = ctx.launch_count()
    call()
    return ctx.launch_count() - n0


@pytest.mark.parametrize("n,nl,one", [
    (8, 6, True), (24, 20, True), (12, 40, True), (24, 70, False)])  # the last: 124 MB
def test_cg_is_one_launch(ctx, n, nl, one):
    p = mg.w0_problem(n, nl, seed=2)
    s = wl.device_w0(ctx, p)
    cg, b, x = lfx.ConjugateGradient(s.op, s.prec, 1e-8, 0.0, 50), s.vector(p.rhs), s.vector()
    count = launches(ctx, lambda: cg.apply(x, b))
    # the state in, the solve, the state out; otherwise some launches an iteration
    assert count == 3 if one else count > 200


@pytest.mark.parametrize("nl,scatter", [(19, False), (21, True)])  # 23.3 MB and 25.8 MB
def test_untuned_apply_scatters_from_24_mb(ctx, nl, scatter):
    p = mg.w0_problem(20, nl, seed=3)
    op = wl._lma(ctx, p, lfx.R64)
    x, y = lfx.FieldVector.from_array(ctx, mg.normal(5, p.undf)), lfx.FieldVector(ctx, [p.undf])
    colours = int(np.count_nonzero(p.mesh.colour_lookup()[0]))
    assert colours > 1
    assert launches(ctx, lambda: op.apply(x, y)) == (colours if scatter else 1)


def test_batch_groups_at_the_tested_size(ctx):
    """The sizes of test_gpu_batch_groups: 16 chunks of 4096 a block of the largest
    grid (three blocks an SM) and more."""
    undf = (6 * 47 * 47 + 2) * 71
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert 32 * ((undf + 4095) // 4096) >= 16 * 3 * sms


def test_mrhs_kinds_and_autotune_give_the_same_bits(ctx):
    p = mg.w0_problem(6, 9, seed=4)
    s = wl.device_w0(ctx, p)
    X = np.random.default_rng(4).standard_normal((p.undf, 32)).astype(np.float32)
    tf32, bf16 = (lfx.MultiRhsOperator(s.op, k, 32) for k in (lfx.MRHS_TF32, lfx.MRHS_BF16))
    Y = mrhs_apply(ctx, tf32, X)
    assert np.array_equal(Y, mrhs_apply(ctx, bf16, X))
    tf32.autotune(reps=2)
    assert np.array_equal(Y, mrhs_apply(ctx, tf32, X))


@pytest.mark.parametrize("n,nl", [(8, 6), (16, 12), (10, 40)])
@pytest.mark.parametrize("value", [np.inf, np.nan, 1e300])
def test_persistent_cg_beyond_numbers(ctx, n, nl, value):
    p = mg.w0_problem(n, nl, seed=8)
    s = wl.device_w0(ctx, p)
    rhs = p.rhs.copy()
    rhs[p.undf // 3] = value  # (1e300: its square overflows)
    b, x, got = s.vector(rhs), s.vector(), []
    for kernel in (-1, 1):
        cg = lfx.ConjugateGradient(s.op, s.prec, 1e-8, 0.0, 100)
        x.set_scalar(0.0)
        ctx.set_apply_kernel(kernel)
        status = 0
        try:
            cg.apply(x, b)
        except lfx.LfxError as e:
            status = e.status
        finally:
            ctx.set_apply_kernel(-1)
        got.append((status, repr(cg.last_info.as_dict()), x.export_field()))
    assert got[0][:2] == got[1][:2]
    assert np.array_equal(got[0][2], got[1][2], equal_nan=True)


def test_gmres_fp32_past_shared_memory(ctx):
    """Thirty chunks of w a block where shared memory holds 28, in FP32, on a
    diagonal operator with entries in [1, 2]: eight steps reduce the residual by
    2 (3 - sqrt 8)^8 = 1.5e-6, so one cycle or two reach 1e-5 and the solution is
    within 2e-5 (and FP32's 2e-6) of b / a."""
    nc, nl = 10000, 900
    n = nc * nl
    a = 1.0 + np.random.default_rng(1).random(n)
    m = (np.arange(nc, dtype=np.int32) * nl + 1).reshape(nc, 1)
    cells = np.arange(1, nc + 1, dtype=np.int32).reshape(nc, 1)
    op = lfx.LmaOperator(ctx, nc, nl, 1, 1, m, m, n, n, a, np.array([nc], np.int32), cells,
                         precision=lfx.R32)
    rhs = np.random.default_rng(2).standard_normal(n)
    b, x = lfx.FieldVector.from_array(ctx, rhs, lfx.R32), lfx.FieldVector(ctx, [n], lfx.R32)
    x.set_scalar(0.0)
    info = lfx.GMRES(op, lfx.NullPreconditioner(ctx), 8, 1e-5, 0.0, 10).apply(x, b)
    assert info.converged and info.iterations <= 2
    want = rhs / a
    assert np.linalg.norm(x.export_field() - want) <= 2.2e-5 * np.linalg.norm(want)
