"""Batches of several slices of 8 tokens in one launch (a grid row per slice): matrices whose slices share one wave of
CTAs, matrices taller than that, and token counts that leave 0 .. 7 tokens for the smaller forms, all equal to the
one-token kernel bit for bit (the contract of tm_metal.h:160-164)."""
import numpy as np
import pytest

from tuckmill_b200 import testing as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols", [(5, 4096), (1184, 4160), (1201, 6912), (4096, 12288), (32768, 4096), (32784, 4096)])
@pytest.mark.parametrize("prologue", ["none", "norm", "silu"])
def test_wide_matrices_of_one_token(ctx, oracle, rows, cols, prologue):
    """Row tiles shared by the warps of two CTAs: fewer tiles than clusters, one more than clusters, column counts that
    leave half a pair of chunks or a part of the last 4096, the tallest matrix of the form and the first beyond it;
    against the oracle and, bit for bit, two tokens of the batched form."""
    raw = T.q8_0_matrix(5, 6, rows, cols)
    w = ctx.q8_0_matrix(raw, rows, cols)
    x, p = T.activations(7, 8, 2 * cols).reshape(2, cols), T.activations(9, 10, 2 * cols).reshape(2, cols)
    if prologue == "norm":
        p[1] = p[0]
    code = {"none": 0, "norm": 1, "silu": 2}[prologue]
    y2, y1 = ctx.floats(np.ones(2 * rows, np.float32)), ctx.floats(np.ones(rows, np.float32))
    pro2 = ctx.floats(p[0] if prologue == "norm" else p.reshape(-1)) if code else None
    ctx.q8_0_gemm_fused(w, ctx.floats(x.reshape(-1)), y2, rows, cols, 2, code, pro2, 1e-6, 1)
    both = y2.download(0, 2 * rows * 4, np.float32).reshape(2, rows)
    for b in range(2):
        one = ctx.floats(np.ones(rows, np.float32))
        ctx.q8_0_gemv_fused(w, ctx.floats(x[b]), one, rows, cols, code, ctx.floats(p[b]) if code else None, 1e-6, 1)
        np.testing.assert_array_equal(one.download(0, rows * 4, np.float32), both[b])
    v = x[0].astype(np.float64)
    if prologue == "norm":
        v = v / np.sqrt((v * v).mean() + 1e-6) * p[0]
    elif prologue == "silu":
        v = v / (1 + np.exp(-v)) * p[0]
    want = 1 + oracle.matmul_q8_0(raw, rows, cols, v.astype(np.float32)[None])[0]
    assert np.abs(both[0] - want).max() <= 1e-4 * max(1.0, np.abs(want).max())


@pytest.mark.parametrize("f16", [False, True])
@pytest.mark.parametrize("rows,cols", [(24, 64), (4736, 96), (40009, 64), (300, 12288)])
@pytest.mark.parametrize("batch", [16, 25, 32])
def test_every_slice_is_the_one_token_kernel(ctx, f16, rows, cols, batch):
    x = T.activations(1, 2, batch * cols).reshape(batch, cols)
    if f16:
        w = ctx.from_array((T.normals(3, 77, 1, 0, rows * cols).reshape(rows, cols) * 0.25).astype(np.float16))
        gemm, gemv = ctx.f16_gemm, ctx.f16_gemv
    else:
        w = ctx.q8_0_matrix(T.q8_0_matrix(3, 4, rows, cols), rows, cols)
        gemm, gemv = ctx.q8_0_gemm, ctx.q8_0_gemv
    y, y1 = ctx.floats(np.full(batch * rows, np.nan, np.float32)), ctx.floats(np.zeros(rows, np.float32))
    gemm(w, ctx.floats(x.reshape(-1)), y, rows, cols, batch)
    got = y.download(0, batch * rows * 4, np.float32).reshape(batch, rows)
    for b in sorted({0, 7, 8, 15, batch - 1}):
        gemv(w, ctx.floats(x[b]), y1, rows, cols)
        np.testing.assert_array_equal(got[b], y1.download(0, rows * 4, np.float32), err_msg=f"token {b}")
