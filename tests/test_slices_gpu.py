"""Batches of several slices of 8 tokens in one launch (a grid row per slice): matrices whose slices share one wave of
CTAs, matrices taller than that, and token counts that leave 0 .. 7 tokens for the smaller forms, all equal to the
one-token kernel bit for bit (the contract of tm_metal.h:160-164)."""
import numpy as np
import pytest

from tuckmill_b200 import testing as T

pytestmark = pytest.mark.gpu


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
