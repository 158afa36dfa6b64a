"""The multiply for a few rows of activations (tm_cuda_q8_0_gemm_rows) at the edges of its tiles: against an
f16-operand reference (x and d*q rounded once each) to accumulation error, and against the oracle."""
import numpy as np
import pytest

from conftest import rel_err
from tuckmill_b200 import cuda, testing as T

pytestmark = pytest.mark.gpu


def f16_profile_reference(raw, X):
    w16 = T.q8_0_dequant(raw).astype(np.float16).astype(np.float64)
    return X.astype(np.float16).astype(np.float64) @ w16.T


# rows around whole 32-row units, cols from one chunk (fewer than warps) to eight K parts, 1..32 tokens
@pytest.mark.parametrize("rows,cols,batch", [(1, 64, 1), (31, 64, 2), (33, 128, 8), (40, 576, 9), (1024, 1024, 16),
                                             (1024, 2048, 17), (1152, 6912, 24), (4096, 12288, 32), (6144, 4096, 32),
                                             (20000, 1024, 25), (96, 16384, 31)])
def test_gemm_rows_equals_the_f16_profile(ctx, oracle, rows, cols, batch):
    raw = T.q8_0_matrix(11, rows + cols, rows, cols)
    X = T.activations(11, 5, batch * cols).reshape(batch, cols)
    w, xb = ctx.q8_0_matrix(raw, rows, cols), ctx.floats(X)
    base = T.activations(11, 9, batch * rows).reshape(batch, rows)
    yb = ctx.floats(base)
    ctx.q8_0_gemm_rows(w, xb, rows, cols, batch, [yb], [rows])
    Y = yb.download(0, batch * rows * 4, np.float32).reshape(batch, rows)
    assert rel_err(Y, f16_profile_reference(raw, X)) <= 2e-5
    assert float(np.max(np.abs(Y - oracle.matmul_q8_0(raw, rows, cols, X)))) <= 2e-2
    yb.upload(0, base)
    ctx.q8_0_gemm_rows(w, xb, rows, cols, batch, [yb], [rows], epilogue=cuda.EPI_ADD)
    np.testing.assert_array_equal(yb.download(0, batch * rows * 4, np.float32).reshape(batch, rows), base + Y)


@pytest.mark.parametrize("act", [cuda.EPI_SILU_MUL_F16, cuda.EPI_GELU_MUL_F16])
@pytest.mark.parametrize("width,cols,batch", [(16, 64, 1), (3072, 1024, 32), (6912, 1152, 13)])
def test_gemm_rows_gated_output_feeds_the_next_multiply(ctx, act, width, cols, batch):
    eps = 1e-6
    raw, nxt = T.q8_0_matrix(12, 1, 2 * width, cols), T.q8_0_matrix(12, 2, 64, width) if width % 64 == 0 else None
    X = T.activations(12, 5, batch * cols).reshape(batch, cols)
    nw = (1 + 0.1 * T.activations(12, 6, cols)).astype(np.float32)
    xin = X / np.sqrt((X.astype(np.float64) ** 2).mean(axis=1, keepdims=True) + eps) * nw
    gu = f16_profile_reference(raw, xin.astype(np.float32))
    g, u = gu[:, :width], gu[:, width:]
    h = (g / (1 + np.exp(-g)) if act == cuda.EPI_SILU_MUL_F16 else
         0.5 * g * (1 + np.tanh(0.7978845608028654 * (g + 0.044715 * g ** 3)))) * u
    w, hb = ctx.q8_0_matrix(raw, 2 * width, cols), ctx.buffer(batch * width * 2)
    ctx.q8_0_gemm_rows(w, ctx.floats(X), 2 * width, cols, batch, [hb], [width], cuda.PRO_RMSNORM, ctx.floats(nw), eps, act)
    got = hb.download(0, batch * width * 2, np.float16).reshape(batch, width)
    assert rel_err(got.astype(np.float64), h) <= 2e-3
    if nxt is not None:
        y = ctx.buffer(batch * 64 * 4)
        ctx.q8_0_gemm_rows(ctx.q8_0_matrix(nxt, 64, width), hb, 64, width, batch, [y], [64], cuda.PRO_F16)
        assert rel_err(y.download(0, batch * 256, np.float32).reshape(batch, 64), f16_profile_reference(nxt, got)) <= 2e-5


def test_gemm_rows_parts_and_limits(ctx):
    raw = T.q8_0_matrix(13, 1, 160, 128)
    X = T.activations(13, 5, 3 * 128).reshape(3, 128)
    w, xb = ctx.q8_0_matrix(raw, 160, 128), ctx.floats(X)
    ys = [ctx.buffer(3 * n * 4) for n in (64, 32, 64)]
    ctx.q8_0_gemm_rows(w, xb, 160, 128, 3, ys, [64, 32, 64])
    got = np.concatenate([y.download(0, 3 * n * 4, np.float32).reshape(3, n) for y, n in zip(ys, (64, 32, 64))], axis=1)
    assert rel_err(got, f16_profile_reference(raw, X)) <= 2e-5
    for rows_of, batch in (([48, 48, 64], 3), ([64, 32, 64], 33)):
        with pytest.raises(cuda.CudaError):
            ctx.q8_0_gemm_rows(w, xb, 160, 128, batch, ys, rows_of)


# X read where it lies: units of one part and of several, warps without a chunk, more units than find a place at once;
# binary16 rows that lie on a 16-byte boundary only take half-width loads
@pytest.mark.parametrize("rows,cols,batch", [(64, 64, 1), (1024, 3072, 32), (1056, 6912, 7), (4096, 4096, 24), (9504, 576, 31),
                                             (9472, 64, 8), (9504, 5120, 8), (9504, 5120, 9)])
def test_gemm_rows_x_at_either_alignment(ctx, rows, cols, batch, staged=False):
    raw = T.q8_0_matrix(14, rows + cols, rows, cols)
    X = T.activations(14, 5, batch * cols).reshape(batch, cols).astype(np.float16)
    w, yb = ctx.q8_0_matrix(raw, rows, cols), ctx.buffer(batch * rows * 4)
    flat = ctx.buffer(batch * cols * 2 + 32)
    got = []
    for off in (0, 16):
        x = flat.view(off, batch * cols * 2)
        x.upload(0, X)
        yb.zero()
        ctx.q8_0_gemm_rows(w, x, rows, cols, batch, [yb], [rows], cuda.PRO_F16)
        got.append(yb.download(0, batch * rows * 4, np.float32).reshape(batch, rows))
    assert (ctx.gemm_rows_last_form() < 0) == staged
    assert rel_err(got[0], f16_profile_reference(raw, X)) <= 2e-5
    np.testing.assert_array_equal(got[0], got[1])
    base = T.activations(14, 9, batch * rows).reshape(batch, rows)
    yb.upload(0, base)
    ctx.q8_0_gemm_rows(w, x, rows, cols, batch, [yb], [rows], cuda.PRO_F16, epilogue=cuda.EPI_ADD)
    np.testing.assert_array_equal(yb.download(0, batch * rows * 4, np.float32).reshape(batch, rows), base + got[0])


# X staged for CTAs that serve several units (up to 8 tokens, up to 16 in a narrow matrix): either side of every line, fewer
# chunks than warps, one round of units and many, a last unit that is not whole
@pytest.mark.parametrize("rows,cols,batch,staged", [(9472, 512, 8, False), (9473, 512, 8, True), (9473, 576, 8, False),
                                                    (13632, 1920, 8, False), (13632, 1984, 8, True), (11840, 5952, 8, False),
                                                    (11840, 6080, 8, True), (9504, 64, 8, True), (12007, 64, 3, True), (50001, 704, 5, True),
                                                    (11872, 8192, 1, True), (13632, 1984, 9, False), (9472, 512, 9, False),
                                                    (9473, 512, 9, True), (20481, 192, 16, True), (9473, 576, 16, False),
                                                    (9473, 512, 17, False)])
def test_gemm_rows_with_x_staged(ctx, rows, cols, batch, staged):
    test_gemm_rows_x_at_either_alignment(ctx, rows, cols, batch, staged)


def test_gemm_rows_staged_in_parts_and_gated(ctx):
    rows, cols, batch = 32768, 1088, 6
    raw = T.q8_0_matrix(15, 1, rows, cols)
    X = T.activations(15, 5, batch * cols).reshape(batch, cols)
    w, xb, part_rows = ctx.q8_0_matrix(raw, rows, cols), ctx.floats(X), [32, 16384, 16352]
    ys = [ctx.buffer(batch * n * 4) for n in part_rows]
    want = f16_profile_reference(raw, X)
    ctx.q8_0_gemm_rows(w, xb, rows, cols, batch, ys, part_rows)
    assert ctx.gemm_rows_last_form() < 0
    got = np.concatenate([y.download(0, batch * n * 4, np.float32).reshape(batch, n) for y, n in zip(ys, part_rows)], axis=1)
    assert rel_err(got, want) <= 2e-5
    h, (g, u) = ctx.buffer(batch * rows), np.split(want, 2, axis=1)
    ctx.q8_0_gemm_rows(w, xb, rows, cols, batch, [h], [rows // 2], epilogue=cuda.EPI_SILU_MUL_F16)
    assert ctx.gemm_rows_last_form() < 0
    assert rel_err(h.download(0, batch * rows, np.float16).reshape(batch, rows // 2).astype(np.float64), g / (1 + np.exp(-g)) * u) <= 2e-3
