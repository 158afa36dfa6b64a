"""Split-K sums of the tcgen05 multiply taken by groups of 32 tokens: fewer groups than parts and more, a last group of one
token, a second token tile with one group, row tiles that end inside the matrix; repeated calls leave the counters at
zero, so the results are the same bits, and the residual form adds to them."""
import numpy as np
import pytest

from conftest import rel_err
from tuckmill_b200 import cuda, testing as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,batch", [(1000, 2048, 33), (1024, 3072, 65), (1024, 2048, 97), (900, 3072, 129),
                                             (1024, 2048, 161), (2048, 4096, 257), (1024, 3072, 512)])
def test_groups_of_a_split_sum(ctx, oracle, rows, cols, batch):
    raw = T.q8_0_matrix(3, 1, rows, cols)
    x = T.activations(3, 2, batch * cols).reshape(batch, cols)
    w, xb, y = ctx.q8_0_matrix(raw, rows, cols), ctx.floats(x), ctx.buffer(batch * rows * 4)
    runs = []
    for _ in range(3):
        y.zero()
        ctx.q8_0_gemm_mma(w, xb, y, rows, cols, batch)
        runs.append(y.download(0, batch * rows * 4, np.float32).reshape(batch, rows))
    assert ctx.mma_last_split() > 1 and not ctx.mma_aborted()
    np.testing.assert_array_equal(runs[1], runs[0])
    np.testing.assert_array_equal(runs[2], runs[0])
    some = sorted({0, 31, 32, batch // 2, batch - 1})
    assert rel_err(runs[0][some], oracle.matmul_q8_0(raw, rows, cols, x[some])) <= 1e-3
    base = T.activations(3, 4, batch * rows).reshape(batch, rows)
    acc = ctx.floats(base)
    ctx.q8_0_gemm_mma_fused(w, xb, rows, cols, batch, [acc], [rows], cuda.PRO_NONE, None, 0.0, cuda.EPI_ADD)
    np.testing.assert_array_equal(acc.download(0, batch * rows * 4, np.float32).reshape(batch, rows), base + runs[0])


# Parts that meet in a cluster: 2, 3, 4, 6 and 8 of them, shares of the tokens that are uneven or empty, a last four of
# tokens that is not whole, rows that end inside a tile
@pytest.mark.parametrize("rows,cols,batch", [(6144, 1024, 61), (1500, 2304, 3), (1536, 1152, 130), (4000, 1024, 29),
                                             (1152, 6912, 35), (1024, 3072, 9), (1024, 2048, 33), (1024, 3072, 200),
                                             (3000, 4096, 128), (1024, 2048, 512)])
def test_parts_that_meet_in_a_cluster(ctx, rows, cols, batch, parts=None):
    raw = T.q8_0_matrix(6, rows + cols, rows, cols)
    x = T.activations(6, 2, batch * cols).reshape(batch, cols)
    w, xb = ctx.q8_0_matrix(raw, rows, cols), ctx.floats(x)
    base = T.activations(6, 4, batch * rows).reshape(batch, rows)
    got = []
    for _ in range(2):
        y = ctx.floats(np.full((batch, rows), np.nan, np.float32))
        ctx.q8_0_gemm_mma(w, xb, y, rows, cols, batch)
        got.append(y.download(0, batch * rows * 4, np.float32).reshape(batch, rows))
    assert ctx.mma_last_split() > 1 and not ctx.mma_aborted()
    assert ctx.mma_last_cluster() == (parts is None) and parts in (None, ctx.mma_last_split())
    ref = x.astype(np.float16).astype(np.float64) @ T.q8_0_dequant(raw).astype(np.float16).astype(np.float64).T
    assert rel_err(got[0], ref) <= 2e-5
    np.testing.assert_array_equal(got[0], got[1])
    acc = ctx.floats(base)
    ctx.q8_0_gemm_mma_fused(w, xb, rows, cols, batch, [acc], [rows], cuda.PRO_NONE, None, 0.0, cuda.EPI_ADD)
    np.testing.assert_array_equal(acc.download(0, batch * rows * 4, np.float32).reshape(batch, rows), base + got[0])


# Parts that meet in the workspace, because not all clusters have a place: 2, 3, 6 and 8 of them, in the forms with four
# converter sets and with two, fewer groups of 32 tokens than parts and more, a last group of one token; 128-token sub-tiles
# (which have no cluster form)
@pytest.mark.parametrize("rows,cols,batch,parts", [(9344, 2048, 33, 2), (6144, 1152, 29, 3), (6100, 1152, 33, 3), (6144, 1152, 97, 3),
                                                   (2432, 2304, 64, 6), (2432, 2304, 32, 6), (1024, 2048, 161, 8), (1000, 2048, 200, 8)])
def test_parts_that_meet_in_the_workspace(ctx, rows, cols, batch, parts):
    test_parts_that_meet_in_a_cluster(ctx, rows, cols, batch, parts)
