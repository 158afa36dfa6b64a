"""The operators that keep a request's host path short: words stored as kernel arguments, a strided clear, and
groups that go to the stream as they are encoded."""
import numpy as np
import pytest

from tuckmill_b200 import cuda, testing as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 447, 448, 449, 1000])
@pytest.mark.parametrize("indexed", [False, True])
def test_store_u32_lands_where_asked_and_nowhere_else(ctx, n, indexed):
    size = 2 * n + 5
    buf = ctx.buffer(size * 4)
    buf.zero()
    vals = (np.arange(n, dtype=np.uint64) * 2654435761 % 2 ** 32).astype(np.uint32)
    idx = np.random.default_rng(n).permutation(size)[:n].astype(np.uint32) if indexed else np.arange(3, 3 + n)
    buf.store_u32(vals, first=3, index=idx if indexed else None)
    want = np.zeros(size, np.uint32)
    want[idx] = vals
    np.testing.assert_array_equal(buf.download(0, size * 4, np.uint32), want)
    with pytest.raises(cuda.CudaError):
        buf.store_u32(vals, first=size - n + 1)


def test_zero_2d_clears_the_rows_width_only(ctx):
    a = np.arange(1, 7 * 48 + 1, dtype=np.uint32)
    buf = ctx.from_array(a)
    buf.zero_2d(192, 192, 64, 5)
    want = a.reshape(7, 48).copy()
    want[1:6, :16] = 0
    np.testing.assert_array_equal(buf.download(0, a.nbytes, np.uint32).reshape(7, 48), want)
    with pytest.raises(cuda.CudaError):
        buf.zero_2d(192, 192, 64, 7)


def test_burst_counts_as_one_dispatch(ctx):
    x = ctx.floats(T.activations(0, 1, 300))
    y = ctx.buffer(1200)
    before, launches = ctx.committed_dispatches(), ctx.kernel_launches()
    ctx._call("begin_burst")
    ctx.f32_scale(x, y, 2.0, 300)
    ctx.f32_scale(y, y, 2.0, 300)
    with pytest.raises(cuda.CudaError):
        ctx.begin_group()
    ctx._call("end_burst")
    assert ctx.committed_dispatches() == before + 1 and ctx.kernel_launches() == launches + 2
    np.testing.assert_array_equal(y.download(0, 1200, np.float32), x.download(0, 1200, np.float32) * 4)


@pytest.mark.parametrize("n", [65532, 65536, 607744, 1048576, 1048580])  # either side of what passes through pinned memory
def test_downloads_of_any_length(ctx, n):
    a = np.random.default_rng(n).integers(0, 256, n + 64, dtype=np.uint8)
    buf = ctx.from_array(a)
    np.testing.assert_array_equal(buf.download(64, n, np.uint8), a[64:])
    b = a[::-1].copy()
    buf.upload(0, b)
    np.testing.assert_array_equal(buf.download(0, n, np.uint8), b[:n])
