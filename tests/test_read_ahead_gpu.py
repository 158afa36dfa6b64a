"""Operands that kernels read before their predecessors have finished (weights, rotation table, cached rows): an operator
that has just written one must still be seen, whatever the chain in between.  Each sequence runs once with a fence after
the write and once without, in one dispatch; the launch that reads the written operand is the one that waits."""
import numpy as np
import pytest

from tuckmill_b200 import cuda, testing as T

pytestmark = pytest.mark.gpu


def chain(ctx, write, read, out, n, dtype=np.float32):
    """read() after write() with everything finished in between, then the two in one dispatch; the launches that waited
    for the written operand there, and in a second read() behind it."""
    write(), ctx.fence(), read()
    want = out.download(0, n * np.dtype(dtype).itemsize, dtype)
    write(), ctx.fence()
    counts = []

    def both():
        before = ctx.ordered_launches()
        write(), read()
        counts.append(ctx.ordered_launches() - before)
        read()
        counts.append(ctx.ordered_launches() - before - counts[0])

    ctx.grouped(both)
    ctx.fence()
    return want, out.download(0, n * np.dtype(dtype).itemsize, dtype), counts


@pytest.mark.parametrize("rows,cols", [(1, 1152), (3, 4096)])
def test_norm_weight(ctx, rows, cols):
    w, p = ctx.floats(np.ones(cols)), ctx.floats(T.activations(1, 1, rows * cols))
    zero, x, step = ctx.floats(np.zeros(rows * cols)), ctx.buffer(rows * cols * 4), ctx.floats(np.full(cols, 0.5))

    def write():
        ctx.f32_scale(w, w, 0.0, cols)
        ctx.f32_axpy(step, w, 1.0, cols)  # lets its successor start at once

    def read():
        ctx.f32_scale(zero, x, 1.0, rows * cols)
        ctx.rmsnorm_add(p, w, x, rows, cols, 1e-6)

    want, got, counts = chain(ctx, write, read, x, rows * cols)
    np.testing.assert_array_equal(got, want)
    assert counts == [1, 0]


@pytest.mark.parametrize("batch", [1, 8])
def test_f16_matrix(ctx, batch):
    rows, cols = 1024, 512
    src = ctx.floats(T.activations(2, 1, rows * cols))
    w, x, y = ctx.buffer(rows * cols * 2), ctx.floats(T.activations(2, 2, batch * cols)), ctx.buffer(batch * rows * 4)
    want, got, counts = chain(ctx, lambda: ctx.cast_f32_f16(src, w, rows * cols),
                              lambda: ctx.f16_gemm(w, x, y, rows, cols, batch), y, batch * rows)
    np.testing.assert_array_equal(got, want)
    assert counts == [1, 0]


def test_packed_matrix(ctx):
    rows, cols = 2048, 1024
    raw = T.q8_0_matrix(3, 1, rows, cols)
    staged, w = ctx.from_array(raw), ctx.buffer(cuda.packed_bytes(rows, cols))
    x, y = ctx.floats(T.activations(3, 2, cols)), ctx.buffer(rows * 4)
    want, got, counts = chain(ctx, lambda: ctx._call("q8_0_pack", w.handle, rows, cols, staged.handle, 0, 0, rows),
                              lambda: ctx.q8_0_gemv(w, x, y, rows, cols), y, rows)
    np.testing.assert_array_equal(got, want)
    assert counts == [1, 0]


@pytest.mark.parametrize("n_seq", [1, 2])
def test_rotation_table_and_cached_rows(ctx, n_seq):
    heads, kvh, hd, cap, pos = 4, 2, 128, 300, 200
    one = lambda t, n: ctx.floats(T.activations(4, t, n))  # noqa: E731
    q, k, v, qn, kn = one(1, n_seq * heads * hd), one(2, n_seq * kvh * hd), one(3, n_seq * kvh * hd), one(4, hd), one(5, hd)
    inv, freq = ctx.buffer(hd * 2), ctx.floats(1e4 ** (-np.arange(hd // 2) * 2.0 / hd))
    kc, vc = (ctx.from_array(T.activations(4, t, n_seq * kvh * cap * hd).astype(np.float16)) for t in (6, 7))
    rows = one(8, (pos + 1) * kvh * hd)
    out, status = ctx.buffer(n_seq * heads * hd * 4), ctx.buffer(4, shared=True)
    status.zero()
    scratch = ctx.buffer(n_seq * cuda.decode_attention_scratch_bytes(heads, kvh, hd, cap))
    scratch.zero()
    pb = ctx.from_array(np.full(n_seq, pos, np.uint32))

    def read(p=pb, at=0):
        if n_seq > 1:
            ctx.attention_decode_batch(q, k, v, qn, kn, inv, kc, vc, out, scratch, p, status, n_seq, heads, kvh, hd, hd, cap, 0,
                                       1e-6, hd ** -0.5, False)
        else:
            ctx.attention_decode_dev(q, k, v, qn, kn, inv, kc, vc, out, scratch, p, at, status, heads, kvh, hd, hd, cap, 0, 1e-6,
                                     hd ** -0.5, exact=False)

    n = n_seq * heads * hd
    want, got, counts = chain(ctx, lambda: ctx.f32_scale(freq, inv, 1.0, hd // 2), read, out, n)
    np.testing.assert_array_equal(got, want)
    assert counts == [1, 0]
    want, got, counts = chain(ctx, lambda: ctx.qwen35_kv_store_chunk(rows, rows, kc, vc, 0, cap, hd, kvh, pos), read, out, n)
    np.testing.assert_array_equal(got, want)
    assert counts == [1, 0]
    if n_seq == 1:  # the row of a call that took its position from another word is not the one read late
        two = ctx.from_array(np.array([20, pos], np.uint32))
        want, got, counts = chain(ctx, lambda: read(two, 0), lambda: read(two, 1), out, n)
        np.testing.assert_array_equal(got, want)
        assert counts == [1, 0]


def test_a_replayed_graph_counts_as_a_writer(ctx):
    cols = 1024
    w, p, x = ctx.floats(np.ones(cols)), ctx.floats(T.activations(5, 1, cols)), ctx.floats(np.zeros(cols))
    other, step = ctx.floats(np.ones(cols)), ctx.floats(np.ones(cols))
    ctx.fence()
    ctx.begin_group()
    ctx.f32_axpy(step, w, 1.0, cols)
    graph = ctx.end_group_retain()
    ctx.rmsnorm_add(p, w, x, 1, cols, 1e-6)  # the group has not run, yet its operators are younger than the last boundary
    ctx.fence()
    for _ in range(2):
        graph.launch()
        before = ctx.ordered_launches()
        ctx.rmsnorm_add(p, other, x, 1, cols, 1e-6)  # nothing ever wrote this one
        assert ctx.ordered_launches() == before
        ctx.rmsnorm_add(p, w, x, 1, cols, 1e-6)
        assert ctx.ordered_launches() == before + 1
        ctx.rmsnorm_add(p, w, x, 1, cols, 1e-6)
        assert ctx.ordered_launches() == before + 1
    graph.free()


def test_a_request_overlaps_its_launches(ctx, tmp_path):
    """An engine's operands are written at load: no launch of a request waits for them."""
    from tuckmill_b200 import engine
    from tuckmill_b200.testing import DecoderShape, write_gguf
    shape = DecoderShape("qwen3", 2, 1024, 3072, 16, 8, 128, 600)
    path = tmp_path / "m.gguf"
    write_gguf(path, shape)
    eng = engine.Engine(path, context=128)
    count = lambda: cuda.load_library().tm_cuda_ordered_launches(eng.cuda_ctx())  # noqa: E731
    eng.generate(np.arange(40, dtype=np.uint32), 8)
    before = count()
    eng.generate(np.arange(40, dtype=np.uint32), 8)
    assert count() == before
    eng.close()
