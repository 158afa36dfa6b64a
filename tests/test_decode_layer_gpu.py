"""The latency forms of a decode step's operators at the sizes where their splits change, against the forms that are
pinned to the oracle."""
import numpy as np
import pytest

from conftest import rel_err
from tuckmill_b200 import cuda, testing as T

pytestmark = pytest.mark.gpu


# positions around a CTA's runs of eight keys, its 64-key tiles and the 1024 keys a cluster of 16 takes in one pass
@pytest.mark.parametrize("pos", [0, 1, 8, 127, 128, 1023, 1024, 1100])
@pytest.mark.parametrize("heads,kvh,hd,window", [(16, 8, 128, 0), (4, 4, 128, 40), (4, 1, 256, 512), (32, 8, 128, 0), (2, 1, 256, 0)])
def test_cluster_attention_equals_the_exact_form(ctx, oracle, heads, kvh, hd, window, pos):
    cap, eps, scale = 1200, 1e-6, 1.0 / np.sqrt(np.float32(hd))
    qn = ctx.floats((1 + 0.1 * T.activations(0, 20, hd)).astype(np.float32))
    kn = ctx.floats((1 + 0.1 * T.activations(0, 21, hd)).astype(np.float32))
    inv = ctx.floats(oracle.rope_inv_freq(hd, 1e6))
    kfill = T.activations(1, 1, kvh * cap * hd).astype(np.float16).reshape(kvh, cap, hd)
    vfill = T.activations(1, 2, kvh * cap * hd).astype(np.float16).reshape(kvh, cap, hd)
    vfill[:, pos + 1:] = np.nan  # rows past the sequence must not reach the result
    q, k, v = (ctx.floats(T.activations(7, t, n * hd)) for t, n in ((30, heads), (31, kvh), (32, kvh)))
    status = ctx.buffer(4, shared=True)
    status.zero()
    scratch = ctx.buffer(cuda.decode_attention_scratch_bytes(heads, kvh, hd, cap))
    outs, caches = [], []
    for exact in (True, False):
        scratch.zero()
        kc, vc, out = ctx.from_array(kfill), ctx.from_array(vfill), ctx.buffer(heads * hd * 4)
        ctx.attention_decode_dev(q, k, v, qn, kn, inv, kc, vc, out, scratch, ctx.from_array(np.array([pos], np.uint32)), 0,
                                 status, heads, kvh, hd, hd, cap, window, eps, scale, exact)
        outs.append(out.download(0, heads * hd * 4, np.float32))
        caches.append([c.download(0, kvh * cap * hd * 2, np.float16).reshape(kvh, cap, hd)[:, :pos + 1].astype(np.float32)
                       for c in (kc, vc)])
    assert rel_err(outs[1], outs[0]) <= 2e-5
    for a, b in zip(*caches):
        assert np.max(np.abs(a - b)) <= 2e-3 * max(1.0, float(np.max(np.abs(a))))  # one f16 step of the fresh row
    assert int(status.download(0, 4, np.uint32)[0]) == 0


# A value that binary16 holds as an infinity stays one: rows past a CTA's run or before the window, whose weight is 0, add no NaN.
@pytest.mark.parametrize("pos", [0, 7, 8, 63, 100, 1099])
@pytest.mark.parametrize("heads,kvh,hd,window", [(16, 8, 128, 0), (4, 1, 256, 40), (4, 2, 128, 40)])
def test_attention_of_infinite_values(ctx, oracle, heads, kvh, hd, window, pos):
    cap, eps, scale = 1200, 1e-6, 1.0 / np.sqrt(np.float32(hd))
    one, inv, pb = ctx.floats(np.ones(hd)), ctx.floats(oracle.rope_inv_freq(hd, 1e6)), ctx.from_array(np.array([pos], np.uint32))
    fill = [T.activations(1, t, kvh * cap * hd).astype(np.float16).reshape(kvh, cap, hd) for t in (1, 2)]
    q, k, v = (T.activations(7, t, n * hd).reshape(n, hd) for t, n in ((30, heads), (31, kvh), (32, kvh)))
    fill[1][:, :, 3], v[:, 3] = np.inf, 1e6  # every row
    v[:, 5] = -1e6                           # this step's
    fill[1][:, :max(0, pos + 1 - window) if window else 0, 7] = np.inf  # not seen
    status = ctx.buffer(4, shared=True)
    status.zero()
    scratch = ctx.buffer(cuda.decode_attention_scratch_bytes(heads, kvh, hd, cap))
    outs = []
    for exact in (True, False):
        scratch.zero()
        kc, vc, out = ctx.from_array(fill[0]), ctx.from_array(fill[1]), ctx.buffer(heads * hd * 4)
        ctx.attention_decode_dev(ctx.floats(q), ctx.floats(k), ctx.floats(v), one, one, inv, kc, vc, out, scratch, pb, 0, status,
                                 heads, kvh, hd, hd, cap, window, eps, scale, exact)
        outs.append(out.download(0, heads * hd * 4, np.float32).reshape(heads, hd))
    # a batch of two such sequences, on the tensor cores for head size 128
    kc, vc, out = ctx.from_array(np.stack([fill[0]] * 2)), ctx.from_array(np.stack([fill[1]] * 2)), ctx.buffer(2 * heads * hd * 4)
    sb = ctx.buffer(2 * cuda.decode_attention_scratch_bytes(heads, kvh, hd, cap))
    sb.zero()
    ctx.attention_decode_batch(*(ctx.floats(np.stack([r] * 2)) for r in (q, k, v)), one, one, inv, kc, vc, out, sb,
                               ctx.from_array(np.array([pos] * 2, np.uint32)), status, 2, heads, kvh, hd, hd, cap, window, eps, scale, False)
    batch = out.download(0, 2 * heads * hd * 4, np.float32).reshape(2, heads, hd)
    finite = np.delete(np.arange(hd), [3, 5])
    for o in (*outs, *batch):
        assert np.all(o[:, 3] == np.inf) and np.all(o[:, 5] == -np.inf)
    assert rel_err(outs[1][:, finite], outs[0][:, finite]) <= 2e-5  # (as for finite rows, above)
    for b in batch:
        assert rel_err(b[:, finite], outs[0][:, finite]) <= 2e-3  # binary16 queries and weights


# A row whose sum of squares overflows is normed with 1 / infinity: zeros, in every form.
@pytest.mark.parametrize("heads,kvh,hd", [(4, 2, 128), (4, 1, 256)])
@pytest.mark.parametrize("big", ["q", "k"])
def test_attention_of_a_row_beyond_the_range_of_its_norm(ctx, oracle, heads, kvh, hd, big):
    cap, pos, eps, scale = 300, 200, 1e-6, 1.0 / np.sqrt(np.float32(hd))
    qn = ctx.floats((1 + 0.1 * T.activations(0, 20, hd)).astype(np.float32))
    inv, pb = ctx.floats(oracle.rope_inv_freq(hd, 1e6)), ctx.from_array(np.array([pos], np.uint32))
    fill = [T.activations(1, t, kvh * cap * hd).astype(np.float16) for t in (1, 2)]
    q, k, v = (T.activations(7, t, n * hd) * np.float32(1e25 if name == big else 1)
               for name, t, n in (("q", 30, heads), ("k", 31, kvh), ("v", 32, kvh)))
    status = ctx.buffer(4, shared=True)
    status.zero()
    scratch = ctx.buffer(cuda.decode_attention_scratch_bytes(heads, kvh, hd, cap))
    outs = []
    for exact in (True, False):
        scratch.zero()
        kc, vc, out = ctx.from_array(fill[0]), ctx.from_array(fill[1]), ctx.buffer(heads * hd * 4)
        ctx.attention_decode_dev(ctx.floats(q), ctx.floats(k), ctx.floats(v), qn, qn, inv, kc, vc, out, scratch, pb, 0, status,
                                 heads, kvh, hd, hd, cap, 0, eps, scale, exact)
        outs.append(out.download(0, heads * hd * 4, np.float32))
        new = kc.download(0, fill[0].nbytes, np.float16).reshape(kvh, cap, hd)[:, pos]
        assert np.all(new == 0) if big == "k" else np.all(np.isfinite(new))
    assert rel_err(outs[1], outs[0]) <= 2e-5  # (as for rows of an ordinary size, above)
    if big == "q":  # every key weighs the same
        vals = fill[1].astype(np.float64).reshape(kvh, cap, hd)[:, :pos]
        mean = (vals.sum(axis=1) + v.reshape(kvh, hd).astype(np.float16)) / (pos + 1)
        assert rel_err(outs[1].reshape(kvh, heads // kvh, hd), np.repeat(mean[:, None], heads // kvh, axis=1)) <= 2e-5


def test_feed_forward_block_of_a_row_beyond_the_range_of_its_norm(ctx):
    hidden, width = 1024, 3072
    gu, dn = ctx.q8_0_matrix(T.q8_0_matrix(3, 1, 2 * width, hidden), 2 * width, hidden), ctx.q8_0_matrix(T.q8_0_matrix(3, 2, hidden, width), hidden, width)
    one, xo, so = ctx.floats(np.ones(hidden)), ctx.buffer(hidden * 4), ctx.buffer(8 * hidden * 4)
    x = T.activations(3, 3, hidden)
    # the slots' sum under its output norm: adds nothing
    ctx.decode_ffn_block(ctx.floats(x), ctx.floats(np.full(hidden, 1e25)), 1, one, one, xo, gu, dn, so, hidden, width, False, 1e-6)
    np.testing.assert_array_equal(xo.download(0, hidden * 4, np.float32), x)
    assert np.all(np.isfinite(so.download(0, 8 * hidden * 4, np.float32)))
    # the stream itself under the block's input norm: the block adds nothing
    ctx.decode_ffn_block(ctx.floats(x * np.float32(1e25)), None, 0, None, one, xo, gu, dn, so, hidden, width, False, 1e-6)
    assert np.all(so.download(0, 8 * hidden * 4, np.float32) == 0)


def f64_layer(x, slots, add_w, norm_w, eps):
    p = slots.astype(np.float64).sum(axis=0) if slots is not None else 0.0
    if add_w is not None:
        p = p / np.sqrt((p ** 2).mean() + eps) * add_w
    x = x + p
    return x, x / np.sqrt((x ** 2).mean() + eps) * norm_w


# widths that cut evenly over clusters and CTAs, that leave remainders, and the narrowest there is
@pytest.mark.parametrize("hidden,width,n_slots,normed", [(1024, 3072, 8, False), (64, 512, 0, False), (320, 576, 1, True),
                                                         (1088, 1024, 3, True), (1024, 2112, 8, True)])
@pytest.mark.parametrize("gelu", [False, True])
def test_feed_forward_block(ctx, hidden, width, n_slots, normed, gelu, clusters=0):
    eps = 1e-6
    raw_gu, raw_dn = T.q8_0_matrix(3, 1, 2 * width, hidden), T.q8_0_matrix(3, 2, hidden, width)
    x, nw = T.activations(3, 3, hidden), (1 + 0.1 * T.activations(3, 4, hidden)).astype(np.float32)
    slots = T.activations(3, 5, n_slots * hidden).reshape(n_slots, hidden) if n_slots else None
    aw = (1 + 0.1 * T.activations(3, 6, hidden)).astype(np.float32) if normed else None
    want_x, h = f64_layer(x, slots, aw, nw, eps)
    g, u = np.split(T.q8_0_dequant(raw_gu).astype(np.float64) @ h, 2)
    act = (0.5 * g * (1 + np.tanh(0.7978845608028654 * (g + 0.044715 * g ** 3))) if gelu else g / (1 + np.exp(-g))) * u
    want = T.q8_0_dequant(raw_dn).astype(np.float64) @ act
    xo, so = ctx.buffer(hidden * 4), ctx.buffer(8 * hidden * 4)
    ctx.decode_ffn_block(ctx.floats(x), ctx.floats(slots) if n_slots else None, n_slots, ctx.floats(aw) if normed else None,
                         ctx.floats(nw), xo, ctx.q8_0_matrix(raw_gu, 2 * width, hidden), ctx.q8_0_matrix(raw_dn, hidden, width),
                         so, hidden, width, gelu, eps)
    assert rel_err(xo.download(0, hidden * 4, np.float32), want_x) <= 2e-6
    out = so.download(0, 8 * hidden * 4, np.float32).reshape(8, hidden).astype(np.float64)
    assert rel_err(out.sum(axis=0), want) <= 2e-6
    if clusters:  # every slot is its share of the width, the rest are zeros
        cut = [64 * (width // 64 * c // clusters) for c in range(clusters + 1)]
        shares = [T.q8_0_dequant(raw_dn).astype(np.float64)[:, a:b] @ act[a:b] for a, b in zip(cut, cut[1:])]
        assert rel_err(out[:clusters], np.array(shares)) <= 2e-6
        assert np.all(out[clusters:] == 0)


# the narrowest width that takes eight clusters, the widest that takes six, clusters with one chunk of columns and with two
@pytest.mark.parametrize("hidden,width,n_slots,clusters", [(1024, 4096, 8, 8), (1024, 3136, 2, 8), (1024, 3072, 0, 6), (192, 704, 5, 6)])
def test_feed_forward_block_by_clusters(ctx, hidden, width, n_slots, clusters):
    test_feed_forward_block(ctx, hidden, width, n_slots, False, False, clusters)


@pytest.mark.parametrize("hidden,heads,kvh,hd,pos,window", [(1024, 16, 8, 128, 700, 0), (256, 4, 2, 128, 0, 0), (64, 3, 3, 128, 129, 50),
                                                            (128, 4, 1, 256, 1030, 40), (1088, 8, 8, 128, 15, 0)])
def test_attention_block_equals_the_operators_it_replaces(ctx, oracle, hidden, heads, kvh, hd, pos, window):
    eps, cap, scale, n_slots = 1e-6, 1100, 1.0 / np.sqrt(np.float32(hd)), 4
    rows = (heads + 2 * kvh) * hd
    qkv = ctx.q8_0_matrix(T.q8_0_matrix(4, 1, rows, hidden), rows, hidden)
    o = ctx.q8_0_matrix(T.q8_0_matrix(4, 2, hidden, heads * hd), hidden, heads * hd)
    x, nw = T.activations(4, 3, hidden), (1 + 0.1 * T.activations(4, 4, hidden)).astype(np.float32)
    slots = T.activations(4, 5, n_slots * hidden).reshape(n_slots, hidden)
    qn, kn = (ctx.floats((1 + 0.1 * T.activations(4, t, hd)).astype(np.float32)) for t in (20, 21))
    inv, pb = ctx.floats(oracle.rope_inv_freq(hd, 1e6)), ctx.from_array(np.array([pos], np.uint32))
    kfill, vfill = (T.activations(4, t, kvh * cap * hd).astype(np.float16) for t in (30, 31))
    status = ctx.buffer(4, shared=True)
    status.zero()
    want_x = f64_layer(x, slots, None, nw, eps)[0].astype(np.float32)
    # the operators: norm + q|k|v, exact attention, o
    xb, y, att, out = ctx.floats(want_x), ctx.buffer(rows * 4), ctx.buffer(heads * hd * 4), ctx.buffer(hidden * 4)
    ctx.q8_0_gemv_fused(qkv, xb, y, rows, hidden, cuda.PRO_RMSNORM, ctx.floats(nw), eps)
    scratch = ctx.buffer(cuda.decode_attention_scratch_bytes(heads, kvh, hd, cap))
    scratch.zero()
    kc, vc = ctx.from_array(kfill), ctx.from_array(vfill)
    ctx.attention_decode_dev(y.view(0, heads * hd * 4), y.view(heads * hd * 4, kvh * hd * 4),
                             y.view((heads + kvh) * hd * 4, kvh * hd * 4), qn, kn, inv, kc, vc, att, scratch, pb, 0, status,
                             heads, kvh, hd, hd, cap, window, eps, scale, True)
    ctx.q8_0_gemv(o, att, out, hidden, heads * hd)
    # the block
    kc2, vc2, xo, so = ctx.from_array(kfill), ctx.from_array(vfill), ctx.buffer(hidden * 4), ctx.buffer(8 * hidden * 4)
    ctx.decode_attn_block(ctx.floats(x), ctx.floats(slots), n_slots, None, ctx.floats(nw), xo, qkv, o, qn, kn, inv, kc2, vc2, pb,
                          0, status, so, hidden, heads, kvh, hd, cap, window, eps, scale)
    assert rel_err(xo.download(0, hidden * 4, np.float32), want_x) <= 2e-6
    got = so.download(0, kvh * hidden * 4, np.float32).reshape(kvh, hidden).astype(np.float64).sum(axis=0)
    assert rel_err(got, out.download(0, hidden * 4, np.float32)) <= 1e-4
    for a, b in ((kc, kc2), (vc, vc2)):
        d = np.abs(a.download(0, kfill.nbytes, np.float16).astype(np.float32) - b.download(0, kfill.nbytes, np.float16).astype(np.float32))
        assert float(np.max(d)) <= 4e-3  # one f16 step of the fresh row
    # a position past the capacity is flagged, not stored
    pb.upload(0, np.array([cap], np.uint32))
    ctx.decode_attn_block(ctx.floats(x), None, 0, None, ctx.floats(nw), xo, qkv, o, qn, kn, inv, kc2, vc2, pb, 0, status, so,
                          hidden, heads, kvh, hd, cap, window, eps, scale)
    assert int(status.download(0, 4, np.uint32)[0]) == 1


# x_out does not hang on the position: it is stored where the rest of the block is not
@pytest.mark.parametrize("hidden,heads,kvh,hd,n_slots,normed", [(256, 4, 2, 128, 2, True), (128, 4, 1, 256, 0, False),
                                                                 (1088, 8, 8, 128, 8, False)])
@pytest.mark.parametrize("past", [0, 1, 2**32 - 65])
def test_attention_block_past_the_capacity_stores_the_sum_alone(ctx, oracle, hidden, heads, kvh, hd, n_slots, normed, past):
    cap, rows, eps = 64, (heads + 2 * kvh) * hd, 1e-6
    qkv = ctx.q8_0_matrix(T.q8_0_matrix(4, 1, rows, hidden), rows, hidden)
    o = ctx.q8_0_matrix(T.q8_0_matrix(4, 2, hidden, heads * hd), hidden, heads * hd)
    x, nw = T.activations(4, 3, hidden), (1 + 0.1 * T.activations(4, 4, hidden)).astype(np.float32)
    aw = (1 + 0.1 * T.activations(4, 6, hidden)).astype(np.float32) if normed else None
    slots = T.activations(4, 5, n_slots * hidden).reshape(n_slots, hidden)
    fill, so_fill = T.activations(4, 30, kvh * cap * hd).astype(np.float16), T.activations(4, 7, 8 * hidden)
    kc, vc, xo = ctx.from_array(fill), ctx.from_array(fill), ctx.buffer(hidden * 4)
    so, status = ctx.floats(so_fill), ctx.buffer(4, shared=True)
    xo.zero(), status.zero()
    one, inv = ctx.floats(np.ones(hd)), ctx.floats(oracle.rope_inv_freq(hd, 1e6))
    ctx.decode_attn_block(ctx.floats(x), ctx.floats(slots) if n_slots else None, n_slots, ctx.floats(aw) if normed else None,
                          ctx.floats(nw), xo, qkv, o, one, one, inv, kc, vc,
                          ctx.from_array(np.array([cap + past], np.uint32)), 0, status, so, hidden, heads, kvh, hd, cap, 0, eps, hd ** -0.5)
    assert int(status.download(0, 4, np.uint32)[0]) == cuda.STATUS_PAST_CAPACITY
    assert rel_err(xo.download(0, hidden * 4, np.float32), f64_layer(x, slots, aw, nw, eps)[0]) <= 2e-6
    for c in (kc, vc):
        np.testing.assert_array_equal(c.download(0, fill.nbytes, np.float16), fill)
    np.testing.assert_array_equal(so.download(0, so_fill.nbytes, np.float32), so_fill)


@pytest.mark.parametrize("block", ["attention", "feed-forward"])
def test_blocks_refuse_outputs_in_what_other_clusters_read(ctx, oracle, block):
    hidden, width, heads, kvh, hd, cap = 256, 1024, 4, 2, 128, 64
    vec = lambda: ctx.floats(np.ones(hidden))  # noqa: E731
    x, nw, aw, xo, arena = vec(), vec(), vec(), vec(), ctx.floats(np.zeros(20 * hidden))
    slots, out = arena.view(0, 8 * hidden * 4), arena.view(8 * hidden * 4, 8 * hidden * 4)
    if block == "attention":
        rows = (heads + 2 * kvh) * hd
        qkv, o = ctx.q8_0_matrix(T.q8_0_matrix(4, 1, rows, hidden), rows, hidden), ctx.q8_0_matrix(T.q8_0_matrix(4, 2, hidden, heads * hd), hidden, heads * hd)
        kc, vc, status = ctx.buffer(kvh * cap * hd * 2), ctx.buffer(kvh * cap * hd * 2), ctx.buffer(4, shared=True)
        kc.zero(), vc.zero(), status.zero()
        qn, inv, pb = ctx.floats(np.ones(hd)), ctx.floats(oracle.rope_inv_freq(hd, 1e6)), ctx.from_array(np.zeros(1, np.uint32))
        call = lambda xo, so: ctx.decode_attn_block(x, slots, 2, aw, nw, xo, qkv, o, qn, qn, inv, kc, vc, pb, 0, status, so,  # noqa: E731
                                                    hidden, heads, kvh, hd, cap, 0, 1e-6, hd ** -0.5)
    else:
        gu, dn = ctx.q8_0_matrix(T.q8_0_matrix(3, 1, 2 * width, hidden), 2 * width, hidden), ctx.q8_0_matrix(T.q8_0_matrix(3, 2, hidden, width), hidden, width)
        call = lambda xo, so: ctx.decode_ffn_block(x, slots, 2, aw, nw, xo, gu, dn, so, hidden, width, False, 1e-6)  # noqa: E731
    call(xo, out)
    row = hidden * 4
    for bad_xo, bad_so in ((x, out), (arena.view(row, row), out), (nw, out), (aw, out), (xo, slots), (xo, arena.view(row, 8 * row))):
        with pytest.raises(cuda.CudaError) as e:
            call(bad_xo, bad_so)
        assert e.value.code == -5
    call(xo, arena.view(2 * row, 8 * row))  # behind the two slots that are read
    ctx.fence()
