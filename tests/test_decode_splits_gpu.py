"""Decode attention of many sequences: one split a head while every CTA finds a place at once (37 sequences of 8 KV heads
on 148 SMs), the shorter ring beyond that, two splits below; ragged positions at the edges of the 64-key tiles; against
the one-sequence kernel on the same caches."""
import numpy as np
import pytest

from tuckmill_b200 import cuda, testing as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S", [18, 37, 38])
@pytest.mark.parametrize("heads,window", [(8, 0), (16, 0), (32, 70)])
def test_every_sequence_is_the_single_call(ctx, S, heads, window):
    kv, hd, cap, eps, scale = 8, 128, 400, 1e-6, 128 ** -0.5
    pos = np.resize(np.array([0, 62, 63, 64, 127, 128, 191, 192, 399, 256, 5], np.uint32), S)
    one = lambda i: (1 + 0.1 * T.activations(0, i, hd)).astype(np.float32)  # noqa: E731
    freq = (1e4 ** (-np.arange(hd // 2) * 2.0 / hd)).astype(np.float32)
    qn, kn, inv = ctx.floats(one(1)), ctx.floats(one(2)), ctx.floats(freq)
    plane = kv * cap * hd
    kf, vf = (T.activations(1, i, S * plane).astype(np.float16) for i in (1, 2))
    q, k, v = (T.activations(2, i, S * n * hd).reshape(S, n * hd) for i, n in enumerate((heads, kv, kv)))
    status, per = ctx.buffer(4, shared=True), cuda.decode_attention_scratch_bytes(heads, kv, hd, cap)
    status.zero()
    kc, vc, out, sb = ctx.from_array(kf), ctx.from_array(vf), ctx.buffer(S * heads * hd * 4), ctx.buffer(S * per)
    sb.zero()
    for _ in range(2):
        ctx.attention_decode_batch(ctx.floats(q), ctx.floats(k), ctx.floats(v), qn, kn, inv, kc, vc, out, sb, ctx.from_array(pos),
                                   status, S, heads, kv, hd, hd, cap, window, eps, scale, False)
    ctx.fence()
    got = out.download(0, S * heads * hd * 4, np.float32).reshape(S, heads * hd)
    for s in sorted({0, 1, 2, 3, 8, S - 1}):
        k1, v1 = ctx.from_array(kf[s * plane:(s + 1) * plane]), ctx.from_array(vf[s * plane:(s + 1) * plane])
        o1, s1 = ctx.buffer(heads * hd * 4), ctx.buffer(per)
        s1.zero()
        ctx.attention_decode_dev(ctx.floats(q[s]), ctx.floats(k[s]), ctx.floats(v[s]), qn, kn, inv, k1, v1, o1, s1,
                                 ctx.from_array(pos[s:s + 1]), 0, status, heads, kv, hd, hd, cap, window, eps, scale, exact=True)
        ctx.fence()
        want = o1.download(0, heads * hd * 4, np.float32)
        assert np.abs(got[s] - want).max() <= 2e-3 * max(1.0, np.abs(want).max()), f"sequence {s}"
    assert int(status.download(0, 4, np.uint32)[0]) == 0
