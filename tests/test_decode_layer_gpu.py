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
