"""Prefill attention over several runs of rows in one launch: against float32 torch, at the edges of the query tiles (64
and 128 rows), of the key blocks (32) and of the window, for every head size, and a batch whose prompts share passes
against the same prompts prefilled one by one."""
import numpy as np
import pytest
import torch

from tuckmill_b200 import engine as E, testing as T

pytestmark = pytest.mark.gpu


def norm_rope(x, w, freq, pos, n_rot, eps):
    x = x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w
    ang = pos[:, None, None].float() * freq
    c, s, h = ang.cos(), ang.sin(), n_rot // 2
    a, b = x[..., :h].clone(), x[..., h:n_rot].clone()
    x[..., :h], x[..., h:n_rot] = a * c - b * s, a * s + b * c
    return x


@pytest.mark.parametrize("heads,kv,hd,n_rot,window,runs", [
    (16, 8, 128, 128, 0, [(0, 0, 64), (1, 0, 65), (2, 31, 1), (3, 33, 130)]),
    (16, 8, 128, 128, 0, [(0, 0, 700), (2, 100, 640), (1, 0, 900)]),  # enough tiles for 128 queries a CTA
    (4, 1, 256, 256, 33, [(0, 200, 63), (1, 0, 129)]),
    (4, 2, 64, 64, 32, [(1, 96, 32), (0, 95, 34)]),
    (2, 1, 32, 32, 0, [(0, 0, 5)]),
    (4, 4, 128, 64, 1, [(0, 10, 40), (1, 0, 1)]),  # partly rotated heads
])
def test_runs_against_float32(ctx, heads, kv, hd, n_rot, window, runs):
    cap, seqs, eps, scale = 1024, 4, 1e-6, hd ** -0.5
    rows = sum(r[2] for r in runs)
    g = torch.Generator().manual_seed(rows)
    q, k, v = (torch.randn(rows, n, hd, generator=g) for n in (heads, kv, kv))
    qw, kw = 1 + 0.1 * torch.randn(hd, generator=g), 1 + 0.1 * torch.randn(hd, generator=g)
    freq = 10000.0 ** (-torch.arange(n_rot // 2) * 2.0 / n_rot)
    kc, vc = (torch.randn(seqs, kv, cap, hd, generator=g).half() for _ in range(2))
    bufs = [ctx.from_array(t.numpy()) for t in (q, k, v, qw, kw, freq.float(), kc, vc)]
    out, out16 = ctx.floats(np.zeros(rows * heads * hd, np.float32)), ctx.buffer(rows * heads * hd * 2)
    for o, f16 in ((out, False), (out16, True)):
        ctx.attention_prefill(*bufs, o, heads, kv, hd, n_rot, cap, window, eps, scale, runs, f16)
    got = out.download(0, rows * heads * hd * 4, np.float32).reshape(rows, heads, hd)
    np.testing.assert_array_equal(got.astype(np.float16), out16.download(0, got.size * 2, np.float16).reshape(got.shape))
    at = 0
    for seq, pos0, n in runs:
        pos = torch.arange(pos0, pos0 + n)
        kc[seq, :, pos0:pos0 + n] = norm_rope(k[at:at + n].clone(), kw, freq, pos, n_rot, eps).transpose(0, 1).half()
        vc[seq, :, pos0:pos0 + n] = v[at:at + n].transpose(0, 1).half()
        qq = norm_rope(q[at:at + n].clone(), qw, freq, pos, n_rot, eps).transpose(0, 1)
        keys, vals = (c[seq, :, :pos0 + n].float().repeat_interleave(heads // kv, 0) for c in (kc, vc))
        j = torch.arange(pos0 + n)
        hidden = (j > pos[:, None]) | ((j + window <= pos[:, None]) if window else torch.zeros(1, 1, dtype=torch.bool))
        p = (qq @ keys.transpose(1, 2) * scale).masked_fill(hidden, float("-inf")).softmax(-1)
        want = (p @ vals).transpose(0, 1).numpy()
        assert np.abs(got[at:at + n] - want).max() <= 4e-3 * np.abs(want).max()
        at += n
    for b, want in ((bufs[6], kc), (bufs[7], vc)):  # the rows of the runs stored, all others untouched
        have = b.download(0, want.numel() * 2, np.float16).reshape(want.shape)
        assert np.abs(have.astype(np.float32) - want.float().numpy()).max() <= 4e-3
        assert np.mean(have != want.numpy()) < 0.02


# Any scale: zero (every visible key weighs the same) and negative ones, whose largest score is the smallest product.
@pytest.mark.parametrize("scale", [0.0, -0.5, 0.5])
@pytest.mark.parametrize("hd,window", [(128, 0), (128, 33), (256, 0), (64, 33)])
def test_scales_of_any_sign(ctx, scale, hd, window):
    heads, kv, cap, pos0, n = 4, 2, 128, 40, 70
    g = torch.Generator().manual_seed(hd)
    q, k, v = (torch.randn(n, m, hd, generator=g) for m in (heads, kv, kv))
    one, freq = torch.ones(hd), 10000.0 ** (-torch.arange(hd // 2) * 2.0 / hd)
    kc, vc = (torch.randn(1, kv, cap, hd, generator=g).half() for _ in range(2))
    bufs = [ctx.from_array(t.numpy()) for t in (q, k, v, one, one, freq.float(), kc, vc)]
    out = ctx.buffer(n * heads * hd * 4)
    pos = torch.arange(pos0, pos0 + n)
    ctx.attention_prefill(*bufs, out, heads, kv, hd, hd, cap, window, 1e-6, scale, [(0, pos0, n)], False)
    got = [out.download(0, n * heads * hd * 4, np.float32).reshape(n, heads, hd)]
    qq = norm_rope(q.clone(), one, freq, pos, hd, 1e-6)
    ctx.attention_chunk_mma(ctx.floats(qq.numpy()), bufs[6], bufs[7], out, heads, pos0, cap, hd, heads // kv, scale, n, window)
    got.append(out.download(0, n * heads * hd * 4, np.float32).reshape(n, heads, hd))
    kc[0, :, pos0:pos0 + n] = norm_rope(k.clone(), one, freq, pos, hd, 1e-6).transpose(0, 1).half()
    vc[0, :, pos0:pos0 + n] = v.transpose(0, 1).half()
    keys, vals = (c[0, :, :pos0 + n].float().repeat_interleave(heads // kv, 0) for c in (kc, vc))
    j = torch.arange(pos0 + n)
    hidden = (j > pos[:, None]) | ((j + window <= pos[:, None]) if window else torch.zeros(1, 1, dtype=torch.bool))
    p = (qq.transpose(0, 1) @ keys.transpose(1, 2) * scale).masked_fill(hidden, float("-inf")).softmax(-1)
    want = (p @ vals).transpose(0, 1).numpy()
    for have in got:  # scores to 2^-12 sqrt(hd) / 2 (binary16 queries), weights to 2^-11
        assert np.abs(have - want).max() <= 4e-3 * np.abs(want).max()


@pytest.mark.parametrize("lengths", [[40, 3, 17], [1, 1, 1], [16, 16, 33], [7, 50, 9]])
@pytest.mark.parametrize("shape", [T.SMALL_QWEN3, T.TINY_GEMMA3], ids=["qwen3", "gemma3"])
def test_shared_passes_give_the_tokens_of_passes_of_their_own(tmp_path, shape, lengths):
    path = tmp_path / "m.gguf"
    T.write_gguf(path, shape, seed=3, norm_jitter=0.1)
    prompts = [T.token_ids(40 + i, n, shape.vocab) for i, n in enumerate(lengths)]
    many = E.Engine(path, context=64, sequences=3, prefill_batch=16)
    one = E.Engine(path, context=64, prefill_batch=16)
    got, _ = many.generate_batch(prompts, 6)
    for p, t in zip(prompts, got):
        np.testing.assert_array_equal(t, one.generate(p, 6)[0])
    many.close()
    one.close()
