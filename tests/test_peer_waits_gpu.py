"""Waits of a cluster's CTAs for one another's values: every one is bounded, says so in its own status word when it runs
out, and leaves the context usable.  A barrier that expects more than is sent makes it run out."""
import contextlib
import ctypes as C
import dataclasses
import time

import numpy as np
import pytest

from tuckmill_b200 import cuda, engine as E, testing as T

pytestmark = pytest.mark.gpu

LIMIT = 2000  # polls: past the first look at the status word


class Attention:
    starved, heads, kvh, hd, cap, pos = (1,), 4, 2, 128, 300, 200

    def __init__(self, c, oracle):
        hd, plane = self.hd, self.kvh * self.cap * self.hd
        self.ops = [c.floats(T.activations(7, t, n * hd)) for t, n in ((30, self.heads), (31, self.kvh), (32, self.kvh))]
        one, self.out = c.floats(np.ones(hd)), c.buffer(self.heads * hd * 4)
        self.ops += [one, one, c.floats(oracle.rope_inv_freq(hd, 1e6))]
        self.ops += [c.from_array(T.activations(1, t, plane).astype(np.float16)) for t in (1, 2)]
        self.scratch = c.buffer(cuda.decode_attention_scratch_bytes(self.heads, self.kvh, hd, self.cap))
        self.pb, self.status = c.from_array(np.array([self.pos], np.uint32)), c.buffer(4, shared=True)
        self.scratch.zero(), self.status.zero()

    def run(self, c):
        c.attention_decode_dev(*self.ops, self.out, self.scratch, self.pb, 0, self.status, self.heads, self.kvh, self.hd, self.hd,
                               self.cap, 0, 1e-6, self.hd ** -0.5, False)

    def result(self):
        return self.out.download(0, self.heads * self.hd * 4, np.float32)

    def words(self, c):
        return int(self.status.download(0, 4, np.uint32)[0]), c.mma_aborted()


class Block:
    hidden, width, heads, kvh, hd, cap, pos = 256, 1024, 4, 2, 128, 300, 200

    def __init__(self, c, oracle):
        H, hd = self.hidden, self.hd
        vec = lambda t: c.floats((1 + 0.1 * T.activations(4, t, H)).astype(np.float32))  # noqa: E731
        mat = lambda t, r, k: c.q8_0_matrix(T.q8_0_matrix(4, t, r, k), r, k)  # noqa: E731
        self.x, self.nw, self.xo, self.so = c.floats(T.activations(4, 3, H)), vec(4), c.buffer(H * 4), c.buffer(8 * H * 4)
        self.qkv, self.o = mat(1, (self.heads + 2 * self.kvh) * hd, H), mat(2, H, self.heads * hd)
        self.gu, self.dn = mat(5, 2 * self.width, H), mat(6, H, self.width)
        self.kc, self.vc = (c.from_array(T.activations(4, t, self.kvh * self.cap * hd).astype(np.float16)) for t in (30, 31))
        self.qn, self.inv = c.floats(np.ones(hd)), c.floats(oracle.rope_inv_freq(hd, 1e6))
        self.pb, self.status = c.from_array(np.array([self.pos], np.uint32)), c.buffer(4, shared=True)
        self.so.zero(), self.status.zero()

    def result(self):
        return self.so.download(0, 8 * self.hidden * 4, np.float32)

    def words(self, c):
        return int(self.status.download(0, 4, np.uint32)[0]), c.mma_aborted()


class AttentionBlock(Block):
    starved = (1, 2)

    def run(self, c):
        c.decode_attn_block(self.x, None, 0, None, self.nw, self.xo, self.qkv, self.o, self.qn, self.qn, self.inv, self.kc, self.vc,
                            self.pb, 0, self.status, self.so, self.hidden, self.heads, self.kvh, self.hd, self.cap, 0, 1e-6,
                            self.hd ** -0.5)


class FeedForwardBlock(Block):
    starved = (1,)

    def run(self, c):
        c.decode_ffn_block(self.x, None, 0, None, self.nw, self.xo, self.gu, self.dn, self.so, self.hidden, self.width, False, 1e-6)


class SplitMultiply:
    starved, rows, cols, tokens = (1, 2), 1024, 3072, 48

    def __init__(self, c, oracle):
        self.w = c.q8_0_matrix(T.q8_0_matrix(11, 1, self.rows, self.cols), self.rows, self.cols)
        self.x, self.y = c.floats(T.activations(11, 5, self.tokens * self.cols)), c.buffer(self.tokens * self.rows * 4)

    def run(self, c):
        c.q8_0_gemm_mma(self.w, self.x, self.y, self.rows, self.cols, self.tokens)
        assert c.mma_last_split() > 1  # (its parts fit as clusters)

    def result(self):
        return self.y.download(0, self.tokens * self.rows * 4, np.float32)

    def words(self, c):
        return 0, c.mma_aborted()


@pytest.mark.parametrize("op,starve", [(op, s) for op in (Attention, AttentionBlock, FeedForwardBlock, SplitMultiply)
                                       for s in op.starved])
def test_a_wait_that_runs_out_says_so_and_ends(ctx, oracle, op, starve):
    with contextlib.closing(cuda.CudaContext(0)) as c:  # the word of a context stays set
        o = op(c, oracle)
        o.run(c)
        want = o.result()
        assert o.words(c) == (0, False)
        c.wait_debug(starve, LIMIT)
        o.run(c)
        c.fence()
        assert o.words(c) == ((cuda.STATUS_LATE, False) if op is Attention else (0, True))
        # what is launched behind it does not wait its own time out: 20 launches of a second each
        c.wait_debug(starve, 0)
        if op is not SplitMultiply:  # (which has a word of its own in every CTA)
            t = time.perf_counter()
            for _ in range(20):
                o.run(c)
            c.fence()
            assert time.perf_counter() - t < 1.0
        c.wait_debug()
        o.run(c)
        np.testing.assert_array_equal(o.result(), want)


def starved_engine_message(path, prompt, **kw):
    """What an engine says after a step whose waits ran out."""
    eng = E.Engine(path, context=128, **kw)
    eng.prefill(prompt, want_token=True)
    err = C.create_string_buffer(256)
    assert cuda.load_library().tm_cuda_wait_debug(C.c_void_p(eng.cuda_ctx()), 1, LIMIT, err, 256) == 0
    eng.decode_ungrouped(1)
    with pytest.raises(E.EngineError) as e:
        eng.logits()
    eng.close()
    assert e.value.code == "INTERNAL"
    return e.value.message


def test_the_engine_names_the_wait(ctx, tmp_path):
    prompt = T.token_ids(3, 9, 512)
    # no layer has the blocks' shape: decode attention by itself
    wide = dataclasses.replace(T.SMALL_QWEN3, hidden=2304)
    assert not cuda.load_library().tm_cuda_decode_attn_block_supported(2304, wide.heads, wide.kv_heads, wide.head_dim, wide.head_dim)
    T.write_gguf(tmp_path / "wide.gguf", wide)
    message = starved_engine_message(tmp_path / "wide.gguf", prompt)
    assert "decode attention" in message and "capacity" not in message
    T.write_gguf(tmp_path / "small.gguf", T.SMALL_QWEN3)
    assert "decode layer" in starved_engine_message(tmp_path / "small.gguf", prompt)
