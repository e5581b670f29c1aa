"""Latent steps whose plan travels as kernel arguments, and whose first tile of older rows is asked for before the launch in front is complete:
against an append and a decode call, bit for bit, around the ends of pages and tiles and around the number of items that fits; and in a
captured graph, which runs with the lengths of its launch."""
import ctypes as C

import numpy as np
import pytest

from tests.helpers import permuted_tables
from tests.test_gpu_attention import dev  # noqa: F401

pytestmark = pytest.mark.gpu

H, DH, DC, DHR = 16, 128, 512, 64
SCALE = (DH + DHR) ** -0.5


def latent_pool(dev, oracle, ctx, seed):  # noqa: F811
    import relux_b200 as rb
    from relux_b200 import lib as L
    rng = np.random.default_rng(seed)
    B, pages = len(ctx), (max(ctx) + 16 + 63) // 64
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, 64, B, pages, dC=DC, dHR=DHR)
    pool.set_tables(permuted_tables(rng, B, pages))
    c, r = (oracle.bf16_from_f32(rng.standard_normal((sum(ctx), w)).astype(np.float32)) for w in (DC, DHR))
    pool.append(0, c, r, B, n_new=np.asarray(ctx, np.int32))
    return pool


def weights(dev, oracle, rng):  # noqa: F811
    return [dev.upload(oracle.bf16_from_f32(rng.standard_normal((DC, H * DH)).astype(np.float32) * 0.02)) for _ in range(2)]


@pytest.mark.parametrize("ctx,new", [([126, 127, 128, 129], 1), ([125, 126, 253, 254], 3), ([64, 190, 1000, 1], 2), ([128] * 7 + [4000], 1),
                                     ([150] * 160, 1), ([150] * 161, 1), ([40] * 100 + [300] * 40, 2)])
def test_a_step_is_append_then_decode(dev, oracle, ctx, new):  # noqa: F811
    B = len(ctx)
    rng = np.random.default_rng(B + new)
    wuk, wuv = weights(dev, oracle, rng)
    two, one = (latent_pool(dev, oracle, ctx, 7) for _ in range(2))
    for i in range(3):
        c, r = (rng.standard_normal((B * new, w)).astype(np.float32) for w in (DC, DHR))
        q, qr = (oracle.bf16_from_f32(rng.standard_normal((B, 1, H, w)).astype(np.float32)) for w in (DH, DHR))
        n_new = np.full(B, new, np.int32)
        want, got = np.empty((B, 1, H, DH), np.float32), np.full((B, 1, H, DH), np.nan, np.float32)
        two.append(0, c, r, B, n_new=n_new)
        two.decode(0, B, q, want, H, DH, SCALE, q_rope=qr, w_uk=wuk, w_uv=wuv)
        one.step(0, B, c, r, q, got, H, DH, SCALE, q_rope=qr, w_uk=wuk, w_uv=wuv, n_new=n_new)
        assert np.array_equal(got, want), i
    assert one.status() == 0 and two.status() == 0
    for b in (one, two):
        b.destroy()
    wuk.free()
    wuv.free()


def test_a_step_of_prompts(dev, oracle):  # noqa: F811
    """2048 new rows and query tokens for each of 32 sequences: a plan of few items, 65536 rows of attention."""
    import relux_b200 as rb
    from relux_b200 import lib as L
    B, S, pages = 32, 2048, 32
    rng = np.random.default_rng(3)
    wuk, wuv = weights(dev, oracle, rng)
    few = lambda w: np.tile(oracle.bf16_from_f32(rng.standard_normal((1 << 16, w)).astype(np.float32)), (B * S * H // (1 << 16), 1))  # noqa: E731
    q, qr = dev.upload(few(DH)), dev.upload(few(DHR))
    c, r = (dev.upload(oracle.bf16_from_f32(rng.standard_normal((B * S, w)).astype(np.float32))) for w in (DC, DHR))
    n_new, outs = np.full(B, S, np.int32), []
    for fused in (True, False):
        pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, 64, B, pages, dC=DC, dHR=DHR)
        pool.set_tables(permuted_tables(np.random.default_rng(4), B, pages))
        pool.tune(L.TUNE_MLA_PROMPT_MIN_TOKENS, 1 << 20)     # by the decode kernel both times
        out = dev.upload(np.full((B, S, H, DH), 0x7fc0, np.uint16))
        kw = dict(q_dtype=L.DTYPE_BF16, out_dtype=L.DTYPE_BF16)
        if fused:
            ap = pool._append_args(0, c, r, B, None, n_new, L.LAYOUT_TOKEN_MAJOR, True, L.DTYPE_BF16)
            at = pool._attn_args(0, B, q, qr, out, H, DH, SCALE, S, 0, True, L.ATTN_FAST, wuk, wuv, None, L.LAYOUT_TOKEN_MAJOR, L.LAYOUT_TOKEN_MAJOR,
                                 L.DTYPE_BF16, L.DTYPE_BF16)
            L.check(pool.lib.relux_mla_step(pool.h, C.byref(ap), C.byref(at)))
        else:
            pool.append(0, c, r, B, n_new=n_new, dtype=L.DTYPE_BF16)
            pool.decode(0, B, q, out, H, DH, SCALE, q_rope=qr, w_uk=wuk, w_uv=wuv, q_tokens=S, **kw)
        dev.sync()
        assert pool.status() == 0
        outs.append(out.download((B, S, H, DH), np.uint16))
        pool.destroy()
        out.free()
    assert np.array_equal(outs[0], outs[1]) and not (outs[0] == 0x7fc0).any()
    for b in (q, qr, c, r, wuk, wuv):
        b.free()


def test_a_captured_step_runs_with_the_lengths_of_its_launch(dev, oracle):  # noqa: F811
    from relux_b200 import lib as L
    rt = C.CDLL("libcudart.so.12")
    ctx = [70, 300, 130]
    B = len(ctx)
    rng = np.random.default_rng(11)
    wuk, wuv = weights(dev, oracle, rng)
    plain, graphed = (latent_pool(dev, oracle, ctx, 8) for _ in range(2))
    q, qr = (dev.upload(oracle.bf16_from_f32(rng.standard_normal((B, 1, H, w)).astype(np.float32))) for w in (DH, DHR))
    c, r = (dev.upload(oracle.bf16_from_f32(rng.standard_normal((B, w)).astype(np.float32))) for w in (DC, DHR))
    outs = [dev.upload(np.zeros((B, 1, H, DH), np.float32)) for _ in range(2)]

    def step(pool, out):
        pool.step(0, B, c, r, q, out, H, DH, SCALE, q_rope=qr, w_uk=wuk, w_uv=wuv, q_dtype=L.DTYPE_BF16, out_dtype=L.DTYPE_F32, kv_dtype=L.DTYPE_BF16)

    for pool, out in ((plain, outs[0]), (graphed, outs[1])):
        step(pool, out)                          # everything that a first call sets up
    dev.sync()
    stream, graph, ready = C.c_void_p(), C.c_void_p(), C.c_void_p()
    L.check(dev.lib.relux_cuda_stream(dev.h, C.byref(stream)))
    assert rt.cudaStreamBeginCapture(stream, 2) == 0
    step(graphed, outs[1])
    assert rt.cudaStreamEndCapture(stream, C.byref(graph)) == 0
    assert rt.cudaGraphInstantiate(C.byref(ready), graph, C.c_ulonglong(0)) == 0
    for i in range(4):
        step(plain, outs[0])
        assert rt.cudaGraphLaunch(ready, stream) == 0
        dev.sync()
        want, got = (o.download((B, 1, H, DH), np.float32) for o in outs)
        # a graph's rows are always kept in two halves: its numbers are those of a plain call up to the rounding of one
        assert np.max(np.abs(want - got)) <= 2e-2 * np.sqrt(np.mean(want ** 2)), i
    assert rt.cudaGraphExecDestroy(ready) == 0 and rt.cudaGraphDestroy(graph) == 0
    assert plain.status() == 0 and graphed.status() == 0
    for p in (plain, graphed):
        p.destroy()
    for b in [q, qr, c, r, wuk, wuv] + outs:
        b.free()
