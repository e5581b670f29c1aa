"""Prompt attention on scores that rise along the keys, so that the running maximum of every row is raised in tile after tile and the
output is rescaled in tensor memory: by whole warps, at different tiles for different rows, in both output accumulators."""
import numpy as np
import pytest

from tests.helpers import check_attention
from tests.test_gpu_attention import EDGE_MAX, EDGE_MEAN, dev  # noqa: F401

pytestmark = pytest.mark.gpu


# one block pair, several, an odd number of pairs; one row per token up to 32; rows past the last token; a cached part before
@pytest.mark.parametrize("H,Hkv,S,cached", [(8, 8, 129, 0), (16, 8, 300, 64), (32, 8, 150, 261), (32, 2, 95, 700), (32, 1, 41, 130), (8, 2, 1100, 0)])
@pytest.mark.parametrize("rise", [3.0, 14.0])   # binary orders of magnitude per 128 keys: below and above the rescale's threshold
def test_gqa_prompt_with_rising_scores(dev, oracle, H, Hkv, S, cached, rise):  # noqa: F811
    import relux_b200 as rb
    from relux_b200 import lib as L
    rng = np.random.default_rng(S + Hkv)
    B, D, P = 2, 128, 64
    scale = D ** -0.5
    ctx = np.asarray([cached + S, cached + S + 37], np.int32)
    T = int(ctx.max())
    pages = (T + P - 1) // P
    pool = rb.Pool(dev, L.POOL_GQA, 1, B * pages, P, B, pages, num_kv_heads=Hkv, head_dim=D)
    pool.set_tables(rng.permutation(B * pages).astype(np.int32).reshape(B, pages))
    # the first dim of a key grows with its place; the query's first dim differs per row, so rows are raised at different tiles
    K = 0.3 * rng.standard_normal((B, T, Hkv, D)).astype(np.float32)
    K[..., 0] = np.arange(T, dtype=np.float32)[None, :, None] / 16.0
    V = rng.standard_normal((B, T, Hkv, D)).astype(np.float32)
    kb, vb = oracle.bf16_from_f32(K), oracle.bf16_from_f32(V)
    pool.append(0, np.concatenate([kb[i, :ctx[i]] for i in range(B)]), np.concatenate([vb[i, :ctx[i]] for i in range(B)]), B, n_new=ctx)
    q = 0.3 * rng.standard_normal((B, S, H, D)).astype(np.float32)
    q[..., 0] = rise * np.log(2.0) / (scale * 128 / 16.0) * rng.uniform(0.4, 1.0, (B, S, H))
    qb = oracle.bf16_from_f32(q)
    out = np.full(q.shape, np.nan, np.float32)
    pool.decode(0, B, qb, out, H, D, scale, q_tokens=S)
    for i in range(B):
        kb[i, ctx[i]:] = 0
        vb[i, ctx[i]:] = 0
    with oracle.exact_exp():
        ref = oracle.gqa_attend(kb, vb, ctx, oracle.f32_from_bf16(qb), scale, causal=True)
    check_attention(out, ref, "rising scores", max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    assert pool.status() == 0
    pool.destroy()


# the 192-wide kernel over expanded rows: one block pair, several, rows past the last token, a cached part before
@pytest.mark.parametrize("S,cached", [(128, 0), (300, 64), (131, 517), (1100, 0)])
@pytest.mark.parametrize("rise", [3.0, 14.0])
def test_mla_prompt_with_rising_scores(dev, oracle, S, cached, rise):  # noqa: F811
    import relux_b200 as rb
    from relux_b200 import lib as L
    rng = np.random.default_rng(S)
    H, DH, DC, DHR, P, B = 16, 128, 512, 64, 64, 2
    scale = (DH + DHR) ** -0.5
    ctx = np.asarray([cached + S, cached + S + 37], np.int32)
    T = int(ctx.max())
    pages = (T + P - 1) // P
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, P, B, pages, dC=DC, dHR=DHR)
    pool.set_tables(rng.permutation(B * pages).astype(np.int32).reshape(B, pages))
    c = 0.3 * rng.standard_normal((B, T, DC)).astype(np.float32)
    r = 0.3 * rng.standard_normal((B, T, DHR)).astype(np.float32)
    r[..., 0] = np.arange(T, dtype=np.float32)[None] / 16.0
    cb, rb_ = oracle.bf16_from_f32(c), oracle.bf16_from_f32(r)
    pool.append(0, np.concatenate([cb[i, :ctx[i]] for i in range(B)]), np.concatenate([rb_[i, :ctx[i]] for i in range(B)]), B, n_new=ctx)
    q = oracle.bf16_from_f32(0.3 * rng.standard_normal((B, S, H, DH)).astype(np.float32))
    qr = 0.3 * rng.standard_normal((B, S, H, DHR)).astype(np.float32)
    qr[..., 0] = rise * np.log(2.0) / (scale * 128 / 16.0) * rng.uniform(0.4, 1.0, (B, S, H))
    qr = oracle.bf16_from_f32(qr)
    wuk, wuv = (oracle.bf16_from_f32(rng.standard_normal((DC, H * DH)).astype(np.float32) * 0.02) for _ in range(2))
    d_uk, d_uv = dev.upload(wuk), dev.upload(wuv)
    out = np.full(q.shape, np.nan, np.float32)
    pool.decode(0, B, q, out, H, DH, scale, q_rope=qr, w_uk=d_uk, w_uv=d_uv, q_tokens=S)
    for i in range(B):
        cb[i, ctx[i]:] = 0
        rb_[i, ctx[i]:] = 0
    with oracle.exact_exp():
        ref = oracle.mla_attend(cb, rb_, ctx, oracle.f32_from_bf16(q), oracle.f32_from_bf16(qr), wuk, wuv, scale, causal=True,
                                absorbed=False)
    check_attention(out, ref, "rising scores, expanded", max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    assert pool.status() == 0
    pool.destroy()
    d_uk.free()
    d_uv.free()
