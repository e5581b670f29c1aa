"""Merge of the split partials and up-projection on either side of the row counts that choose the kernel and its tile (16, 32, 64 rows
of a block), with sequences of one item, of more than 32 items, and several query tokens to a sequence."""
import numpy as np
import pytest

from tests.helpers import check_attention, permuted_tables, ragged_to_padded
from tests.test_gpu_attention import EDGE_MAX, EDGE_MEAN, dev  # noqa: F401

pytestmark = pytest.mark.gpu

DH, DC, DHR = 128, 512, 64


@pytest.mark.parametrize("B,S,H,out_bf16", [(16, 1, 16, False), (17, 1, 16, False), (17, 1, 128, True), (32, 1, 16, False), (33, 1, 32, True),
                                            (64, 1, 16, False), (65, 1, 16, False), (80, 1, 16, False), (9, 2, 16, False), (20, 4, 16, True)])
def test_merge_and_up_projection_of_any_row_count(dev, oracle, B, S, H, out_bf16):  # noqa: F811
    from relux_b200 import lib as L
    import relux_b200 as rb
    rng = np.random.default_rng(B * 100 + S)
    ctx = [int(n) for n in rng.integers(S, 150, B)]
    ctx[B // 2] = 4200                          # alone it fills most of the ranges: more than 32 items of one sequence
    pages = (max(ctx) + 63) // 64
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, 64, B, pages, dC=DC, dHR=DHR)
    pool.set_tables(permuted_tables(rng, B, pages))
    c, r = (oracle.bf16_from_f32(rng.standard_normal((sum(ctx), w)).astype(np.float32)) for w in (DC, DHR))
    pool.append(0, c, r, B, n_new=np.asarray(ctx, np.int32))
    pool.tune(L.TUNE_CHUNK_PAGES, 2)
    q, qr = (oracle.bf16_from_f32(rng.standard_normal((B, S, H, w)).astype(np.float32)) for w in (DH, DHR))
    wuk, wuv = (oracle.bf16_from_f32(rng.standard_normal((DC, H * DH)).astype(np.float32) * 0.02) for _ in range(2))
    d_uk, d_uv = dev.upload(wuk), dev.upload(wuv)
    out = np.full((B, S, H, DH), 0x7fc0 if out_bf16 else np.nan, np.uint16 if out_bf16 else np.float32)
    scale = (DH + DHR) ** -0.5
    pool.decode(0, B, q, out, H, DH, scale, q_rope=qr, w_uk=d_uk, w_uv=d_uv, q_tokens=S)
    with oracle.exact_exp():
        ref = oracle.mla_attend(ragged_to_padded(c, ctx, (DC,)), ragged_to_padded(r, ctx, (DHR,)), ctx, oracle.f32_from_bf16(q),
                                oracle.f32_from_bf16(qr), wuk, wuv, scale, absorbed=True)
    got = oracle.f32_from_bf16(out) if out_bf16 else out
    check_attention(got, ref, "merge of %d x %d rows" % (B, S), bf16_output=out_bf16, max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    assert pool.status() == 0
    pool.destroy()
    d_uk.free()
    d_uv.free()


@pytest.mark.parametrize("B,S,H,dc,out_bf16", [(17, 1, 16, 128, False), (33, 1, 32, 128, True), (65, 1, 16, 128, False), (17, 1, 128, 256, False),
                                               (33, 1, 16, 256, True), (65, 1, 16, 256, False), (12, 4, 16, 256, False)])
def test_merge_of_narrower_latents(dev, oracle, B, S, H, dc, out_bf16):  # noqa: F811
    from relux_b200 import lib as L
    import relux_b200 as rb
    rng = np.random.default_rng(B * 100 + dc)
    ctx = [int(n) for n in rng.integers(S, 150, B)]
    ctx[B // 2] = 2200                          # pieces of one page: 35 items of one sequence
    pages = (max(ctx) + 63) // 64
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, 64, B, pages, dC=dc, dHR=DHR)
    pool.set_tables(permuted_tables(rng, B, pages))
    c, r = (oracle.bf16_from_f32(rng.standard_normal((sum(ctx), w)).astype(np.float32)) for w in (dc, DHR))
    pool.append(0, c, r, B, n_new=np.asarray(ctx, np.int32))
    pool.tune(L.TUNE_CHUNK_PAGES, 1)
    q, qr = (oracle.bf16_from_f32(rng.standard_normal((B, S, H, w)).astype(np.float32)) for w in (DH, DHR))
    wuk, wuv = (oracle.bf16_from_f32(rng.standard_normal((dc, H * DH)).astype(np.float32) * 0.02) for _ in range(2))
    d_uk, d_uv = dev.upload(wuk), dev.upload(wuv)
    out = np.full((B, S, H, DH), 0x7fc0 if out_bf16 else np.nan, np.uint16 if out_bf16 else np.float32)
    scale = (DH + DHR) ** -0.5
    pool.decode(0, B, q, out, H, DH, scale, q_rope=qr, w_uk=d_uk, w_uv=d_uv, q_tokens=S)
    with oracle.exact_exp():
        ref = oracle.mla_attend(ragged_to_padded(c, ctx, (dc,)), ragged_to_padded(r, ctx, (DHR,)), ctx, oracle.f32_from_bf16(q),
                                oracle.f32_from_bf16(qr), wuk, wuv, scale, absorbed=True)
    got = oracle.f32_from_bf16(out) if out_bf16 else out
    check_attention(got, ref, "latent of %d, %d x %d rows" % (dc, B, S), bf16_output=out_bf16, max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    assert pool.status() == 0
    pool.destroy()
    d_uk.free()
    d_uv.free()
