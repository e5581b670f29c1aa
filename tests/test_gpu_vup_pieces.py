"""The up-projection of a latent call's pieces where its blocks, stages and groups end: rows of one piece (one bf16 half), rows of many (two),
more columns than a block (96, 192), than a CTA (240), and a sequence that the knob would cut into more pieces than a CTA takes."""
import numpy as np
import pytest

from tests.helpers import check_attention, permuted_tables, ragged_to_padded
from tests.test_gpu_attention import EDGE_MAX, EDGE_MEAN, dev  # noqa: F401

pytestmark = pytest.mark.gpu

DH, DC, DHR = 128, 512, 64


@pytest.mark.parametrize("ctx,H,chunk,S,out_bf16", [
    ([100] * 15, 16, 0, 1, False), ([100] * 16, 24, 0, 1, True), ([100] * 17, 100, 0, 1, False), ([70] * 70, 16, 0, 1, False),   # one piece a row
    ([128 * 12], 17, 2, 1, False), ([128 * 95 + 1], 16, 2, 1, True), ([128 * 96 + 1], 16, 2, 1, False), ([128 * 191 + 5, 300], 16, 2, 1, False),
    ([60 + i % 9 for i in range(245)], 75, 0, 1, False),   # more columns than a CTA has room for, and one group of heads' CTAs
    ([1, 200, 3, 130 * 5, 64], 16, 2, 1, False),
    ([128 * 260], 16, 2, 1, False),                         # 260 pieces asked for
    ([900, 1500, 64], 40, 2, 3, False),
])
def test_pieces_at_the_borders_of_blocks_and_groups(dev, oracle, ctx, H, chunk, S, out_bf16):  # noqa: F811
    from relux_b200 import lib as L
    import relux_b200 as rb
    rng = np.random.default_rng(len(ctx) * 100 + H)
    B, pages = len(ctx), (max(ctx) + 63) // 64
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, 64, B, pages, dC=DC, dHR=DHR)
    pool.set_tables(permuted_tables(rng, B, pages))
    c, r = (oracle.bf16_from_f32(rng.standard_normal((sum(ctx), w)).astype(np.float32)) for w in (DC, DHR))
    pool.append(0, c, r, B, n_new=np.asarray(ctx, np.int32))
    if chunk:
        pool.tune(L.TUNE_CHUNK_PAGES, chunk)
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
    for b in range(B):
        if ctx[b] == 0:
            assert not got[b].any()
            ref[b] = 0.0
    check_attention(got, ref, "pieces of %d sequences, %d heads" % (B, H), bf16_output=out_bf16, max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    assert pool.status() == 0
    pool.destroy()
    d_uk.free()
    d_uv.free()


def test_more_workers_than_a_row_may_have_pieces(dev, oracle):  # noqa: F811
    """The knob MLA_WORKERS asks for 1000 ranges: 4100 pages of one sequence and a short one beside it, against the plan of the call's choice."""
    from relux_b200 import lib as L
    import relux_b200 as rb
    rng = np.random.default_rng(12)
    ctx, H, pages = [4100 * 64 - 5, 300], 16, 4100
    pool = rb.Pool(dev, L.POOL_MLA, 1, 2 * pages, 64, 2, pages, dC=DC, dHR=DHR)
    pool.set_tables(permuted_tables(rng, 2, pages))
    block = [oracle.bf16_from_f32(rng.standard_normal((4096, w)).astype(np.float32)) for w in (DC, DHR)]
    for at in range(0, max(ctx), 4096):
        n = [min(4096, max(0, c - at)) for c in ctx]
        pool.append(0, *(np.concatenate([x[:k] for k in n]) for x in block), 2, n_new=np.asarray(n, np.int32))
    q, qr = (oracle.bf16_from_f32(rng.standard_normal((2, 1, H, w)).astype(np.float32)) for w in (DH, DHR))
    wuk, wuv = (dev.upload(oracle.bf16_from_f32(rng.standard_normal((DC, H * DH)).astype(np.float32) * 0.02)) for _ in range(2))
    outs = []
    for workers in (0, 241, 1000, 1 << 20):
        pool.tune(L.TUNE_MLA_WORKERS, workers)
        outs.append(np.full((2, 1, H, DH), np.nan, np.float32))
        pool.decode(0, 2, q, outs[-1], H, DH, (DH + DHR) ** -0.5, q_rope=qr, w_uk=wuk, w_uv=wuv)
    # P is rounded to 8 bits against other maxima: 2^-9 of a value with a random sign, over the largest of 4096 values
    for out in outs[1:]:
        assert np.isfinite(out).all() and np.max(np.abs(out - outs[0])) <= 2e-2 * np.sqrt(np.mean(outs[0] ** 2))
    assert pool.status() == 0
    pool.destroy()
    wuk.free()
    wuv.free()


def test_chunks_of_other_calls_have_no_such_limit(dev, oracle):  # noqa: F811
    """A grouped-query prompt in slices takes chunks as short as the knob says over 300 pages as over 60: pieces of one page and of two add up in another
    order, so that their bits differ."""
    from relux_b200 import lib as L
    from tests.test_gpu_attention import build_gqa
    H, Hkv, D, S = 16, 8, 128, 40
    for tokens in (60 * 64, 300 * 64):
        rng = np.random.default_rng(tokens)
        pool = build_gqa(dev, oracle, rng, [tokens], Hkv, D)[0]
        pool.tune(L.TUNE_GQA_PROMPT_SLICES, 1)
        q, outs = rng.standard_normal((1, S, H, D)).astype(np.float32), []
        for pages in (1, 2, 1):
            pool.tune(L.TUNE_CHUNK_PAGES, pages)
            outs.append(np.empty_like(q))
            pool.decode(0, 1, q, outs[-1], H, D, D ** -0.5, q_tokens=S)
        assert np.array_equal(outs[0], outs[2]) and not np.array_equal(outs[0], outs[1])
        assert np.max(np.abs(outs[0] - outs[1])) <= 1e-2 * np.sqrt(np.mean(outs[0] ** 2)) + 5e-3
        pool.destroy()
