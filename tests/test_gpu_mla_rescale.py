"""Latent decode on scores that rise along the cache, by another amount for every head: the running maxima of a warp's rows are raised
at different tiles, and what rescales the output in tensor memory are loads and stores of whole warps.  A head without a finite score
(NaN query) beside ordinary ones takes part in them too."""
import numpy as np
import pytest

from tests.helpers import check_attention
from tests.test_gpu_attention import EDGE_MAX, EDGE_MEAN, build_mla, dev  # noqa: F401

pytestmark = pytest.mark.gpu

DH, DC, DHR = 128, 512, 64


def rising(dev, oracle, rng, ctx, rise, H):  # noqa: F811
    """A pool whose rope rows' first dim grows with the place, and queries whose first rope dim differs per head."""
    from relux_b200 import lib as L
    import relux_b200 as rb
    from tests.helpers import permuted_tables, ragged_to_padded
    B, scale = len(ctx), (DH + DHR) ** -0.5
    pages = (max(ctx) + 63) // 64
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, 64, B, pages, dC=DC, dHR=DHR)
    pool.set_tables(permuted_tables(rng, B, pages))
    c = 0.5 * rng.standard_normal((sum(ctx), DC)).astype(np.float32)
    r = 0.3 * rng.standard_normal((sum(ctx), DHR)).astype(np.float32)
    r[:, 0] = np.concatenate([np.arange(n) for n in ctx]) / 16.0
    cb, r_b = oracle.bf16_from_f32(c), oracle.bf16_from_f32(r)
    pool.append(0, cb, r_b, B, n_new=np.asarray(ctx, np.int32))
    q = rng.standard_normal((B, 1, H, DH)).astype(np.float32)
    qr = 0.3 * rng.standard_normal((B, 1, H, DHR)).astype(np.float32)
    qr[..., 0] = rise * np.log(2.0) / (scale * 128 / 16.0) * rng.uniform(0.3, 1.0, (B, 1, H))
    return pool, ragged_to_padded(cb, ctx, (DC,)), ragged_to_padded(r_b, ctx, (DHR,)), oracle.bf16_from_f32(q), oracle.bf16_from_f32(qr), scale


@pytest.mark.parametrize("H", [128, 48])
@pytest.mark.parametrize("rise", [3.0, 12.0])   # binary orders of magnitude per tile: below and above what makes the kernel rescale
def test_mla_decode_with_rising_scores(dev, oracle, H, rise):  # noqa: F811
    rng = np.random.default_rng(H)
    ctx = [900, 130, 1700, 64, 2500]
    pool, cl, rl, q, qr, scale = rising(dev, oracle, rng, ctx, rise, H)
    wuk, wuv = (oracle.bf16_from_f32(rng.standard_normal((DC, H * DH)).astype(np.float32) * 0.02) for _ in range(2))
    d_uk, d_uv = dev.upload(wuk), dev.upload(wuv)
    out = np.full(q.shape, np.nan, np.float32)
    pool.decode(0, len(ctx), q, out, H, DH, scale, q_rope=qr, w_uk=d_uk, w_uv=d_uv)
    with oracle.exact_exp():
        ref = oracle.mla_attend(cl, rl, ctx, oracle.f32_from_bf16(q), oracle.f32_from_bf16(qr), wuk, wuv, scale, absorbed=True)
    check_attention(out, ref, "rising scores", max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    # few workers, so that a range holds many tiles; the same outputs up to the order of the sums
    from relux_b200 import lib as L
    pool.tune(L.TUNE_MLA_WORKERS, 3)
    few = np.full(q.shape, np.nan, np.float32)
    pool.decode(0, len(ctx), q, few, H, DH, scale, q_rope=qr, w_uk=d_uk, w_uv=d_uv)
    check_attention(few, ref, "rising scores, three ranges", max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    assert pool.status() == 0
    pool.destroy()
    d_uk.free()
    d_uv.free()


def test_mla_decode_with_a_nan_head(dev, oracle):  # noqa: F811
    rng = np.random.default_rng(5)
    H, ctx = 128, [700, 300]
    pool, cl, rl, q, qr, scale = rising(dev, oracle, rng, ctx, 6.0, H)
    wuk, wuv = (oracle.bf16_from_f32(rng.standard_normal((DC, H * DH)).astype(np.float32) * 0.02) for _ in range(2))
    d_uk, d_uv = dev.upload(wuk), dev.upload(wuv)
    plain, out = np.empty(q.shape, np.float32), np.empty(q.shape, np.float32)
    pool.decode(0, 2, q, plain, H, DH, scale, q_rope=qr, w_uk=d_uk, w_uv=d_uv)
    bad = q.copy()
    bad[0, 0, 5] = 0x7fc0
    pool.decode(0, 2, bad, out, H, DH, scale, q_rope=qr, w_uk=d_uk, w_uv=d_uv)
    keep = np.ones((2, 1, H), bool)
    keep[0, 0, 5] = False
    assert np.array_equal(out[keep], plain[keep]) and pool.status() == 0
    pool.destroy()
    d_uk.free()
    d_uv.free()
