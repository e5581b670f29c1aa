"""The absorb of the queries around the rows that choose its kernel (32), its tiles (16, 64 rows) and the chunks of latent columns that a CTA takes
(one, two or four by the number of heads), for bf16 and float32 queries, as a step (with its append) and as a decode call."""
import numpy as np
import pytest

from tests.helpers import check_attention, permuted_tables, ragged_to_padded
from tests.test_gpu_attention import EDGE_MAX, EDGE_MEAN, dev  # noqa: F401

pytestmark = pytest.mark.gpu

DH, DHR = 128, 64


@pytest.mark.parametrize("B,H,dc,f32,step", [(1, 128, 512, False, True), (16, 37, 512, True, True), (17, 16, 512, False, False), (32, 38, 512, False, True),
                                             (33, 38, 512, False, True), (33, 37, 512, True, True), (64, 75, 512, False, False), (65, 75, 512, True, True),
                                             (100, 16, 512, False, True), (40, 128, 512, False, True), (129, 74, 512, False, False),
                                             (33, 16, 128, False, False), (70, 80, 128, True, False), (33, 80, 256, False, False), (20, 16, 256, True, False)])
def test_rows_heads_and_latents(dev, oracle, B, H, dc, f32, step):  # noqa: F811
    from relux_b200 import lib as L
    import relux_b200 as rb
    rng = np.random.default_rng(B * 1000 + H)
    ctx = [int(n) for n in rng.integers(2, 40, B)]
    pool = rb.Pool(dev, L.POOL_MLA, 1, B, 64, B, 1, dC=dc, dHR=DHR)
    pool.set_tables(permuted_tables(rng, B, 1))
    c, r = (oracle.bf16_from_f32(rng.standard_normal((sum(ctx), w)).astype(np.float32)) for w in (dc, DHR))
    q, qr = (rng.standard_normal((B, 1, H, w)).astype(np.float32) for w in (DH, DHR))
    qb, qrb = oracle.bf16_from_f32(q), oracle.bf16_from_f32(qr)
    wuk, wuv = (oracle.bf16_from_f32(rng.standard_normal((dc, H * DH)).astype(np.float32) * 0.02) for _ in range(2))
    d_uk, d_uv = dev.upload(wuk), dev.upload(wuv)
    out = np.full((B, 1, H, DH), np.nan, np.float32)
    scale = (DH + DHR) ** -0.5
    kw = dict(q_rope=qr if f32 else qrb, w_uk=d_uk, w_uv=d_uv)
    if step:
        last = np.cumsum(ctx) - 1
        old = np.setdiff1d(np.arange(sum(ctx)), last)
        pool.append(0, c[old], r[old], B, n_new=np.asarray(ctx, np.int32) - 1)
        pool.step(0, B, c[last], r[last], q if f32 else qb, out, H, DH, scale, **kw)
    else:
        pool.append(0, c, r, B, n_new=np.asarray(ctx, np.int32))
        pool.decode(0, B, q if f32 else qb, out, H, DH, scale, **kw)
    with oracle.exact_exp():
        ref = oracle.mla_attend(ragged_to_padded(c, ctx, (dc,)), ragged_to_padded(r, ctx, (DHR,)), ctx, oracle.f32_from_bf16(qb), oracle.f32_from_bf16(qrb),
                                wuk, wuv, scale, absorbed=True)
    check_attention(out, ref, "%d rows, %d heads, latent %d" % (B, H, dc), max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    assert [pool.seq_len(0, i) for i in range(B)] == ctx
    assert pool.status() == 0
    pool.destroy()
    d_uk.free()
    d_uv.free()
