"""Latent decode with one item a worker (short calls) and with ranges over several sequences give the same attention: lengths at the
edges of pages and tiles, sequences without rows, more items than workers allow, draft rows; in a step's preparation and by itself."""
import numpy as np
import pytest

from tests.helpers import check_attention, permuted_tables, ragged_to_padded
from tests.test_gpu_attention import EDGE_MAX, EDGE_MEAN, dev  # noqa: F401

pytestmark = pytest.mark.gpu

DH, DC, DHR, H = 128, 512, 64, 16


@pytest.mark.parametrize("ctx,S", [([300], 1), ([64, 65, 128, 129], 1), ([1, 2100, 63, 640], 1), ([600] * 9, 1), ([127] * 37, 1), ([129] * 37, 1),
                                   ([129] * 38, 1), ([1500, 100, 900], 4), ([200] * 75, 1), ([2000] * 20, 1), ([4, 700, 5], 2)])
def test_both_plans(dev, oracle, ctx, S):  # noqa: F811
    from relux_b200 import lib as L
    import relux_b200 as rb
    rng = np.random.default_rng(len(ctx) * 10 + S)
    B, pages = len(ctx), (max(ctx) + 63) // 64 + 1
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, 64, B, pages, dC=DC, dHR=DHR)
    pool.set_tables(permuted_tables(rng, B, pages))
    c, r = (oracle.bf16_from_f32(rng.standard_normal((sum(ctx), w)).astype(np.float32)) for w in (DC, DHR))
    first = np.cumsum([0] + ctx[:-1])
    last = first + np.asarray(ctx) - 1
    keep = np.ones(sum(ctx), bool)
    keep[last] = False                          # the last row of every sequence comes with a step
    pool.append(0, c[keep], r[keep], B, n_new=np.asarray(ctx, np.int32) - 1)
    q, qr = (oracle.bf16_from_f32(rng.standard_normal((B, S, H, w)).astype(np.float32)) for w in (DH, DHR))
    wuk, wuv = (oracle.bf16_from_f32(rng.standard_normal((DC, H * DH)).astype(np.float32) * 0.02) for _ in range(2))
    d_uk, d_uv = dev.upload(wuk), dev.upload(wuv)
    scale = (DH + DHR) ** -0.5
    kw = dict(q_rope=qr, w_uk=d_uk, w_uv=d_uv)
    outs = []
    if S == 1:
        out = np.full((B, 1, H, DH), np.nan, np.float32)
        pool.step(0, B, c[last], r[last], q, out, H, DH, scale, **kw)
        outs.append(out)
    else:
        pool.append(0, c[last], r[last], B)
    for chunk in (0, 4):                        # the plan of its choice, and ranges of two tiles
        pool.tune(L.TUNE_CHUNK_PAGES, chunk)
        out = np.full((B, S, H, DH), np.nan, np.float32)
        pool.decode(0, B, q, out, H, DH, scale, q_tokens=S, **kw)
        outs.append(out)
    with oracle.exact_exp():
        ref = oracle.mla_attend(ragged_to_padded(c, ctx, (DC,)), ragged_to_padded(r, ctx, (DHR,)), ctx, oracle.f32_from_bf16(q),
                                oracle.f32_from_bf16(qr), wuk, wuv, scale, absorbed=True)
    for k, out in enumerate(outs):
        check_attention(out, ref, "plan %d of %d sequences" % (k, B), max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    assert pool.status() == 0
    pool.destroy()
    d_uk.free()
    d_uv.free()


def test_a_call_with_an_empty_sequence(dev, oracle):  # noqa: F811
    """A step in which one of the named sequences has no row yet besides its new one."""
    from relux_b200 import lib as L
    import relux_b200 as rb
    rng = np.random.default_rng(8)
    pool = rb.Pool(dev, L.POOL_MLA, 1, 12, 64, 3, 4, dC=DC, dHR=DHR)
    pool.set_tables(permuted_tables(rng, 3, 4))
    n_old = [130, 0, 64]
    c, r = (oracle.bf16_from_f32(rng.standard_normal((sum(n_old) + 3, w)).astype(np.float32)) for w in (DC, DHR))
    pool.append(0, c[:194], r[:194], 3, n_new=np.asarray(n_old, np.int32))
    q, qr = (oracle.bf16_from_f32(rng.standard_normal((3, 1, H, w)).astype(np.float32)) for w in (DH, DHR))
    wuk, wuv = (oracle.bf16_from_f32(rng.standard_normal((DC, H * DH)).astype(np.float32) * 0.02) for _ in range(2))
    d_uk, d_uv = dev.upload(wuk), dev.upload(wuv)
    out = np.full((3, 1, H, DH), np.nan, np.float32)
    pool.step(0, 3, c[194:], r[194:], q, out, H, DH, (DH + DHR) ** -0.5, q_rope=qr, w_uk=d_uk, w_uv=d_uv)
    order = list(range(130)) + [194, 195] + list(range(130, 194)) + [196]
    ctx = [131, 1, 65]
    with oracle.exact_exp():
        ref = oracle.mla_attend(ragged_to_padded(c[order], ctx, (DC,)), ragged_to_padded(r[order], ctx, (DHR,)), ctx, oracle.f32_from_bf16(q),
                                oracle.f32_from_bf16(qr), wuk, wuv, (DH + DHR) ** -0.5, absorbed=True)
    check_attention(out, ref, "an empty sequence", max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    pool.destroy()
    d_uk.free()
    d_uv.free()


@pytest.mark.parametrize("ctx,heads", [([100, 90, 70, 3], 16), ([500] * 40, 32), ([299] * 64, 128)])
def test_one_piece_is_rounded_once_it_is_an_average(dev, oracle, ctx, heads):  # noqa: F811
    """All of a sequence's rows are the same, so that its attention is that row, exactly, in bf16: the output is its projection in float32.  Rounded
    ahead of the division by the number of rows it would be off by 2^-9.  (512 products, summed in float32: 1e-5 of the result's size.)"""
    from relux_b200 import lib as L
    import relux_b200 as rb
    rng = np.random.default_rng(heads)
    B, pages = len(ctx), (max(ctx) + 63) // 64
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, 64, B, pages, dC=DC, dHR=DHR)
    pool.set_tables(permuted_tables(rng, B, pages))
    c, r = (oracle.bf16_from_f32(rng.standard_normal((B, w)).astype(np.float32)) for w in (DC, DHR))
    pool.append(0, np.repeat(c, ctx, axis=0), np.repeat(r, ctx, axis=0), B, n_new=np.asarray(ctx, np.int32))
    q, qr = (oracle.bf16_from_f32(rng.standard_normal((B, 1, heads, w)).astype(np.float32)) for w in (DH, DHR))
    wuk, wuv = (oracle.bf16_from_f32(rng.standard_normal((DC, heads * DH)).astype(np.float32) * 0.02) for _ in range(2))
    d_uk, d_uv = dev.upload(wuk), dev.upload(wuv)
    out = np.full((B, 1, heads, DH), np.nan, np.float32)
    pool.decode(0, B, q, out, heads, DH, (DH + DHR) ** -0.5, q_rope=qr, w_uk=d_uk, w_uv=d_uv)
    ref = (oracle.f32_from_bf16(c).astype(np.float64) @ oracle.f32_from_bf16(wuv)).reshape(out.shape)
    assert np.max(np.abs(out - ref)) <= 1e-5 * np.sqrt(np.mean(ref ** 2))
    pool.destroy()
    d_uk.free()
    d_uv.free()
