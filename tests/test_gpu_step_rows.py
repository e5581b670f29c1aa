"""Row counts at which the kernels around an MLA decode step change their division of work (row groups of 16, warps that share a
row, blocks of 64 rows), and appends of the same number of rows per sequence (several rows per block, page crossings)."""
import numpy as np
import pytest

from tests.helpers import check_attention, permuted_tables, ragged_to_padded
from tests.test_gpu_attention import EDGE_MAX, EDGE_MEAN, build_mla, dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 150])
@pytest.mark.parametrize("q_bf16", [False, True])
def test_mla_step_rows(dev, oracle, B, q_bf16):  # noqa: F811
    H, Dh, dC, dHR = 16, 128, 512, 64
    rng = np.random.default_rng(B + 100 * q_bf16)
    ctx = np.asarray([1 + (97 * i + 1300 * (i == 0)) % 1500 // (1 + i % 3) for i in range(B)], np.int32)
    pool, cl, rl = build_mla(dev, oracle, rng, ctx, dC, dHR)
    wuk, wuv = (oracle.bf16_from_f32(rng.standard_normal((dC, H * Dh)).astype(np.float32) * 0.05) for _ in range(2))
    d_wuk, d_wuv = dev.upload(wuk), dev.upload(wuv)
    c, r = rng.standard_normal((B, dC)).astype(np.float32), rng.standard_normal((B, dHR)).astype(np.float32)
    qc, qr = rng.standard_normal((B, 1, H, Dh)).astype(np.float32), rng.standard_normal((B, 1, H, dHR)).astype(np.float32)
    if q_bf16:
        qc, qr = (oracle.f32_from_bf16(oracle.bf16_from_f32(a)) for a in (qc, qr))
    out = np.full(qc.shape, np.nan, np.float32)
    scale = float((Dh + dHR) ** -0.5)
    qs = [oracle.bf16_from_f32(a) for a in (qc, qr)] if q_bf16 else [qc, qr]
    pool.step(0, B, c, r, qs[0], out, H, Dh, scale, q_rope=qs[1], w_uk=d_wuk, w_uv=d_wuv)
    cb, rb = oracle.bf16_from_f32(c), oracle.bf16_from_f32(r)
    T = ctx + 1
    full_c = np.concatenate([np.concatenate([cl[i, :ctx[i]], cb[i:i + 1]]) for i in range(B)])
    full_r = np.concatenate([np.concatenate([rl[i, :ctx[i]], rb[i:i + 1]]) for i in range(B)])
    with oracle.exact_exp():
        ref = oracle.mla_attend(ragged_to_padded(full_c, T, (dC,)), ragged_to_padded(full_r, T, (dHR,)), T, qc, qr, wuk, wuv, scale,
                                absorbed=True)
    # outputs of one-row contexts are about one, of long ones smaller: the bound of the other short-context tests
    check_attention(out, ref, "step", max_tol=EDGE_MAX * max(1.0, float(np.abs(ref).max())), mean_tol=EDGE_MEAN)
    assert pool.status() == 0
    d_wuk.free(); d_wuv.free()
    pool.destroy()


@pytest.mark.parametrize("bf16", [False, True])
@pytest.mark.parametrize("n,P", [(2, 16), (7, 64), (8, 16), (9, 64), (70, 16), (2100, 64)])
def test_uniform_appends(dev, oracle, n, P, bf16):  # noqa: F811
    import relux_b200 as rb
    from relux_b200 import lib as L
    rng = np.random.default_rng(n + P + bf16)
    B, Hkv, D, dC, dHR = 3, 2, 128, 64, 16
    per = (2 * n + 5 + P - 1) // P
    for kind, wa, wb, kw in ((L.POOL_GQA, (Hkv, D), (Hkv, D), dict(num_kv_heads=Hkv, head_dim=D)),
                             (L.POOL_MLA, (dC,), (dHR,), dict(dC=dC, dHR=dHR))):
        pool = rb.Pool(dev, kind, 1, B * per, P, B, per, **kw)
        pool.set_tables(permuted_tables(rng, B, per))
        want = [[], []]
        for ids, rows in ((None, n), ([2, 0, 1], 5), (None, n)):   # the second call leaves the cursors inside a page
            a, b = (rng.standard_normal((B * rows,) + w).astype(np.float32) for w in (wa, wb))
            ab, bb = oracle.bf16_from_f32(a).reshape((B * rows,) + wa), oracle.bf16_from_f32(b).reshape((B * rows,) + wb)
            pool.append(0, ab if bf16 else a, bb if bf16 else b, B, seq_ids=ids, n_new=np.full(B, rows, np.int32))
            order = np.argsort(ids) if ids else np.arange(B)
            for k, x in enumerate((ab, bb)):
                want[k].append(x.reshape((B, rows) + x.shape[1:])[order])
        for s in range(B):
            total = 2 * n + 5
            assert pool.seq_len(0, s) == total
            got = pool.read_rows(0, s, 0, total)
            for k in range(2):
                assert np.array_equal(got[k].reshape(total, -1), np.concatenate([x[s] for x in want[k]]).reshape(total, -1))
        assert pool.status() == 0
        pool.destroy()
