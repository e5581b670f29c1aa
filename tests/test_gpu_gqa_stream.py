"""The one-launch GQA step (append + attention + merge of the splits): decode and verify steps at the lengths, group sizes
and batch sizes where its page ranges, its new rows and its two ways of passing the sequences can go wrong."""
import numpy as np
import pytest

from tests.helpers import check_attention, ragged_to_padded
from tests.test_gpu_attention import EDGE_MAX, EDGE_MEAN, build_gqa, dev  # noqa: F401

pytestmark = pytest.mark.gpu

CASES = {
    # one sequence, one row cached; page boundaries; a sequence cut into one range per SM; more streams than ranges
    "one_row": dict(ctx=[1], H=8, Hkv=8),
    "page_edges": dict(ctx=[63, 64, 65, 127, 128, 1], H=32, Hkv=8),
    "long_and_short": dict(ctx=[9000, 5, 64, 700], H=32, Hkv=2),
    "rows_16": dict(ctx=[300, 190, 64], H=32, Hkv=2),
    "rows_17_to_32": dict(ctx=[2100, 63], H=64, Hkv=2),
    "group_of_5": dict(ctx=[130, 61], H=10, Hkv=2),
    # the sequences as kernel arguments (32, 256) and through a device copy
    "seqs_32": dict(ctx=[1 + 7 * i for i in range(32)], H=16, Hkv=2),
    "seqs_33": dict(ctx=[1 + 7 * i for i in range(33)], H=16, Hkv=2),
    "seqs_257": dict(ctx=[1 + i % 130 for i in range(257)], H=4, Hkv=2),
}


@pytest.mark.parametrize("S", [1, 4])
@pytest.mark.parametrize("name", sorted(CASES))
def test_one_launch_step(dev, oracle, name, S):  # noqa: F811
    from relux_b200 import lib as L
    c = CASES[name]
    H, Hkv, D = c["H"], c["Hkv"], 128
    if S > 1 and H // Hkv * S > 32:
        S = 2 if H // Hkv * 2 <= 32 else 1
    rng = np.random.default_rng(len(name) + 10 * S)
    ctx = np.asarray(c["ctx"], np.int32)
    B, scale = len(ctx), 128 ** -0.5
    pool, Kl, Vl = build_gqa(dev, oracle, rng, ctx, Hkv, D)
    k, v = (rng.standard_normal((B * S, Hkv, D)).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((B, S, H, D)).astype(np.float32)
    out = np.full(q.shape, np.nan, np.float32)
    n0 = dev.launch_count()
    if S == 1:
        pool.step(0, B, k, v, q, out, H, D, scale)
    else:
        pool.verify(0, B, q, out, k, v, H, D, scale, S)
    assert dev.launch_count() - n0 == 1
    assert [pool.seq_len(0, s) for s in range(B)] == [int(x) + (S == 1) for x in ctx]
    kb, vb = oracle.bf16_from_f32(k).reshape(B, S, Hkv, D), oracle.bf16_from_f32(v).reshape(B, S, Hkv, D)
    for s in {0, B // 2, B - 1}:   # the new rows, and the cached ones around them, bit for bit
        rk, rv = pool.read_rows(0, s, 0, int(ctx[s]) + S)
        assert np.array_equal(rk[:ctx[s]], Kl[s, :ctx[s]]) and np.array_equal(rk[ctx[s]:], kb[s])
        assert np.array_equal(rv[:ctx[s]], Vl[s, :ctx[s]]) and np.array_equal(rv[ctx[s]:], vb[s])
    full_k = np.concatenate([np.concatenate([Kl[i, :ctx[i]], kb[i]]) for i in range(B)])
    full_v = np.concatenate([np.concatenate([Vl[i, :ctx[i]], vb[i]]) for i in range(B)])
    T = ctx + S
    with oracle.exact_exp():
        ref = oracle.gqa_attend(ragged_to_padded(full_k, T, (Hkv, D)), ragged_to_padded(full_v, T, (Hkv, D)), T, q, scale, causal=True)
    check_attention(out, ref, "step", max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    # bf16 output and bf16 rows from device memory, twice: the counters are armed again, and the bits repeat
    if S > 1:
        d_q, d_k, d_v = (dev.upload(oracle.bf16_from_f32(a)) for a in (q, k, v))
        d_out = dev.alloc(q.size * 2, L.DTYPE_BF16)
        got = []
        for _ in range(2):
            pool.verify(0, B, d_q, d_out, d_k, d_v, H, D, scale, S)
            got.append(d_out.download(q.shape, np.uint16))
        assert np.array_equal(got[0], got[1])
        # the same kernel on the same bf16 queries: the bf16 output is the rounded float32 one
        assert np.array_equal(got[0], oracle.bf16_from_f32(out))
        for b in (d_q, d_k, d_v, d_out):
            b.free()
    assert pool.status() == 0
    pool.destroy()


def test_step_with_uneven_new_rows_and_named_sequences(dev, oracle):  # noqa: F811
    """0, 1 and 70 new rows (over a page boundary), sequences named out of order, head-major rows for one sequence."""
    rng = np.random.default_rng(5)
    H, Hkv, D, ctx = 16, 4, 128, [100, 60, 64, 3]
    pool, Kl, Vl = build_gqa(dev, oracle, rng, ctx, Hkv, D, extra_pages=2)
    ids, n_new = [2, 0, 1], [1, 70, 0]
    k, v = (rng.standard_normal((71, Hkv, D)).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((3, 1, H, D)).astype(np.float32)
    out = np.empty_like(q)
    pool.step(0, 3, k, v, q, out, H, D, 128 ** -0.5, seq_ids=ids, n_new=n_new)
    kb, vb = oracle.bf16_from_f32(k), oracle.bf16_from_f32(v)
    rows = [(kb[:1], vb[:1]), (kb[1:], vb[1:]), (kb[:0], vb[:0])]
    T = np.asarray([ctx[s] + n for s, n in zip(ids, n_new)], np.int32)
    fk = np.concatenate([np.concatenate([Kl[s, :ctx[s]], r[0]]) for s, r in zip(ids, rows)])
    fv = np.concatenate([np.concatenate([Vl[s, :ctx[s]], r[1]]) for s, r in zip(ids, rows)])
    with oracle.exact_exp():
        ref = oracle.gqa_attend(ragged_to_padded(fk, T, (Hkv, D)), ragged_to_padded(fv, T, (Hkv, D)), T, q, 128 ** -0.5, causal=True)
    check_attention(out, ref, "step", max_tol=EDGE_MAX, mean_tol=EDGE_MEAN)
    assert [pool.seq_len(0, s) for s in range(4)] == [170, 60, 65, 3]
    rk, _ = pool.read_rows(0, 0, 0, 170)
    assert np.array_equal(rk[100:], kb[1:])
    # an attention call that is refused leaves the rows appended, as the two calls one after the other do
    from relux_b200 import lib as L
    with pytest.raises(L.ReluxCudaError):
        pool.step(0, 1, k[:1], v[:1], q[:1], out[:1], H, D, -1.0, seq_ids=[3])
    assert pool.seq_len(0, 3) == 4
    assert pool.status() == 0
    pool.destroy()
