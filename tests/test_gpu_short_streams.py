"""GQA steps over many short streams: every range holds many pieces, so the states' two buffers, the query buffers and the new rows
of all warps take turns many times; and the query-row counts on either side of what two buffers hold."""
import numpy as np
import pytest

from tests.helpers import check_attention
from tests.test_gpu_attention import build_gqa, dev  # noqa: F401
from tests.test_gpu_randomized import MAX_ABS, MEAN_ABS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,Hkv,S", [(8, 8, 1), (16, 2, 1), (18, 2, 1), (32, 8, 2), (24, 8, 3), (32, 8, 4), (20, 4, 4), (64, 2, 1)])   # 1, 8, 9, 8, 9, 16, 20, 32 rows
@pytest.mark.parametrize("ctx", [[1 + i % 3 for i in range(150)], [1 + 13 * (i % 10) for i in range(150)], [63 + i % 3 for i in range(20)] + [2000, 5]],
                         ids=["one_page", "one_or_two_pages", "and_a_long_one"])
def test_step_over_short_streams(dev, oracle, H, Hkv, S, ctx):  # noqa: F811
    from relux_b200 import lib as L
    rng = np.random.default_rng(H + 7 * S + len(ctx))
    ctx = np.asarray(ctx, np.int32)
    B, D, scale = len(ctx), 128, 128 ** -0.5
    pool, _, _ = build_gqa(dev, oracle, rng, ctx, Hkv, D)
    k, v = (rng.standard_normal((B * S, Hkv, D)).astype(np.float32) for _ in range(2))
    q = rng.standard_normal((B, S, H, D)).astype(np.float32)
    out, ref = np.full(q.shape, np.nan, np.float32), np.empty(q.shape, np.float32)
    if S == 1:
        pool.step(0, B, k, v, q, out, H, D, scale)
    else:
        pool.verify(0, B, q, out, k, v, H, D, scale, S)
    extra = 0 if S == 1 else S
    pool.decode(0, B, q, ref, H, D, scale, q_tokens=S, extra_tokens=extra, mode=L.ATTN_REFERENCE)
    # the bounds of the randomised tests: REFERENCE mode keeps the reference's approximate exponential
    check_attention(out, ref, "short streams", max_tol=MAX_ABS, mean_tol=MEAN_ABS)
    last = B - 1
    rk, rv = pool.read_rows(0, last, int(ctx[last]), S) if S == 1 else (None, None)
    if S == 1:
        assert np.array_equal(rk, oracle.bf16_from_f32(k).reshape(B, S, Hkv, D)[last])
        assert np.array_equal(rv, oracle.bf16_from_f32(v).reshape(B, S, Hkv, D)[last])
    assert pool.status() == 0
    pool.destroy()
