"""Latent decode calls without rows to append: the partition's builder works beside the absorb of the queries, and what it writes is what the call
before it reads.  Calls of different plans follow one another unsynchronised, each as the call alone."""
import numpy as np
import pytest

from tests.test_gpu_attention import build_mla, dev  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,H,chained", [(1, 128, 1), (2, 32, 1), (3, 128, 0), (4, 16, 1)])
def test_calls_in_a_row_are_the_calls_alone(dev, oracle, S, H, chained):  # noqa: F811
    from relux_b200 import lib as L
    Dh, dC, dHR = 128, 512, 64
    rng = np.random.default_rng(H + S)
    ctx = [70, 1500, 300, 64, 129] + [200] * 40
    pool = build_mla(dev, oracle, rng, ctx, dC, dHR)[0]
    pool.tune(L.TUNE_CHAINED_LAUNCHES, chained)
    w = [dev.upload(oracle.bf16_from_f32(rng.standard_normal((dC, H * Dh)).astype(np.float32) * 0.02)) for _ in range(2)]
    calls = []   # sequences, queries, output: one sequence, a few, more rows than one tile of the absorb, all of them
    for ids in ([1], [4, 0, 1], list(range(5, 40)), list(range(45)), [2], [3, 1, 44]):
        n = len(ids)
        q, qr = (oracle.bf16_from_f32(rng.standard_normal((n, S, H, x)).astype(np.float32)) for x in (Dh, dHR))
        calls.append((np.asarray(ids, np.int32), dev.upload(q), dev.upload(qr), [dev.upload(np.full((n, S, H, Dh), np.nan, np.float32)) for _ in range(2)]))

    def call(c, out):
        pool.decode(0, len(c[0]), c[1], out, H, Dh, 192 ** -0.5, q_rope=c[2], w_uk=w[0], w_uv=w[1], q_tokens=S, seq_ids=c[0], q_dtype=L.DTYPE_BF16,
                    out_dtype=L.DTYPE_F32)
    for c in calls:
        call(c, c[3][0])
        dev.sync()
    for _ in range(3):
        for c in calls:
            call(c, c[3][1])
    dev.sync()
    for c in calls:
        alone, row = (o.download((len(c[0]), S, H, Dh), np.float32) for o in c[3])
        assert np.isfinite(alone).all() and np.array_equal(alone, row)
    assert pool.status() == 0
    pool.destroy()
    for b in w + [x for c in calls for x in (c[1], c[2], *c[3])]:
        b.free()
