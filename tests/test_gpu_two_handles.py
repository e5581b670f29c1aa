"""Two device handles on one GPU."""
import numpy as np
import pytest

from tests.test_gpu_attention import build_mla

pytestmark = pytest.mark.gpu


def test_pools_of_different_widths_on_two_handles(oracle):
    """The shared memory of the latent kernels depends on dC, and the limit a kernel may use is one per GPU: a narrow pool's
    step on another handle in between must not take it away from a wide pool (dC 512, 128, 512)."""
    import relux_b200 as rb
    devs = [rb.Device(0), rb.Device(0)]
    H, Dh, dHR, scale = 16, 128, 64, 0.07
    ctx = [70, 200, 1]
    B = len(ctx)
    pools = []
    for k, dC in ((0, 512), (1, 128)):
        pools.append(build_mla(devs[k], oracle, np.random.default_rng(dC), ctx, dC, dHR, extra_pages=1)[0])
    rng = np.random.default_rng(3)
    bf = oracle.bf16_from_f32
    for turn, k in enumerate((0, 1, 0)):
        dC = (512, 128)[k]
        w = [devs[k].upload(bf(np.random.default_rng(dC + j).standard_normal((dC, H * Dh)).astype(np.float32) * 0.05)) for j in range(2)]
        a, b, q, qr = (rng.standard_normal(s).astype(np.float32) for s in ((B, dC), (B, dHR), (B, 1, H, Dh), (B, 1, H, dHR)))
        out = np.full(q.shape, np.nan, np.float32)
        pools[k].step(0, B, a, b, q, out, H, Dh, scale, q_rope=qr, w_uk=w[0], w_uv=w[1])
        again = np.full(q.shape, np.nan, np.float32)   # the cache as the step left it, by a call of its own
        pools[k].decode(0, B, q, again, H, Dh, scale, q_rope=qr, w_uk=w[0], w_uv=w[1])
        assert np.isfinite(out).all() and np.array_equal(out, again)
        assert [pools[k].seq_len(0, s) for s in range(B)] == [c + 1 + (turn == 2) for c in ctx]
        for x in w:
            x.free()
    for k in range(2):
        assert pools[k].status() == 0
        pools[k].destroy()
        devs[k].close()
