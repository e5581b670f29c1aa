"""The device times a pool keeps of its calls."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RING = 8192   # times that are kept; a kernel clears the slot of the call after it


def test_a_call_that_fails_before_its_launch_takes_no_slot(oracle):
    """More calls than the ring holds, one that is refused when its projections are dealt out (more than 2^31 steps; nothing of
    it but the rounding of its input runs), then one more: its time is its own, not counted from a call 8193 ago."""
    import relux_b200 as rb
    from relux_b200 import lib as L
    dev = rb.Device(0)
    H, dC, dHR, D, big = 8, 64, 16, 64, 1 << 22
    pool = rb.Pool(dev, L.POOL_MLA, 1, 1, 64, 1, 1, dC=dC, dHR=dHR)
    pool.set_tables(np.zeros((1, 1), np.int32))
    rng = np.random.default_rng(0)
    shapes = dict(w_q=(D, D), w_qr=(D, H * dHR), w_dkv=(D, dC), w_kr=(D, dHR), w_uk=(dC, D), w_uv=(dC, D), w_o=(D, D))
    w = {k: dev.upload(oracle.bf16_from_f32(rng.standard_normal(s, dtype=np.float32))) for k, s in shapes.items()}
    x, out = dev.upload(np.ones((1, 1, D), np.float32)), dev.alloc(4 * D, L.DTYPE_F32)
    wide, wide_out = dev.alloc(4 * big, L.DTYPE_F32), dev.alloc(4 * big, L.DTYPE_F32)
    wide.zero()

    def call():
        pool.set_len(0, [0])
        pool.forward_cached(0, 1, x, out, w, D, H)

    for _ in range(RING + 50):
        call()
    pool.set_len(0, [0])
    with pytest.raises(L.ReluxCudaError) as e:
        pool.forward_cached(0, 1, wide, wide_out, w, big, H)
    assert e.value.code == L.ERR_UNSUPPORTED
    for _ in range(3):
        call()
        ms, n = pool.mean_projection_ms(1)
        assert n == 1 and 0 < ms < 5.0
    assert pool.status() == 0
    pool.destroy()
    for b in list(w.values()) + [x, out, wide, wide_out]:
        b.free()
    dev.close()
