"""A step or a layer call that finds no memory for its partial results: nothing of it may stay behind on one side only."""
import numpy as np
import pytest

from tests.helpers import permuted_tables

pytestmark = pytest.mark.gpu

B, DH, DC, DHR, CTX = 16, 128, 512, 64, 2000


def _fill_memory(dev):
    """All of the device's free memory but what no block of 1 MB fits into."""
    held, size = [], 1 << 36
    while size >= 1 << 20:
        try:
            held.append(dev.alloc(size))
        except Exception:
            size >>= 1
    return held


def _world(dev, oracle, kind):
    """(pool, step(i)): a pool whose buffers have served a step over short sequences, and its i-th call."""
    import relux_b200 as rb
    from relux_b200 import lib as L
    mla = kind.startswith("mla")
    H, Hkv, per = (64 if mla else 32), (0 if mla else 2), CTX // 64 + 2
    kw = dict(dC=DC, dHR=DHR) if mla else dict(num_kv_heads=Hkv, head_dim=DH)
    pool = rb.Pool(dev, L.POOL_MLA if mla else L.POOL_GQA, 1, B * per, 64, B, per, **kw)
    rng = np.random.default_rng(5)
    pool.set_tables(permuted_tables(rng, B, per))
    wa, wb = ((DC,), (DHR,)) if mla else ((Hkv, DH), (Hkv, DH))
    bufs = []

    def up(shape, std=1.0):
        b = dev.upload(oracle.bf16_from_f32(rng.standard_normal(shape, dtype=np.float32) * np.float32(std)))
        bufs.append(b)
        return b

    ctx = rng.standard_normal((B * CTX,) + wa, dtype=np.float32), rng.standard_normal((B * CTX,) + wb, dtype=np.float32)
    pool.append(0, *ctx, B, n_new=np.full(B, CTX, np.int32))
    if kind.endswith(("step", "verify")):
        more = dict(w_uk=up((DC, H * DH), 0.05), w_uv=up((DC, H * DH), 0.05)) if mla else {}
        out = dev.alloc(B * H * DH * 4, L.DTYPE_F32)
        bufs.append(out)
        a, b, q, qr = up((4, B) + wa), up((4, B) + wb), up((4, B, 1, H, DH)), up((4, B, 1, H, DHR))

        def step(i):
            off = lambda x, n: x.ptr + 2 * i * B * n   # noqa: E731
            if kind == "gqa_verify":
                pool.verify(0, B, off(q, H * DH), out, off(a, int(np.prod(wa))), off(b, int(np.prod(wb))), H, DH, 0.07, 1, q_dtype=L.DTYPE_BF16,
                            kv_dtype=L.DTYPE_BF16)
                return out.download((B, H, DH), np.float32)
            if mla:
                more["q_rope"] = off(qr, H * DHR)
            pool.step(0, B, off(a, int(np.prod(wa))), off(b, int(np.prod(wb))), off(q, H * DH), out, H, DH, 0.07, q_dtype=L.DTYPE_BF16,
                      kv_dtype=L.DTYPE_BF16, **more)
            return out.download((B, H, DH), np.float32)
    else:
        D = H * DH
        n = dict(w_q=D, w_qr=H * DHR, w_dkv=DC, w_kr=DHR, w_o=D) if mla else dict(w_q=D, w_k=Hkv * DH, w_v=Hkv * DH, w_o=D)
        w = {k: up((D, c), D ** -0.5) for k, c in n.items()}
        if mla:
            w.update(w_uk=up((DC, D), 0.05), w_uv=up((DC, D), 0.05))
        x = rng.standard_normal((4, B, 1, D), dtype=np.float32)

        def step(i):
            out = np.empty((B, 1, D), np.float32)
            pool.forward_cached(0, B, x[i], out, w, D, H)
            return out
    # the buffers of a call, at lengths whose partial results are small
    pool.set_len(0, np.full(B, 40, np.int32))
    pool.append(0, ctx[0][:B], ctx[1][:B], B)   # what a failed call falls back on is loaded too
    step(0)
    pool.set_len(0, np.full(B, CTX, np.int32))

    def close():
        pool.destroy()
        for b in bufs:
            b.free()
    return pool, step, close


@pytest.mark.parametrize("kind", ["mla_step", "gqa_step", "gqa_verify", "mla_layer", "gqa_layer"])
def test_call_without_memory(oracle, kind):
    import relux_b200 as rb
    from relux_b200 import lib as L
    dev = rb.Device(0)
    (pool, step, close), (other, step2, close2) = _world(dev, oracle, kind), _world(dev, oracle, kind)
    held = _fill_memory(dev)
    try:
        with pytest.raises(L.ReluxCudaError) as e:
            step(1)
        assert e.value.code == L.ERR_OUT_OF_MEMORY
    finally:
        for b in held:
            b.free()
    # a GQA step keeps its rows when its attention is refused, as the two calls one after the other do; the other calls leave
    # the lengths as they were.  No later call meets the error again.
    if kind == "gqa_step":
        step2(1)
    n = [other.seq_len(0, s) for s in range(B)]
    assert [pool.seq_len(0, s) for s in range(B)] == n
    for i in (2, 3):   # the device's lengths: where these rows land, and what they see
        assert np.array_equal(step(i), step2(i))
    for s in (0, B - 1):
        for x, y in zip(pool.read_rows(0, s, CTX - 2, n[s] + 3 - CTX), other.read_rows(0, s, CTX - 2, n[s] + 3 - CTX)):
            assert np.array_equal(x, y)
    assert pool.status() == 0
    close(); close2()
    dev.close()
