"""Calls queued back to back with chained launches (each kernel may begin while the one before it still runs) and with plain
launches: the same bits, in the outputs and in the cache.  test_gpu_attention.py does the same for the latent decode step."""
import numpy as np
import pytest

from tests.helpers import permuted_tables

pytestmark = pytest.mark.gpu

DH, DC, DHR = 128, 512, 64

CASES = {   # tokens per sequence and call, heads (GQA: over two kv heads), bf16 results where the call offers them
    "gqa_step": dict(S=1, H=16), "gqa_verify": dict(S=3, H=16), "gqa_prompt": dict(S=150, H=16),
    "mla_verify": dict(S=3, H=32), "mla_prompt": dict(S=150, H=32),
    "gqa_layer": dict(S=1, H=16), "gqa_layer_rows": dict(S=3, H=16), "gqa_layer_prompt": dict(S=150, H=16),
    "mla_layer": dict(S=1, H=16), "mla_layer_rows": dict(S=3, H=16), "mla_layer_prompt": dict(S=150, H=16),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_chained_launches_give_the_bits_of_plain_ones(oracle, name):
    import relux_b200 as rb
    from relux_b200 import lib as L
    S, H = CASES[name]["S"], CASES[name]["H"]
    mla, layer, calls = name.startswith("mla"), "layer" in name, 3 if S > 100 else 8
    ctx = np.asarray([700, 64, 129, 0, 255, 320], np.int32)
    if S == 3:
        ctx[3] = 5
    B, Hkv, per, D, scale = len(ctx), 2, (700 + calls * S) // 64 + 2, H * DH, 0.07
    dev = rb.Device(0)
    rng = np.random.default_rng(len(name))
    held = []

    def up(shape, std=1.0):
        held.append(dev.upload(oracle.bf16_from_f32(rng.standard_normal(shape, dtype=np.float32) * np.float32(std))))
        return held[-1]

    wa, wb = ((DC,), (DHR,)) if mla else ((Hkv, DH), (Hkv, DH))
    rows = [rng.standard_normal((int(ctx.sum()),) + w, dtype=np.float32) for w in (wa, wb)]
    table = permuted_tables(rng, B, per)
    pools = []
    for k in range(2):
        kw = dict(dC=DC, dHR=DHR) if mla else dict(num_kv_heads=Hkv, head_dim=DH)
        p = rb.Pool(dev, L.POOL_MLA if mla else L.POOL_GQA, 1, B * per, 64, B, per, **kw)
        p.set_tables(table)
        p.append(0, rows[0], rows[1], B, n_new=ctx)
        pools.append(p)
    pools[1].tune(L.TUNE_CHAINED_LAUNCHES, 0)
    if layer:
        n = dict(w_q=D, w_qr=H * DHR, w_dkv=DC, w_kr=DHR, w_o=D) if mla else dict(w_q=D, w_k=Hkv * DH, w_v=Hkv * DH, w_o=D)
        w = {k: up((D, c), D ** -0.5) for k, c in n.items()}
    if mla:
        wuk, wuv = up((DC, D), 0.05), up((DC, D), 0.05)
        if layer:
            w.update(w_uk=wuk, w_uv=wuv)
    ins = []
    for _ in range(calls):
        if layer:
            x = dev.upload(rng.standard_normal((B, S, D), dtype=np.float32))
            held.append(x)
            ins.append(x)
        else:
            ins.append((up((B * S,) + wa), up((B * S,) + wb), up((B, S, H, DH)), up((B, S, H, DHR)) if mla else None))
    outs = [[dev.alloc(B * S * D * 4, L.DTYPE_F32) for _ in range(calls)] for _ in range(2)]
    for p, po in zip(pools, outs):
        for i in range(calls):
            if layer:
                p.forward_cached(0, B, ins[i], po[i], w, D, H, q_tokens=S)
                continue
            a, b, q, qr = ins[i]
            more = dict(q_rope=qr, w_uk=wuk, w_uv=wuv) if mla else {}
            if name == "gqa_step":
                p.step(0, B, a, b, q, po[i], H, DH, scale)
            elif S == 3:
                p.verify(0, B, q, po[i], a, b, H, DH, scale, S, **more)
                p.set_len(0, ctx + (i + 1))   # one row of each draft stays
            else:
                p.append(0, a, b, B, n_new=np.full(B, S, np.int32))
                p.decode(0, B, q, po[i], H, DH, scale, q_tokens=S, **more)
    dev.sync()
    for i in range(calls):
        x, y = (po[i].download((B, S, D), np.float32) for po in outs)
        assert np.isfinite(x).all() and np.array_equal(x, y), "call %d differs" % i
    for s in range(B):
        n = pools[0].seq_len(0, s)
        assert pools[1].seq_len(0, s) == n == ctx[s] + calls * (1 if S == 3 and not layer else S)
        m = min(n, calls * S)
        for x, y in zip(pools[0].read_rows(0, s, n - m, m), pools[1].read_rows(0, s, n - m, m)):
            assert np.array_equal(x, y)
    for p in pools:
        assert p.status() == 0
        p.destroy()
    for b in held + outs[0] + outs[1]:
        b.free()
    dev.close()
