"""Pipelined calls share one event a call among their buffers: steps, appends, decode calls and steps whose queries or outputs stay on the device, in
an order in which the buffers' turns drift apart, against the same calls one by one."""
import numpy as np
import pytest

from tests.test_gpu_attention import build_gqa, build_mla, dev  # noqa: F401

pytestmark = pytest.mark.gpu

ORDER = ["step", "append", "step", "decode", "decode", "step_q_dev", "append", "append", "step", "step_all_dev_but_rows", "decode", "step", "step_out_dev",
         "append", "step_q_dev", "decode", "step", "step"]


@pytest.mark.parametrize("kind", ["mla", "gqa"])
def test_calls_of_all_kinds_in_turn(dev, oracle, kind):  # noqa: F811
    from relux_b200 import lib as L
    ctx, B, D, S = [70, 300, 5], 3, 128, 1
    wa, wb, H = (512, 64, 32) if kind == "mla" else (8 * D, 8 * D, 32)
    pools = [(build_mla(dev, oracle, np.random.default_rng(5), ctx, 512, 64)[0] if kind == "mla" else build_gqa(dev, oracle, np.random.default_rng(5), ctx, 8, D)[0])
             for _ in range(2)]
    rng = np.random.default_rng(6)
    bf = lambda *s: oracle.bf16_from_f32(rng.standard_normal(s).astype(np.float32))  # noqa: E731
    more = {}
    if kind == "mla":
        more = dict(w_uk=dev.upload(bf(512, H * D)), w_uv=dev.upload(bf(512, H * D)))
    kw = dict(q_dtype=L.DTYPE_BF16, out_dtype=L.DTYPE_F32)
    held, got, want = [], [], []

    def pinned(a):
        h = dev.pinned(a.shape, a.dtype)
        h.array[...] = a
        held.append(h)
        return h.array
    for op in ORDER:
        rows = [bf(B, wa), bf(B, wb)]
        q, qr, out = bf(B, S, H, D), bf(B, S, H, 64), np.full((B, S, H, D), np.nan, np.float32)
        if op == "append":
            pools[0].append(0, *rows, B)
            pools[1].append(0, *(pinned(x) for x in rows), B, pipelined=True)
            continue
        args = lambda q_, o: (q_, o, H, D, 0.08)  # noqa: E731
        rope = lambda x: dict(q_rope=x) if kind == "mla" else {}  # noqa: E731
        if op == "decode":
            pools[0].decode(0, B, *args(q, out), **rope(qr), **more, **kw)
        else:
            pools[0].step(0, B, *rows, *args(q, out), **rope(qr), **more, **kw, kv_dtype=L.DTYPE_BF16)
        want.append(out.copy())
        q_dev, out_dev = op in ("step_q_dev", "step_all_dev_but_rows"), op in ("step_out_dev", "step_all_dev_but_rows")
        q2, qr2 = (dev.upload(x) if q_dev else pinned(x) for x in (q, qr))
        o2 = dev.upload(np.full_like(out, np.nan)) if out_dev else pinned(np.full_like(out, np.nan))
        if op == "decode":
            pools[1].decode(0, B, *args(q2, o2), **rope(qr2), **more, **kw, pipelined=True)
        else:
            pools[1].step(0, B, *(pinned(x) for x in rows), *args(q2, o2), **rope(qr2), **more, **kw, kv_dtype=L.DTYPE_BF16, pipelined=True)
        got.append(o2)
    dev.sync()
    for i, (a, b) in enumerate(zip(got, want)):
        a = a if isinstance(a, np.ndarray) else a.download(b.shape, np.float32)
        assert np.array_equal(a, b), i
    for s in range(B):
        n = pools[0].seq_len(0, s)
        assert n == pools[1].seq_len(0, s)
        for x, y in zip(pools[0].read_rows(0, s, 0, n), pools[1].read_rows(0, s, 0, n)):
            assert np.array_equal(x, y)
    assert pools[1].status() == 0
    for p in pools:
        p.destroy()


@pytest.mark.parametrize("rows", ["page_locked", "unaligned", "pageable", "one_of_each"])
def test_large_steps_over_short_sequences(dev, oracle, rows):  # noqa: F811
    """Steps whose copies outlast their kernels read page-locked new rows where they are, others are copied; a call's inputs are overwritten as soon as its
    output has landed, two calls are in flight, against ordinary steps."""
    from relux_b200 import lib as L
    B, H, D, steps = 64, 128, 128, 5
    ctx = [3 + (i * 37) % 150 for i in range(B)]
    pools = [build_mla(dev, oracle, np.random.default_rng(5), ctx, 512, 64)[0] for _ in range(2)]
    rng = np.random.default_rng(6)
    bf = lambda *s: oracle.bf16_from_f32(rng.standard_normal(s).astype(np.float32))  # noqa: E731
    more = dict(w_uk=dev.upload(bf(512, H * D)), w_uv=dev.upload(bf(512, H * D)), q_dtype=L.DTYPE_BF16, out_dtype=L.DTYPE_BF16)
    held = []

    def pinned(a, shift=0):
        h = dev.pinned((a.size + 4,), a.dtype)
        held.append(h)
        view = h.array[shift:shift + a.size].reshape(a.shape)
        view[...] = a
        return view

    def place(a, k):
        if rows == "pageable" or (rows == "one_of_each" and k):
            return a.copy()
        return pinned(a, 1 if rows == "unaligned" else 0)
    want, got, calls = [], [], []
    for i in range(steps):
        new = [rng.standard_normal((B, w)).astype(np.float32) for w in (512, 64)]
        q, qr, out = bf(B, 1, H, D), bf(B, 1, H, 64), np.zeros((B, 1, H, D), np.uint16)
        pools[0].step(0, B, *new, q, out, H, D, 0.08, q_rope=qr, **more)
        want.append(out)
        mine = [place(new[k], k) for k in range(2)] + [pinned(q), pinned(qr), pinned(np.full_like(out, 0x7fc0))]
        pools[1].step(0, B, mine[0], mine[1], mine[2], mine[4], H, D, 0.08, q_rope=mine[3], **more, pipelined=True)
        calls.append(mine)
        for k in range(2 if i == steps - 1 else 1):
            if i + k >= 1:
                pools[1].wait_output(1 - k)
                got.append(calls[i - 1 + k][4].copy())
                for a in calls[i - 1 + k][:4]:
                    a[...] = 3
    for i in range(steps):
        assert np.array_equal(got[i], want[i]), i
    dev.sync()
    for s in range(0, B, 7):
        for x, y in zip(*(p.read_rows(0, s, 0, ctx[s] + steps) for p in pools)):
            assert np.array_equal(x, y)
    assert pools[1].status() == 0
    for p in pools:
        p.destroy()
    for b in ("w_uk", "w_uv"):
        more[b].free()
