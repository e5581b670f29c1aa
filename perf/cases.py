"""The work a user of this library has it do: decode steps, speculative verify, prompts, whole layer steps and token selection,
each through the package's own calls, over the range of sizes of the repository's benchmark, tests and example models.

A case is a dict of plain values.  `kind` names the call:

  token         one token of one sequence through the reference-style cache object, host float32 arrays in and out
  gqa_step      one decode step of a batch (append + attention), grouped-query cache
  gqa_verify    a speculative verify step (draft rows past the cursor, causal attention, commit of the accepted prefix)
  mla_step      one decode step of a batch, latent cache
  gqa_prompt    a prompt (or the next chunk of one) into a grouped-query cache
  mla_prompt    the same into a latent cache
  gqa_layer     a whole attention layer step (projections, rotation, append, attention, output projection)
  mla_layer     the same for a latent-cache layer
  select        token selection: acceptance of draft tokens, or (k = 0) sampling one token per row

Decode steps append a row per sequence and pass; after HORIZON tokens a sequence starts again at its first length, as a slot
of a serving program does when its request has ended."""
import random

import numpy as np
import torch

import relux_b200 as rb
from relux_b200 import lib as L

PAGE = 64
HORIZON = 64
DH, DC, DHR = 128, 512, 64      # head width, latent width and rotary width of the latent-attention models
_DEV = []


def listed():
    return [
        # one user, one sequence, the reference's cache object called per token from host code: the smallest call there is
        dict(name="token_gqa_ctx700", kind="token", ctx=700, H=32, Hkv=8),
        # a few interactive sequences on the latent cache, short and uneven: launches and latency count
        dict(name="mla_step_b3_ctx1500", kind="mla_step", B=3, ctx=1500, H=128, ragged=True, io="device"),
        # the standalone latent decode of the benchmark: 64 sequences, 4096 cached tokens
        dict(name="mla_step_b64_ctx4k", kind="mla_step", B=64, ctx=4096, H=128, ragged=False, io="device"),
        # one GPU's share of the long-context batch: 16 sequences of 1k to 32k tokens
        dict(name="mla_step_b16_ragged_32k", kind="mla_step", B=16, ctx=32768, H=128, ragged=True, io="device"),
        # the headline workload end to end: inputs from page-locked host memory, outputs back to it, two steps in flight
        dict(name="mla_step_b64_ctx32k_e2e", kind="mla_step", B=64, ctx=32768, H=128, ragged=False, io="pipelined"),
        # ordinary serving of a grouped-query model: 32 sequences of uneven length
        dict(name="gqa_step_b32_ragged_3k", kind="gqa_step", B=32, ctx=3001, H=32, Hkv=8, ragged=True, io="device"),
        # speculative decoding at full batch: 128 sequences, 8192 tokens, four draft tokens
        dict(name="gqa_verify_b128_ctx8k", kind="gqa_verify", B=128, ctx=8192, H=32, Hkv=8, S=4),
        # prompts of a batch of new requests, grouped-query cache
        dict(name="gqa_prompt_b8_2k", kind="gqa_prompt", B=8, S=2048, cached=0, H=32, Hkv=8),
        # prompts on the latent cache, a length that fills no tile
        dict(name="mla_prompt_b4_1000", kind="mla_prompt", B=4, S=1000, cached=0, H=128),
        # a whole latent-attention layer at a small batch: the weights are streamed once per step
        dict(name="mla_layer_b16_ctx4k", kind="mla_layer", B=16, ctx=4096, H=128),
        # a whole grouped-query layer, one token for each of 24 sequences
        dict(name="gqa_layer_b24_ctx2k", kind="gqa_layer", B=24, ctx=2048, H=32, Hkv=8),
        # acceptance of four draft tokens for 64 sequences over a large vocabulary, with the usual filters
        dict(name="select_b64_k4_v128k", kind="select", B=64, k=4, V=131072, temperature=0.8, top_k=50, top_p=0.95),
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _draw(rng):
    kind = rng.choice(["token", "gqa_step", "gqa_step", "gqa_verify", "mla_step", "mla_step", "mla_step", "gqa_prompt", "mla_prompt",
                       "gqa_layer", "mla_layer", "select"])
    H, Hkv = rng.choice([(32, 8), (32, 8), (16, 8), (64, 8), (32, 4)])
    if kind == "token":
        return dict(kind=kind, ctx=_log(rng, 100, 8000), H=32, Hkv=8)
    if kind == "gqa_step":
        return dict(kind=kind, B=_log(rng, 1, 128), ctx=_log(rng, 200, 16384), H=H, Hkv=Hkv, ragged=rng.random() < 0.5,
                    io=rng.choice(["device", "device", "host"]))
    if kind == "gqa_verify":
        return dict(kind=kind, B=_log(rng, 1, 128), ctx=_log(rng, 200, 8192), H=H, Hkv=8, S=rng.choice([2, 3, 4]))
    if kind == "mla_step":
        return dict(kind=kind, B=_log(rng, 1, 64), ctx=_log(rng, 200, 32768), H=rng.choice([128, 128, 64, 32]), ragged=rng.random() < 0.5,
                    io=rng.choice(["device", "device", "pipelined"]))
    if kind == "gqa_prompt":
        return dict(kind=kind, B=_log(rng, 1, 8), S=_log(rng, 20, 8192), cached=rng.choice([0, 0, _log(rng, 60, 2000)]), H=32, Hkv=8)
    if kind == "mla_prompt":
        return dict(kind=kind, B=_log(rng, 1, 4), S=_log(rng, 20, 2048), cached=rng.choice([0, 0, _log(rng, 60, 2000)]), H=128)
    if kind == "gqa_layer":
        return dict(kind=kind, B=_log(rng, 1, 128), ctx=_log(rng, 200, 8192), H=32, Hkv=8)
    if kind == "mla_layer":
        return dict(kind=kind, B=_log(rng, 1, 64), ctx=_log(rng, 200, 8192), H=rng.choice([128, 32]))
    k = rng.choice([0, 0, 2, 4, 5])
    return dict(kind=kind, B=_log(rng, 1, 64), k=k, V=rng.choice([32000, 50257, 131072, _log(rng, 8000, 131072)]), temperature=0.8,
                top_k=rng.choice([0, 50]), top_p=rng.choice([1.0, 0.95]))


def draw(rng):
    """One more case of the ranges above, never more work than the largest listed one."""
    cost = lambda c: max(work(c)["bytes"], work(c)["flops"] / 50)   # noqa: E731
    most = max(cost(c) for c in listed())
    while True:
        c = _draw(rng)
        if cost(c) <= most:
            return c


# --- sizes -----------------------------------------------------------------------------------------------------------------

def _lens(case):
    """First lengths of the sequences: `ctx` each, or (ragged) uniform down to 1/32 of it, the same for every seed."""
    B, ctx = case["B"], case["ctx"]
    if not case.get("ragged"):
        return np.full(B, ctx, np.int64)
    r = random.Random(11)
    return np.asarray([r.randint(max(1, ctx // 32), ctx) for _ in range(B)], np.int64)


def work(case):
    k = case["kind"]
    if k == "token":
        rows, H, Hkv = case["ctx"] + HORIZON / 2, case["H"], case["Hkv"]
        return dict(bytes=rows * Hkv * DH * 4 + (2 * H + 2 * Hkv) * DH * 4, flops=4.0 * rows * H * DH)
    if k in ("gqa_step", "gqa_verify", "gqa_layer"):
        B, H, Hkv, S = case["B"], case["H"], case["Hkv"], case.get("S", 1)
        rows = float(_lens(case).sum()) + B * HORIZON / 2 + (B * S if k == "gqa_verify" else 0)
        nbytes = rows * Hkv * DH * 4 + B * S * (H * 6 + Hkv * 4) * DH
        flops = 4.0 * S * rows * H * DH
        if k == "gqa_layer":
            D = H * DH
            nw = D * (2 * H + 2 * Hkv) * DH
            nbytes, flops = rows * Hkv * DH * 4 + nw * 2 + B * D * 8, flops + 2.0 * B * nw
        return dict(bytes=nbytes, flops=flops)
    if k in ("mla_step", "mla_layer"):
        B, H = case["B"], case["H"]
        rows = float(_lens(case).sum()) + B * HORIZON / 2
        up = 2 * DC * H * DH
        nbytes = rows * (DC + DHR) * 2 + up * 2
        flops = 2.0 * H * rows * (2 * DC + DHR) + 2.0 * B * up
        if k == "mla_step":
            return dict(bytes=nbytes + B * (H * (DH * (4 if case["io"] == "pipelined" else 6) + DHR * 2) + (DC + DHR) * 2), flops=flops)
        D = H * DH
        nw = D * (2 * H * DH + H * DHR + DC + DHR)
        return dict(bytes=nbytes + nw * 2 + B * D * 8, flops=flops + 2.0 * B * nw)
    if k in ("gqa_prompt", "mla_prompt"):
        B, S, c, H = case["B"], case["S"], case["cached"], case["H"]
        scores = B * (S * c + S * (S + 1) / 2.0) * H
        if k == "gqa_prompt":
            Hkv = case["Hkv"]
            return dict(bytes=B * (c * Hkv * DH * 4 + S * Hkv * DH * 8 + S * H * DH * 6), flops=scores * 4 * DH)
        return dict(bytes=B * (c * (DC + DHR) * 2 + S * (DC + DHR) * 4 + S * H * (DH * 6 + DHR * 2)) + 4 * DC * H * DH,
                    flops=scores * 2 * (2 * DH + DHR) + B * (S + c) * 2.0 * DC * 2 * H * DH)
    B, kk, V = case["B"], case["k"], case["V"]
    rows = B * (2 * kk + 1)
    return dict(bytes=rows * V * 4.0, flops=rows * V * 4.0)


def tolerance(case):
    """Attention and projections take bf16 operands and sum in float32: probabilities and products rounded to 8 bits.  Selection
    returns token ids: equal but for a draw that falls within rounding distance of a boundary."""
    return dict(rel=0.0, differ=0.01) if case["kind"] == "select" else dict(rel=1e-2)


# --- inputs ----------------------------------------------------------------------------------------------------------------

def _device():
    if not _DEV:
        _DEV.append(rb.Device(torch.cuda.current_device()))
    return _DEV[0]


class _State:
    """What a program holds between calls; the pool, the cache and the buffers go back when it does."""

    def __init__(self, case):
        self.case, self.dev, self.pool, self.cache, self.held = case, _device(), None, None, []
        self.done = 0

    def __del__(self):
        try:
            self.dev.sync()
            for h in self.held:
                h.free()
            if self.cache is not None:
                self.cache.close()
            elif self.pool is not None:
                self.pool.destroy()
        except Exception:
            pass


class _Rand:
    def __init__(self, seed):
        self.g = torch.Generator("cuda").manual_seed(seed)

    def f32(self, *shape):
        return torch.randn(shape, generator=self.g, device="cuda", dtype=torch.float32)

    def bf16(self, *shape, std=1.0):
        return torch.randn(shape, generator=self.g, device="cuda", dtype=torch.bfloat16).mul_(std)


def _pool(st, kind, B, max_len, seed, **kw):
    """A pool with a random page table and B sequences of up to max_len tokens."""
    per = (max_len + PAGE - 1) // PAGE
    st.pool = rb.Pool(st.dev, kind, 1, B * per, PAGE, B, per, **kw)
    st.pool.set_tables(np.random.default_rng(seed).permutation(B * per).astype(np.int32).reshape(B, per))


def _fill(st, R, lens, wa, wb):
    """Caches lens[i] random rows of widths wa and wb for every sequence, block by block from device memory."""
    B, top = len(lens), int(max(lens))
    blk = max(1, min(top, 2048, (1 << 27) // max(1, B * (wa + wb))))
    for off in range(0, top, blk):
        n = np.clip(lens - off, 0, blk).astype(np.int32)
        rows = int(n.sum())
        a, b = R.bf16(rows, wa), R.bf16(rows, wb)
        torch.cuda.synchronize()
        st.pool.append(0, a.data_ptr(), b.data_ptr(), B, n_new=n, dtype=L.DTYPE_BF16)
        st.dev.sync()


def _pinned(t):
    """(array, tensor) over the same page-locked host memory, holding the values of t; a bf16 array is its bit patterns."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return (h.view(torch.int16).numpy().view(np.uint16) if t.dtype == torch.bfloat16 else h.numpy()), h


def prepare(case, seed):
    st, R, k = _State(case), _Rand(seed), case["kind"]
    if k == "token":
        H, Hkv, ctx = case["H"], case["Hkv"], case["ctx"]
        st.cache = rb.KVCache(st.dev, 1, ctx + HORIZON, Hkv, DH)
        st.cache.Append(0, R.f32(1, Hkv, ctx, DH).cpu().numpy(), R.f32(1, Hkv, ctx, DH).cpu().numpy())
        st.q, st.k, st.v = R.f32(1, H, 1, DH).cpu().numpy(), R.f32(1, Hkv, 1, DH).cpu().numpy(), R.f32(1, Hkv, 1, DH).cpu().numpy()
    elif k in ("gqa_step", "gqa_verify", "gqa_layer"):
        B, H, Hkv, S = case["B"], case["H"], case["Hkv"], case.get("S", 1)
        st.lens = _lens(case).astype(np.int32)
        _pool(st, L.POOL_GQA, B, int(st.lens.max()) + HORIZON + 2 * S, seed, num_kv_heads=Hkv, head_dim=DH)
        _fill(st, R, st.lens, Hkv * DH, Hkv * DH)
        if k == "gqa_layer":
            D = H * DH
            st.w = {n: R.bf16(D, c, std=D ** -0.5) for n, c in (("w_q", D), ("w_k", Hkv * DH), ("w_v", Hkv * DH), ("w_o", D))}
            st.x = st.dev.upload(R.f32(B, 1, D).cpu().numpy())
            st.held.append(st.x)
            st.out = torch.empty(B, 1, D, device="cuda")
        else:
            q, a, b = R.bf16(B, S, H, DH), R.bf16(B * S, Hkv, DH), R.bf16(B * S, Hkv, DH)
            if case.get("io") == "host":      # a host program with float32 activations in ordinary memory
                st.q, st.a, st.b = (t.float().cpu().numpy() for t in (q, a, b))
                st.out = np.zeros((B, S, H, DH), np.float32)
            else:
                st.q, st.a, st.b, st.out = q, a, b, torch.empty(B, S, H, DH, device="cuda")
        if k == "gqa_verify":                 # accepted prefixes of the steps to come, until a sequence starts again
            acc = np.random.default_rng(seed).integers(1, S + 1, (HORIZON // S, B))
            st.plan = [np.ascontiguousarray(x) for x in (st.lens + np.cumsum(acc, axis=0)).astype(np.int32)[:-1]] + [st.lens]
    elif k in ("mla_step", "mla_layer"):
        B, H = case["B"], case["H"]
        st.lens = _lens(case).astype(np.int32)
        _pool(st, L.POOL_MLA, B, int(st.lens.max()) + HORIZON, seed, dC=DC, dHR=DHR)
        _fill(st, R, st.lens, DC, DHR)
        st.wuk, st.wuv = R.bf16(DC, H * DH, std=0.02), R.bf16(DC, H * DH, std=0.02)
        if k == "mla_layer":
            D = H * DH
            st.w = {n: R.bf16(D, c, std=D ** -0.5) for n, c in (("w_q", D), ("w_qr", H * DHR), ("w_dkv", DC), ("w_kr", DHR), ("w_o", D))}
            st.w.update(w_uk=st.wuk, w_uv=st.wuv)
            st.x = st.dev.upload(R.f32(B, 1, D).cpu().numpy())
            st.held.append(st.x)
            st.out = torch.empty(B, 1, D, device="cuda")
        else:
            q, qr, a, b = R.bf16(B, 1, H, DH), R.bf16(B, 1, H, DHR), R.bf16(B, DC), R.bf16(B, DHR)
            if case["io"] == "pipelined":     # bf16 queries, float32 new rows, page-locked; two outputs in turn
                st.q, st.qr, st.a, st.b = (_pinned(t)[0] for t in (q, qr, a.float(), b.float()))
                st.outs, st.views = zip(*(_pinned(torch.zeros_like(q)) for _ in range(2)))
            else:
                st.q, st.qr, st.a, st.b, st.out = q, qr, a, b, torch.empty(B, 1, H, DH, device="cuda")
    elif k in ("gqa_prompt", "mla_prompt"):
        B, S, c, H = case["B"], case["S"], case["cached"], case["H"]
        st.lens, st.n_new = np.full(B, c, np.int32), np.full(B, S, np.int32)
        wa, wb = (case["Hkv"] * DH,) * 2 if k == "gqa_prompt" else (DC, DHR)
        kw = dict(num_kv_heads=case["Hkv"], head_dim=DH) if k == "gqa_prompt" else dict(dC=DC, dHR=DHR)
        _pool(st, L.POOL_GQA if k == "gqa_prompt" else L.POOL_MLA, B, c + S, seed, **kw)
        if c:
            _fill(st, R, st.lens, wa, wb)
        st.a, st.b, st.q = R.bf16(B * S, wa), R.bf16(B * S, wb), R.bf16(B, S, H, DH)
        st.out = torch.empty(B, S, H, DH, device="cuda")
        if k == "mla_prompt":
            st.qr, st.wuk, st.wuv = R.bf16(B, S, H, DHR), R.bf16(DC, H * DH, std=0.02), R.bf16(DC, H * DH, std=0.02)
    else:
        # logits of a verify pass: the target follows the draft up to noise, the draft token is the draft's best
        B, kk, V = case["B"], case["k"], case["V"]
        st.pool = rb.Pool(st.dev, L.POOL_MLA, 1, 2, PAGE, 1, 2, dC=64, dHR=16)
        st.draws = torch.rand((B, kk + 1), generator=R.g, device="cuda")
        st.target = torch.empty(B, kk + 1, V, device="cuda")
        if kk:
            st.draft = R.f32(B, kk, V).mul_(2.5)
            st.target[:, :kk] = st.draft + 0.6 * R.f32(B, kk, V)
            st.tokens = st.draft.argmax(dim=2).to(torch.int32).contiguous()
        st.target[:, kk] = 2.5 * R.f32(B, V)
    torch.cuda.synchronize()
    st.dev.sync()
    return st


# --- one pass --------------------------------------------------------------------------------------------------------------

def _restart(st, pool, seq_ids=None):
    st.done += 1
    if st.done % HORIZON == 0:
        pool.set_len(0, st.lens if seq_ids is None else [st.case["ctx"]], seq_ids)


def run(st):
    c, k = st.case, st.case["kind"]
    if k == "token":
        st.cache.Append(0, st.k, st.v)
        out = st.cache.attend(0, st.q, DH ** -0.5)
        _restart(st, st.cache.pool, [st.cache.seq])
        return out
    if k == "gqa_step":
        host = c["io"] == "host"
        p = (lambda t: t) if host else (lambda t: t.data_ptr())
        dt = {} if host else dict(q_dtype=L.DTYPE_BF16, out_dtype=L.DTYPE_F32, kv_dtype=L.DTYPE_BF16)
        st.pool.step(0, c["B"], p(st.a), p(st.b), p(st.q), p(st.out), c["H"], DH, DH ** -0.5, **dt)
        _restart(st, st.pool)
        return st.out
    if k == "gqa_verify":
        st.pool.verify(0, c["B"], st.q.data_ptr(), st.out.data_ptr(), st.a.data_ptr(), st.b.data_ptr(), c["H"], DH, DH ** -0.5, c["S"],
                       q_dtype=L.DTYPE_BF16, out_dtype=L.DTYPE_F32, kv_dtype=L.DTYPE_BF16)
        st.pool.set_len(0, st.plan[st.done % len(st.plan)])
        st.done += 1
        return st.out
    if k == "mla_step":
        scale = (DH + DHR) ** -0.5
        if c["io"] == "pipelined":
            i = st.done
            st.pool.step(0, c["B"], st.a, st.b, st.q, st.outs[i % 2], c["H"], DH, scale, q_rope=st.qr, w_uk=st.wuk.data_ptr(),
                         w_uv=st.wuv.data_ptr(), pipelined=True)
            if i >= 1:
                st.pool.wait_output(1)
            _restart(st, st.pool)
            return st.views[i % 2]
        st.pool.step(0, c["B"], st.a.data_ptr(), st.b.data_ptr(), st.q.data_ptr(), st.out.data_ptr(), c["H"], DH, scale,
                     q_rope=st.qr.data_ptr(), w_uk=st.wuk.data_ptr(), w_uv=st.wuv.data_ptr(), q_dtype=L.DTYPE_BF16,
                     out_dtype=L.DTYPE_F32, kv_dtype=L.DTYPE_BF16)
        _restart(st, st.pool)
        return st.out
    if k in ("gqa_prompt", "mla_prompt"):
        more = {} if k == "gqa_prompt" else dict(q_rope=st.qr.data_ptr(), w_uk=st.wuk.data_ptr(), w_uv=st.wuv.data_ptr())
        st.pool.set_len(0, st.lens)
        st.pool.append(0, st.a.data_ptr(), st.b.data_ptr(), c["B"], n_new=st.n_new, dtype=L.DTYPE_BF16)
        st.pool.decode(0, c["B"], st.q.data_ptr(), st.out.data_ptr(), c["H"], DH, DH ** -0.5 if k == "gqa_prompt" else (DH + DHR) ** -0.5,
                       q_tokens=c["S"], q_dtype=L.DTYPE_BF16, out_dtype=L.DTYPE_F32, **more)
        return st.out
    if k in ("gqa_layer", "mla_layer"):
        st.pool.forward_cached(0, c["B"], st.x, st.out.data_ptr(), {n: w.data_ptr() for n, w in st.w.items()}, c["H"] * DH, c["H"])
        _restart(st, st.pool)
        return st.out
    kw = dict(temperature=c["temperature"], top_k=c["top_k"], top_p=c["top_p"])
    if c["k"] == 0:
        return st.pool.sample(st.target.data_ptr(), st.draws.data_ptr(), vocab=c["V"], n_rows=c["B"], **kw)
    return st.pool.spec_accept(c["B"], c["k"], c["V"], st.tokens.data_ptr(), st.draft.data_ptr(), st.target.data_ptr(),
                               st.draws.data_ptr(), **kw)
