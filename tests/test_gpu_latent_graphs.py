"""Latent calls captured in a graph: its launches run with the lengths that the device has then, and plain calls behind them on the same pool do so
too, against the same calls, none of them captured, on another pool."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_attention import dev  # noqa: F401
from tests.test_gpu_listed_plan import DC, DH, DHR, SCALE, latent_pool

pytestmark = pytest.mark.gpu


class Calls:
    """Steps (S = 1) and decode calls of all sequences of a pool, inputs on the device."""

    def __init__(self, dev, oracle, B, H, S=1):  # noqa: F811
        from relux_b200 import lib as L
        rng = np.random.default_rng(B + H)
        bf = lambda *s: dev.upload(oracle.bf16_from_f32(rng.standard_normal(s).astype(np.float32)))  # noqa: E731
        self.dev, self.shape, self.S = dev, (B, S, H, DH), S
        self.q, self.qr, self.c, self.r = bf(B, S, H, DH), bf(B, S, H, DHR), bf(B, DC), bf(B, DHR)
        self.w = [dev.upload(oracle.bf16_from_f32(rng.standard_normal((DC, H * DH)).astype(np.float32) * 0.02)) for _ in range(2)]
        self.kw = dict(q_rope=self.qr, w_uk=self.w[0], w_uv=self.w[1], q_dtype=L.DTYPE_BF16, out_dtype=L.DTYPE_F32)
        self.outs = [dev.upload(np.full(self.shape, np.nan, np.float32)) for _ in range(2)]

    def step(self, pool, k):
        from relux_b200 import lib as L
        B, _, H, _ = self.shape
        pool.step(0, B, self.c, self.r, self.q, self.outs[k], H, DH, SCALE, kv_dtype=L.DTYPE_BF16, **self.kw)

    def decode(self, pool, k):
        B, _, H, _ = self.shape
        pool.decode(0, B, self.q, self.outs[k], H, DH, SCALE, q_tokens=self.S, **self.kw)

    def same(self, what):
        self.dev.sync()
        want, got = (o.download(self.shape, np.float32) for o in self.outs)
        # the rounding of a row kept in one half, and of P under another cut of the sequences: a few times 1.7e-3 of the result's size, over all values
        assert np.isfinite(got).all() and np.max(np.abs(want - got)) <= 2e-2 * np.sqrt(np.mean(want ** 2)), what

    def free(self):
        for b in [self.q, self.qr, self.c, self.r] + self.w + self.outs:
            b.free()


class Graph:
    def __init__(self, dev, call):  # noqa: F811
        from relux_b200 import lib as L
        self.rt, self.stream, self.graph, self.ready = C.CDLL("libcudart.so.12"), C.c_void_p(), C.c_void_p(), C.c_void_p()
        L.check(dev.lib.relux_cuda_stream(dev.h, C.byref(self.stream)))
        assert self.rt.cudaStreamBeginCapture(self.stream, 2) == 0
        call()
        assert self.rt.cudaStreamEndCapture(self.stream, C.byref(self.graph)) == 0
        assert self.rt.cudaGraphInstantiate(C.byref(self.ready), self.graph, C.c_ulonglong(0)) == 0

    def launch(self):
        assert self.rt.cudaGraphLaunch(self.ready, self.stream) == 0

    def free(self):
        assert self.rt.cudaGraphExecDestroy(self.ready) == 0 and self.rt.cudaGraphDestroy(self.graph) == 0


@pytest.mark.parametrize("captured", ["step", "append"])
@pytest.mark.parametrize("after", ["step", "decode"])
def test_a_plain_call_behind_launches_of_a_graph(dev, oracle, captured, after):  # noqa: F811
    """The host has seen one call captured and none launched: the keys that the graph has appended must be attended to all the same."""
    from relux_b200 import lib as L
    ctx, H = [70, 300, 130, 40], 16
    calls = Calls(dev, oracle, len(ctx), H)
    plain, graphed = (latent_pool(dev, oracle, ctx, 8) for _ in range(2))

    def once(pool, k):
        if captured == "step":
            calls.step(pool, k)
        else:
            pool.append(0, calls.c, calls.r, len(ctx), dtype=L.DTYPE_BF16)
    for k, pool in enumerate((plain, graphed)):
        once(pool, k)
        calls.decode(pool, k)
    graph = Graph(dev, lambda: once(graphed, 1))
    for _ in range(5):
        once(plain, 0)
        graph.launch()
    for k, pool in enumerate((plain, graphed)):
        (calls.step if after == "step" else calls.decode)(pool, k)
    calls.same((captured, after))
    assert plain.status() == 0 and graphed.status() == 0
    graph.free()
    plain.destroy()
    graphed.destroy()
    calls.free()


def _random(n, most, seed):
    return [int(x) for x in np.random.default_rng(seed).integers(1, most, n)]


@pytest.mark.parametrize("ctx,H,later", [
    ([126] * 37, 16, None),                          # a piece a sequence: six tokens on none fits its worker
    (_random(65, 3050, 1), 16, None),                # ranges and five groups of heads' CTAs: borders move between the groups
    (_random(80, 1500, 2), 40, "turned"),
    ([1000, 64, 2500, 130], 128, "turned"),
    ([640] * 30, 32, "one"),                         # one sequence of all the length there is, the others almost empty
])
def test_a_graph_whose_lengths_have_outgrown_its_plan(dev, oracle, ctx, H, later):  # noqa: F811
    """Six launches, then lengths that the host sets: what a group of rows has in pieces is not what it had when the call was captured."""
    B, room = len(ctx), max(ctx)
    calls = Calls(dev, oracle, B, H)
    plain, graphed = (latent_pool(dev, oracle, [room] * B, 8) for _ in range(2))
    for k, pool in enumerate((plain, graphed)):
        pool.set_len(0, np.asarray(ctx, np.int32))
        calls.step(pool, k)
    graph = Graph(dev, lambda: calls.step(graphed, 1))
    graphed.set_len(0, np.asarray(ctx, np.int32) + 1)   # the host counts the captured call, which did not run
    for i in range(6):
        calls.step(plain, 0)
        graph.launch()
        calls.same(i)
    if later:
        for pool in (plain, graphed):
            pool.set_len(0, np.asarray(ctx[::-1] if later == "turned" else [room] + [3] * (B - 1), np.int32))
        for i in range(3):
            calls.step(plain, 0)
            graph.launch()
            calls.same((later, i))
    assert plain.status() == 0 and graphed.status() == 0
    graph.free()
    plain.destroy()
    graphed.destroy()
    calls.free()


@pytest.mark.parametrize("full", [0, 1, 9])
def test_a_graph_that_finds_empty_sequences(dev, oracle, full):  # noqa: F811
    """A captured decode call launched when all, or all but the first few, of its sequences have been emptied: zeros, and CTAs without a column."""
    B, H = 60, 16
    calls = Calls(dev, oracle, B, H)
    plain, graphed = (latent_pool(dev, oracle, [200] * B, 8) for _ in range(2))
    for k, pool in enumerate((plain, graphed)):
        calls.decode(pool, k)
    graph = Graph(dev, lambda: calls.decode(graphed, 1))
    calls.same("full")
    graphed.set_len(0, np.asarray([200] * full + [0] * (B - full), np.int32))
    for _ in range(3):
        graph.launch()
    dev.sync()
    want, got = (o.download(calls.shape, np.float32) for o in calls.outs)
    assert not got[full:].any()
    if full:
        assert np.max(np.abs(want[:full] - got[:full])) <= 2e-2 * np.sqrt(np.mean(want ** 2))
    assert graphed.status() == 0
    graph.free()
    plain.destroy()
    graphed.destroy()
    calls.free()


@pytest.mark.parametrize("dc,S", [(64, 1), (128, 1), (128, 3), (64, 2)])
def test_a_graph_of_the_plain_kernels_whose_chunks_become_fewer_or_more(dev, oracle, dc, S):  # noqa: F811
    """Latents that the CUDA-core kernels serve.  A decode call captured at ten pages a sequence and launched at one has CTAs without a chunk; captured at
    one and launched at ten it has more chunks than it has room for: nothing is written past that, zeros, and the status word says so."""
    import relux_b200 as rb
    from relux_b200 import lib as L
    B, H, pages = 5, 16, 10
    rng = np.random.default_rng(dc + S)
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, 64, B, pages, dC=dc, dHR=DHR)
    pool.set_tables(np.arange(B * pages, dtype=np.int32).reshape(B, pages))
    bf = lambda *s: oracle.bf16_from_f32(rng.standard_normal(s).astype(np.float32))  # noqa: E731
    pool.append(0, bf(B * 640, dc), bf(B * 640, DHR), B, n_new=np.full(B, 640, np.int32))
    pool.tune(L.TUNE_CHUNK_PAGES, 1)
    shape = (B, S, H, DH)
    q, qr, wuk, wuv = (dev.upload(x) for x in (bf(*shape), bf(B, S, H, DHR), bf(dc, H * DH), bf(dc, H * DH)))
    out = dev.upload(np.full(shape, np.nan, np.float32))

    def call():
        pool.decode(0, B, q, out, H, DH, 0.01, q_rope=qr, w_uk=wuk, w_uv=wuv, q_tokens=S, q_dtype=L.DTYPE_BF16, out_dtype=L.DTYPE_F32)

    def result():
        dev.sync()
        return out.download(shape, np.float32), pool.status()

    def launched(graph, tokens):
        pool.set_len(0, np.full(B, tokens, np.int32))
        graph.launch()
        return result()

    def same(a, b):
        return np.max(np.abs(a - b)) <= 1e-2 * np.sqrt(np.mean(b ** 2))
    want, graphs = {}, {}
    for tokens in (640, 60):
        pool.set_len(0, np.full(B, tokens, np.int32))
        call()
        want[tokens] = result()[0]
        graphs[tokens] = Graph(dev, call)
    for at, tokens in ((60, 60), (640, 60), (640, 640), (640, 60)):
        got, status = launched(graphs[at], tokens)
        assert status == 0 and same(got, want[tokens]), (at, tokens)
    got, status = launched(graphs[60], 640)
    assert status == L.ERR_UNSUPPORTED and not got.any()
    got, status = launched(graphs[60], 60)
    assert status == 0 and same(got, want[60])
    for g in graphs.values():
        g.free()
    pool.destroy()
    for b in (q, qr, wuk, wuv, out):
        b.free()


@pytest.mark.parametrize("dc,H,S", [(128, 16, 1), (256, 16, 2), (512, 8, 1)])
def test_a_graph_of_the_plain_kernels_whose_chunks_move(dev, oracle, dc, H, S):  # noqa: F811
    """As many chunks as at capture, in other sequences: one group of rows of the up-projection has those of two."""
    import relux_b200 as rb
    from relux_b200 import lib as L
    B, pages = 24, 10
    rng = np.random.default_rng(dc + S)
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * pages, 64, B, pages, dC=dc, dHR=DHR)
    pool.set_tables(np.arange(B * pages, dtype=np.int32).reshape(B, pages))
    bf = lambda *s: oracle.bf16_from_f32(rng.standard_normal(s).astype(np.float32))  # noqa: E731
    pool.append(0, bf(B * 640, dc), bf(B * 640, DHR), B, n_new=np.full(B, 640, np.int32))
    pool.tune(L.TUNE_CHUNK_PAGES, 1)
    shape = (B, S, H, DH)
    q, qr, wuk, wuv = (dev.upload(x) for x in (bf(*shape), bf(B, S, H, DHR), bf(dc, H * DH), bf(dc, H * DH)))
    outs = [dev.upload(np.full(shape, np.nan, np.float32)) for _ in range(2)]

    def call(k):
        pool.decode(0, B, q, outs[k], H, DH, 0.01, q_rope=qr, w_uk=wuk, w_uv=wuv, q_tokens=S, q_dtype=L.DTYPE_BF16, out_dtype=L.DTYPE_F32)

    def lengths(longest):
        pool.set_len(0, np.asarray([630 if i in longest else 50 for i in range(B)], np.int32))
    lengths((0, 1, 22, 23))
    call(1)
    graph = Graph(dev, lambda: call(1))
    for longest in ((0, 1, 22, 23), (20, 21, 22, 23), (0, 1, 2, 3), (11, 12)):
        lengths(longest)
        call(0)
        graph.launch()
        dev.sync()
        want, got = (o.download(shape, np.float32) for o in outs)
        assert pool.status() == 0 and np.max(np.abs(want - got)) <= 1e-2 * np.sqrt(np.mean(want ** 2)), longest
    graph.free()
    pool.destroy()
    for b in [q, qr, wuk, wuv] + outs:
        b.free()
