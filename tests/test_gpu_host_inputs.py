"""Small inputs from host memory: the block they pass through starts again behind its end and behind a call that waits; their source
may be reused at once; sizes on either side of the limit; an address in device memory given as host memory."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_attention import dev  # noqa: F401

pytestmark = pytest.mark.gpu

HKV, D, PAGE = 8, 128, 64


def gqa_pool(dev, tokens, kv=HKV):  # noqa: F811
    import relux_b200 as rb
    from relux_b200 import lib as L
    pages = (tokens + PAGE - 1) // PAGE
    pool = rb.Pool(dev, L.POOL_GQA, 1, pages, PAGE, 1, pages, num_kv_heads=kv, head_dim=D)
    pool.set_tables(np.arange(pages, dtype=np.int32).reshape(1, pages))
    return pool


def test_rows_appended_one_after_another_pass_the_end_of_the_block(dev, oracle):  # noqa: F811
    n = 400                                     # 2 x 4 KB each: three times the block
    pool = gqa_pool(dev, n)
    rng = np.random.default_rng(0)
    rows = rng.standard_normal((n, 2, HKV, D)).astype(np.float32)
    k, v = np.empty((1, HKV, D), np.float32), np.empty((1, HKV, D), np.float32)
    for i in range(n):                          # one source, written again as soon as the call returns
        k[0], v[0] = rows[i]
        pool.append(0, k, v, 1)
    got_k, got_v = pool.read_rows(0, 0, 0, n)
    assert np.array_equal(got_k, oracle.bf16_from_f32(rows[:, 0])) and np.array_equal(got_v, oracle.bf16_from_f32(rows[:, 1]))
    assert pool.status() == 0
    pool.destroy()


@pytest.mark.parametrize("n", [1, 7, 8, 9, 16])   # rows of 4 KB: 32 KB, the limit, and past it
def test_sizes_around_the_limit_and_steps_between_appends(dev, oracle, n):  # noqa: F811
    pool = gqa_pool(dev, 200)
    rng = np.random.default_rng(n)
    H, want = 16, []
    for step in range(3):
        a, b = (rng.standard_normal((n, HKV, D)).astype(np.float32) for _ in range(2))
        pool.append(0, a, b, 1, n_new=[n])
        k, v = (rng.standard_normal((1, HKV, D)).astype(np.float32) for _ in range(2))
        q, out = rng.standard_normal((1, 1, H, D)).astype(np.float32), np.full((1, 1, H, D), np.nan, np.float32)
        pool.step(0, 1, k, v, q, out, H, D, D ** -0.5)   # waits: the block starts again behind it
        assert np.isfinite(out).all()
        want.append((np.concatenate([a, k]), np.concatenate([b, v])))
    got_k, got_v = pool.read_rows(0, 0, 0, 3 * (n + 1))
    assert np.array_equal(got_k, oracle.bf16_from_f32(np.concatenate([w[0] for w in want])))
    assert np.array_equal(got_v, oracle.bf16_from_f32(np.concatenate([w[1] for w in want])))
    pool.destroy()


def test_a_device_address_given_as_host_memory(dev, oracle):  # noqa: F811
    from relux_b200 import lib as L
    pool = gqa_pool(dev, 10)
    rows = np.random.default_rng(3).standard_normal((2, HKV, D)).astype(np.float32)
    d_k, d_v = dev.upload(rows[:1]), dev.upload(rows[1:])
    args = L.AppendArgs(layer=0, n_seqs=1, a=d_k.ptr, b=d_v.ptr, dtype=L.DTYPE_F32, mem=L.MEM_HOST, layout=L.LAYOUT_TOKEN_MAJOR, advance=1)
    L.check(pool.lib.relux_gqa_append(pool.h, C.byref(args)))
    dev.sync()
    got_k, got_v = pool.read_rows(0, 0, 0, 1)
    assert np.array_equal(got_k, oracle.bf16_from_f32(rows[:1])) and np.array_equal(got_v, oracle.bf16_from_f32(rows[1:]))
    pool.destroy()
    d_k.free()
    d_v.free()


def check_rows(dev, oracle, seed, per_call):  # noqa: F811
    n = sum(per_call)
    pool = gqa_pool(dev, n)
    rows = np.random.default_rng(seed).standard_normal((2, n, HKV, D)).astype(np.float32)
    at = 0
    for m in per_call:
        k, v = rows[:, at:at + m].copy()        # gone as soon as the call returns
        pool.append(0, k, v, 1, n_new=[m])
        k[:], v[:] = np.nan, np.nan
        at += m
    got_k, got_v = pool.read_rows(0, 0, 0, n)
    assert np.array_equal(got_k, oracle.bf16_from_f32(rows[0])) and np.array_equal(got_v, oracle.bf16_from_f32(rows[1]))
    assert pool.status() == 0
    pool.destroy()


@pytest.mark.parametrize("rows", [3, 5])        # 12 and 20 KB a tensor: the block's end falls between a call's two tensors
def test_pairs_that_do_not_divide_the_block(dev, oracle, rows):  # noqa: F811
    check_rows(dev, oracle, rows, [rows] * 180)  # four and seven turns of the block


def test_mixed_sizes_over_several_turns_of_the_block(dev, oracle):  # noqa: F811
    check_rows(dev, oracle, 9, [int(m) for m in np.random.default_rng(9).integers(1, 11, 200)])   # past the limit (8 rows) too


def test_latent_rows_over_several_turns_of_the_block(dev, oracle):  # noqa: F811
    import relux_b200 as rb
    from relux_b200 import lib as L
    calls, m, dc, dhr = 180, 8, 512, 64         # 16 KB + 2 KB a call
    n = calls * m
    pages = (n + PAGE - 1) // PAGE
    pool = rb.Pool(dev, L.POOL_MLA, 1, pages, PAGE, 1, pages, dC=dc, dHR=dhr)
    pool.set_tables(np.arange(pages, dtype=np.int32).reshape(1, pages))
    rng = np.random.default_rng(4)
    c, r = (rng.standard_normal((n, w)).astype(np.float32) for w in (dc, dhr))
    for i in range(0, n, m):
        pool.append(0, c[i:i + m].copy(), r[i:i + m].copy(), 1, n_new=[m])
    got_c, got_r = pool.read_rows(0, 0, 0, n)
    assert np.array_equal(got_c, oracle.bf16_from_f32(c)) and np.array_equal(got_r, oracle.bf16_from_f32(r))
    pool.destroy()
