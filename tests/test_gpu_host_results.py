"""Results for host memory: small ones are written to page-locked memory by the kernel, larger ones are copied; either way they are
the bits that the same call leaves in device memory.  Named sequences 0, 1, ... are the unnamed ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HKV, D, H = 8, 128, 32


@pytest.fixture(scope="module")
def dev():
    import relux_b200 as rb
    d = rb.Device(0)
    yield d
    d.close()


# 512 KB is 32 rows of 32 heads x 128 float32: below, at and above it; a prompt (12 query tokens) keeps to device memory
@pytest.mark.parametrize("B,S", [(1, 1), (32, 1), (33, 1), (16, 2), (17, 2), (1, 12)])
@pytest.mark.parametrize("out_dtype", [np.float32, np.uint16])
@pytest.mark.parametrize("head_major", [False, True])
def test_gqa_result_in_host_memory_equals_the_one_in_device_memory(dev, B, S, out_dtype, head_major):
    import relux_b200 as rb
    from relux_b200 import lib as L
    rng = np.random.default_rng(B * 31 + S)
    lens = rng.integers(S, 150, B).astype(np.int32)
    pool = rb.Pool(dev, L.POOL_GQA, 1, B * 3, 64, B, 3, num_kv_heads=HKV, head_dim=D)
    pool.set_tables(rng.permutation(B * 3).astype(np.int32).reshape(B, 3))
    rows = int(lens.sum())
    pool.append(0, rng.standard_normal((rows, HKV, D)).astype(np.float32), rng.standard_normal((rows, HKV, D)).astype(np.float32), B, n_new=lens)
    shape = (B, H, S, D) if head_major else (B, S, H, D)
    q = rng.standard_normal(shape).astype(np.float32)
    lay = L.LAYOUT_HEAD_MAJOR if head_major else L.LAYOUT_TOKEN_MAJOR
    out = np.zeros(shape, out_dtype)
    pool.decode(0, B, q, out, H, D, D ** -0.5, q_tokens=S, q_layout=lay, out_layout=lay)
    named = np.zeros(shape, out_dtype)
    pool.decode(0, B, q, named, H, D, D ** -0.5, q_tokens=S, q_layout=lay, out_layout=lay, seq_ids=list(range(B)))
    buf = dev.alloc(out.nbytes, L.DTYPE_F32 if out_dtype == np.float32 else L.DTYPE_BF16)
    pool.decode(0, B, q, buf, H, D, D ** -0.5, q_tokens=S, q_layout=lay, out_layout=lay)
    dev.sync()
    want = buf.download(shape, out_dtype)
    assert np.array_equal(out, want) and np.array_equal(named, want)
    assert np.abs(want.astype(np.float32)).max() > 0 and pool.status() == 0
    buf.free()
    pool.destroy()


def test_device_memory_given_as_host_memory_is_copied_to(dev):
    """The copy behind a kernel takes whatever address it is given; a result by way of page-locked memory does too."""
    import ctypes as C

    import relux_b200 as rb
    from relux_b200 import lib as L
    rng = np.random.default_rng(3)
    pool = rb.Pool(dev, L.POOL_GQA, 1, 3, 64, 1, 3, num_kv_heads=HKV, head_dim=D)
    pool.set_tables(np.arange(3, dtype=np.int32).reshape(1, 3))
    pool.append(0, rng.standard_normal((100, HKV, D)).astype(np.float32), rng.standard_normal((100, HKV, D)).astype(np.float32), 1,
                n_new=np.asarray([100], np.int32))
    q = rng.standard_normal((1, 1, H, D)).astype(np.float32)
    out = np.zeros_like(q)
    pool.decode(0, 1, q, out, H, D, D ** -0.5)
    buf = dev.alloc(out.nbytes, L.DTYPE_F32)
    args = pool._attn_args(0, 1, q, None, out, H, D, D ** -0.5, 1, 0, True, L.ATTN_FAST, None, None, None, L.LAYOUT_TOKEN_MAJOR,
                           L.LAYOUT_TOKEN_MAJOR, None, None)
    args.out = buf.ptr
    assert args.out_mem == L.MEM_HOST
    L.check(pool.lib.relux_gqa_decode(pool.h, C.byref(args)))
    assert np.array_equal(buf.download(out.shape, np.float32), out) and pool.status() == 0
    buf.free()
    pool.destroy()


# 512 KB is 8 rows of 128 heads x 128 float32; three query tokens of head-major rows go through the conversion
@pytest.mark.parametrize("B,S", [(1, 1), (8, 1), (9, 1), (2, 3), (3, 3)])
@pytest.mark.parametrize("out_dtype", [np.float32, np.uint16])
@pytest.mark.parametrize("head_major", [False, True])
@pytest.mark.parametrize("generic", [0, 1])    # the merge that projects up, and the kernels for other shapes
def test_latent_result_in_host_memory_equals_the_one_in_device_memory(dev, B, S, out_dtype, head_major, generic):
    import relux_b200 as rb
    from relux_b200 import lib as L
    from oracle import binding as orc
    H, DC, DHR = 128, 512, 64
    rng = np.random.default_rng(B * 17 + S)
    lens = rng.integers(S, 150, B).astype(np.int32)
    pool = rb.Pool(dev, L.POOL_MLA, 1, B * 3, 64, B, 3, dC=DC, dHR=DHR)
    pool.set_tables(rng.permutation(B * 3).astype(np.int32).reshape(B, 3))
    pool.tune(L.TUNE_MLA_GENERIC, generic)
    rows = int(lens.sum())
    pool.append(0, rng.standard_normal((rows, DC)).astype(np.float32), rng.standard_normal((rows, DHR)).astype(np.float32), B, n_new=lens)
    w = [dev.upload(orc.bf16_from_f32(0.02 * rng.standard_normal((DC, H * D)).astype(np.float32))) for _ in range(2)]
    shape = (B, H, S, D) if head_major else (B, S, H, D)
    q = rng.standard_normal(shape).astype(np.float32)
    qr = rng.standard_normal(shape[:3] + (DHR,)).astype(np.float32)
    lay = L.LAYOUT_HEAD_MAJOR if head_major else L.LAYOUT_TOKEN_MAJOR
    kw = dict(q_rope=qr, w_uk=w[0], w_uv=w[1], q_tokens=S, q_layout=lay, out_layout=lay)
    out = np.zeros(shape, out_dtype)
    pool.decode(0, B, q, out, H, D, (D + DHR) ** -0.5, **kw)
    buf = dev.alloc(out.nbytes, L.DTYPE_F32 if out_dtype == np.float32 else L.DTYPE_BF16)
    pool.decode(0, B, q, buf, H, D, (D + DHR) ** -0.5, **kw)
    dev.sync()
    assert np.array_equal(out, buf.download(shape, out_dtype))
    assert out.any() and pool.status() == 0
    for x in (buf, *w):
        x.free()
    pool.destroy()
