"""Loads and stores with an L2 priority on either side of the sizes that choose them: cached pages of more than half of L2, weights of more
than 16 MB with one block of rows and with several, results of 32 rows and of more."""
import numpy as np
import pytest

from tests.test_gpu_attention import dev  # noqa: F401

pytestmark = pytest.mark.gpu


# bf16 operands, float32 sums: products of rounded operands are exact in float32, what remains is the order of K sums
@pytest.mark.parametrize("m,k,n", [(16, 4096, 2048), (16, 4096, 2056), (32, 4096, 2304), (33, 4096, 2304), (300, 4096, 2304), (64, 1024, 512)])
def test_projection_around_the_limits(dev, oracle, m, k, n):  # noqa: F811
    import relux_b200 as rb
    from relux_b200 import lib as L
    rng = np.random.default_rng(m + n)
    pool = rb.Pool(dev, L.POOL_MLA, 1, 2, 64, 1, 2, dC=64, dHR=16)
    a = oracle.f32_from_bf16(oracle.bf16_from_f32(rng.standard_normal((m, k)).astype(np.float32)))
    w = oracle.bf16_from_f32(rng.standard_normal((k, n)).astype(np.float32))
    d_w = dev.upload(w)
    got = pool.matmul(a, d_w, n)
    ref = a.astype(np.float64) @ oracle.f32_from_bf16(w).astype(np.float64)
    # k float32 additions of terms of size 1: k * 2^-24 of the sum of their magnitudes (0.64 k) at the very most
    assert np.abs(got - ref).max() <= k * 2.0 ** -24 * 0.64 * k
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
    d_w.free()
    pool.destroy()


@pytest.mark.parametrize("B", [7, 8])            # 33 pages x 8 kv heads x 32 KB a sequence: 58 and 66 MB (half of L2: 63)
def test_cached_pages_around_half_of_l2(dev, oracle, B):  # noqa: F811
    import relux_b200 as rb
    from relux_b200 import lib as L
    rng = np.random.default_rng(B)
    H, HKV, D, T = 32, 8, 128, 2100
    pages = (T + 63) // 64
    pool = rb.Pool(dev, L.POOL_GQA, 1, B * pages, 64, B, pages, num_kv_heads=HKV, head_dim=D)
    pool.set_tables(rng.permutation(B * pages).astype(np.int32).reshape(B, pages))
    k, v = (oracle.bf16_from_f32(rng.standard_normal((B * T, HKV, D)).astype(np.float32)) for _ in range(2))
    pool.append(0, k, v, B, n_new=np.full(B, T, np.int32))
    q, out = rng.standard_normal((B, 1, H, D)).astype(np.float32), np.full((B, 1, H, D), np.nan, np.float32)
    pool.decode(0, B, q, out, H, D, D ** -0.5)
    kf, vf = (oracle.f32_from_bf16(x).reshape(B, T, HKV, D).astype(np.float64) for x in (k, v))
    qf = oracle.f32_from_bf16(oracle.bf16_from_f32(q)).astype(np.float64).reshape(B, HKV, H // HKV, D)
    s = np.einsum("bhgd,bthd->bhgt", qf, kf) * D ** -0.5
    p = np.exp(s - s.max(axis=-1, keepdims=True))
    ref = (np.einsum("bhgt,bthd->bhgd", p, vf) / p.sum(axis=-1)[..., None]).reshape(B, 1, H, D)
    assert np.linalg.norm(out - ref) <= 1e-2 * np.linalg.norm(ref)     # probabilities rounded to bf16
    assert pool.status() == 0
    pool.destroy()


# results of half of L2 (63 MB) and more are not stored to stay there: 2730 rows of 6144 columns are 67 MB, 2500 are 61
@pytest.mark.parametrize("m", [2500, 2730])
def test_a_result_that_does_not_fit_in_l2(dev, oracle, m):  # noqa: F811
    import relux_b200 as rb
    from relux_b200 import lib as L
    k, n = 256, 6144
    rng = np.random.default_rng(m)
    pool = rb.Pool(dev, L.POOL_MLA, 1, 2, 64, 1, 2, dC=64, dHR=16)
    a = oracle.f32_from_bf16(oracle.bf16_from_f32(rng.standard_normal((m, k)).astype(np.float32)))
    w = oracle.bf16_from_f32(rng.standard_normal((k, n)).astype(np.float32))
    d_w = dev.upload(w)
    got = pool.matmul(a, d_w, n)
    ref = a.astype(np.float64) @ oracle.f32_from_bf16(w).astype(np.float64)
    assert np.abs(got - ref).max() <= k * 2.0 ** -24 * 0.64 * k
    assert np.linalg.norm(got - ref) <= 1e-5 * np.linalg.norm(ref)
    d_w.free()
    pool.destroy()
