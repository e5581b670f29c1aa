"""The tcgen05 projection GEMM at the sizes where its row blocks (16 to 256), its 128-column tiles and its ranges of K steps
can go wrong, and where its row blocks fill the SMs in turns, against float64 on the same bf16 operands."""
import numpy as np
import pytest

from tests.test_gpu_backend import dev, pool  # noqa: F401

pytestmark = pytest.mark.gpu

# (M, K, N): row blocks exactly full, one over, several; K below a step, ragged, many steps; N below a tile, ragged, a tile and
# a bit; pieces that begin and end inside a tile (units that are no multiple of the SMs)
CASES = [(1, 8, 8), (16, 64, 128), (17, 72, 136), (32, 4096, 64), (33, 1000, 264), (64, 2048, 4096), (65, 16384, 200), (128, 520, 1032),
         (129, 4096, 384), (256, 192, 72), (257, 640, 520), (700, 328, 1160), (5, 4096, 19200),
         (200, 4096, 1024), (300, 4096, 6144), (520, 2048, 1160), (2049, 520, 264), (4700, 264, 1032), (12801, 328, 136), (19200, 136, 640),
         (40001, 72, 72)]


@pytest.mark.parametrize("M,K,N", CASES)
def test_projection_gemm_sizes(dev, pool, oracle, M, K, N):  # noqa: F811
    rng = np.random.default_rng(M * 7 + K * 3 + N)
    a = rng.standard_normal((M, K)).astype(np.float32)
    w = oracle.bf16_from_f32(rng.standard_normal((K, N)).astype(np.float32))
    d_w = dev.upload(w)
    a64 = oracle.f32_from_bf16(oracle.bf16_from_f32(a)).astype(np.float64)
    w64 = oracle.f32_from_bf16(w).astype(np.float64)
    for _ in range(2):   # the second call meets the first one's leftovers in the scratch
        out = pool.matmul(a, d_w, N)
        # float32 sums of K products of about unit size, in an order of the kernel's own: K * 2^-24 times the sum of the
        # products' sizes bounds every order
        bound = K * 2.0 ** -24 * (np.abs(a64) @ np.abs(w64)) + 1e-30
        assert (np.abs(out - a64 @ w64) <= bound).all()
    d_w.free()
    assert pool.status() == 0
