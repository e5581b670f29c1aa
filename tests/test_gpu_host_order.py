"""New rows in page-locked memory are read in the order of the device's stream, as everything else that is queued there: behind a copy that
is still filling it, and, in a captured graph, when the graph is launched."""
import ctypes as C

import numpy as np
import pytest

from tests.test_gpu_attention import dev  # noqa: F401
from tests.test_gpu_host_inputs import D, HKV, gqa_pool

pytestmark = pytest.mark.gpu

ROW = HKV * D


def locked(dev, n):  # noqa: F811
    """(float32 array, address) of page-locked memory."""
    p = C.c_void_p()
    from relux_b200 import lib as L
    L.check(dev.lib.relux_cuda_host_alloc(dev.h, n * 4, C.byref(p)))
    return np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), (n,)), p


@pytest.mark.parametrize("step", [False, True])
def test_rows_that_an_earlier_copy_still_writes(dev, oracle, step):  # noqa: F811
    from relux_b200 import lib as L
    pool = gqa_pool(dev, 100)
    rng = np.random.default_rng(int(step))
    rows = rng.standard_normal((2, 1, HKV, D)).astype(np.float32)
    d_rows = dev.upload(rows)
    host, at = locked(dev, 2 * ROW)
    host[:] = -7.0
    big = C.c_void_p()
    size = 2 << 30
    L.check(dev.lib.relux_cuda_dev_alloc(dev.h, size, C.byref(big)))
    q = dev.upload(rng.standard_normal((1, 1, 16, D)).astype(np.float32))
    out = dev.upload(np.zeros((1, 1, 16, D), np.float32))
    dev.sync()
    for _ in range(8):                          # some milliseconds of work ahead of the copy
        L.check(dev.lib.relux_cuda_memset(dev.h, big, 1, size))
    rt, stream = C.CDLL("libcudart.so.12"), C.c_void_p()
    L.check(dev.lib.relux_cuda_stream(dev.h, C.byref(stream)))
    assert rt.cudaMemcpyAsync(at, C.c_void_p(d_rows.ptr), C.c_size_t(host.nbytes), 2, stream) == 0
    k, v = host[:ROW].reshape(1, HKV, D), host[ROW:].reshape(1, HKV, D)
    if step:
        pool.step(0, 1, k, v, q, out, 16, D, D ** -0.5, q_dtype=L.DTYPE_F32, out_dtype=L.DTYPE_F32)
    else:
        pool.append(0, k, v, 1)
    got_k, got_v = pool.read_rows(0, 0, 0, 1)
    assert np.array_equal(got_k, oracle.bf16_from_f32(rows[0])) and np.array_equal(got_v, oracle.bf16_from_f32(rows[1]))
    pool.destroy()
    for b in (d_rows, q, out):
        b.free()
    L.check(dev.lib.relux_cuda_dev_free(dev.h, big))
    L.check(dev.lib.relux_cuda_host_free(dev.h, at))


def test_a_captured_append_reads_its_rows_at_launch(dev, oracle):  # noqa: F811
    from relux_b200 import lib as L
    rt = C.CDLL("libcudart.so.12")
    pool = gqa_pool(dev, 100)
    rng = np.random.default_rng(5)
    host, at = locked(dev, 2 * ROW)
    k, v = host[:ROW].reshape(1, HKV, D), host[ROW:].reshape(1, HKV, D)
    host[:] = 1.0
    pool.append(0, k, v, 1)                     # everything that a first call sets up
    dev.sync()
    stream, graph, ready = C.c_void_p(), C.c_void_p(), C.c_void_p()
    L.check(dev.lib.relux_cuda_stream(dev.h, C.byref(stream)))
    assert rt.cudaStreamBeginCapture(stream, 2) == 0
    pool.append(0, k, v, 1, advance=False)
    assert rt.cudaStreamEndCapture(stream, C.byref(graph)) == 0
    assert rt.cudaGraphInstantiate(C.byref(ready), graph, C.c_ulonglong(0)) == 0
    for _ in range(3):
        rows = rng.standard_normal((2, 1, HKV, D)).astype(np.float32)
        host[:] = rows.reshape(-1)
        assert rt.cudaGraphLaunch(ready, stream) == 0
        dev.sync()
        got_k, got_v = pool.read_rows(0, 0, 1, 1)
        assert np.array_equal(got_k, oracle.bf16_from_f32(rows[0])) and np.array_equal(got_v, oracle.bf16_from_f32(rows[1]))
    assert rt.cudaGraphExecDestroy(ready) == 0 and rt.cudaGraphDestroy(graph) == 0
    pool.destroy()
    L.check(dev.lib.relux_cuda_host_free(dev.h, at))
