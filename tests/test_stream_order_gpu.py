"""Rows of calls on one stream in which each reads what the one before wrote:
elementwise updates, products and reductions are launched so that a call may
be scheduled while its predecessor finishes, and none may read early.  The
entries are small integers, so every result is exact."""
import numpy as np
import pytest

from gpu_utils import dev, host
from high_precision_blas1_b200 import Context, _lib

pytestmark = pytest.mark.gpu


def sizes(torch):
    """One element to a little more than 32 blocks of 256 two-element packs an SM."""
    cap = torch.cuda.get_device_properties(0).multi_processor_count * 32 * 256 * 2
    return [1, 511, 513, 100001, cap - 1, cap, cap + 3]


@pytest.mark.parametrize("which", range(7))
@pytest.mark.parametrize("shift", [0, 1])
def test_dependent_updates(gpu, which, shift):
    ctx, torch = gpu
    n = sizes(torch)[which]
    L = _lib.lib
    rng = np.random.default_rng(n)
    x, y = (rng.integers(-3, 4, n + shift).astype(float) for _ in range(2))
    dx, dy = dev(torch, x), dev(torch, y)
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    px, py = dx.data_ptr() + 8 * shift, dy.data_ptr() + 8 * shift
    for k in range(6):
        ctx.check(L.hpb_axpy_f64(ctx.h, n, 2.0, px, py), "axpy")
        ctx.check(L.hpb_axpby_f64(ctx.h, n, 1.0, py, -1.0, px), "axpby")
        ctx.check(L.hpb_dot2_f64(ctx.h, n, px, py, out.data_ptr()), "dot2")
    torch.cuda.synchronize()
    x, y = x[shift:], y[shift:]
    for k in range(6):
        y = y + 2 * x
        x = y - x
    assert np.array_equal(host(dx)[shift:], x) and np.array_equal(host(dy)[shift:], y)
    assert host(out)[0] == float(int(x.astype(np.int64) @ y.astype(np.int64)))


@pytest.mark.parametrize("n", [33, 4097, 300000])
def test_dependent_products(gpu, n):
    """x <- A x by products, an update in place and the product with its inner product."""
    ctx, torch = gpu
    L = _lib.lib
    i = np.arange(n)
    rp = np.arange(0, 2 * n + 1, 2).astype(np.int32)
    ci = np.stack([i, (i + 7) % n], 1).ravel().astype(np.int32)
    val = np.tile([2.0, -1.0], n)
    x = np.random.default_rng(n).integers(-3, 4, n).astype(float)
    a, b = dev(torch, x), torch.zeros(n, dtype=torch.float64, device="cuda")
    R, Cc, V = dev(torch, rp), dev(torch, ci), dev(torch, val)
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    A = lambda v: 2 * v - np.roll(v, -7)  # noqa: E731
    ar = (R.data_ptr(), Cc.data_ptr(), V.data_ptr())
    for k in range(4):
        ctx.check(L.hpb_csr_spmv_f64(ctx.h, n, n, 2 * n, *ar, 1.0, a.data_ptr(), 0.0, b.data_ptr()), "spmv")
        ctx.check(L.hpb_axpy_f64(ctx.h, n, 1.0, b.data_ptr(), a.data_ptr()), "axpy")
        ctx.check(L.hpb_csr_spmv_dot2_f64(ctx.h, n, n, 2 * n, *ar, a.data_ptr(), b.data_ptr(), a.data_ptr(),
                                          out.data_ptr()), "spmv_dot2")
    torch.cuda.synchronize()
    for k in range(4):
        x = x + A(x)
        y = A(x)
    assert np.array_equal(host(a), x) and np.array_equal(host(b), y)
    assert host(out)[0] == float(int(x.astype(np.int64) @ y.astype(np.int64)))


def test_captured_row_of_calls(gpu):
    """The same in a captured graph, replayed."""
    ctx, torch = gpu
    L = _lib.lib
    n = 100001
    x = np.random.default_rng(1).integers(-3, 4, n).astype(float)
    a, b = dev(torch, x), dev(torch, x)
    out = torch.zeros(4, dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    c2 = Context(0, s.cuda_stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        for k in range(3):
            c2.check(L.hpb_axpy_f64(c2.h, n, 2.0, a.data_ptr(), b.data_ptr()), "axpy")
            c2.check(L.hpb_axpby_f64(c2.h, n, 1.0, b.data_ptr(), -1.0, a.data_ptr()), "axpby")
        c2.check(L.hpb_dot2_f64(c2.h, n, a.data_ptr(), b.data_ptr(), out.data_ptr()), "dot2")
    for k in range(2):
        g.replay()
    torch.cuda.synchronize()
    x, y = x, x
    for k in range(6):
        y = y + 2 * x
        x = y - x
    assert np.array_equal(host(a), x) and np.array_equal(host(b), y)
    assert host(out)[0] == float(int(x.astype(np.int64) @ y.astype(np.int64)))
