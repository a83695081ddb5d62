"""Reductions at the sizes around the one-block form's line (4096 packs of 16
bytes, 4096 elements off a 16-byte boundary): small integers, so that every
sum is exact in each storage type."""
import numpy as np
import pytest

from gpu_utils import dev, red_ptr
from high_precision_blas1_b200 import _lib

pytestmark = pytest.mark.gpu
DT = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("t", ["f32", "f64", "c64", "c128"])
def test_line(gpu, t, shift):
    ctx, torch = gpu
    cplx = t[0] == "c"
    K = 16 // np.dtype(DT[t]).itemsize
    rng = np.random.default_rng(K)
    top = 4097 * K + 1
    x, y = ((rng.integers(-2, 3, top + 1) + (1j * rng.integers(-2, 3, top + 1) if cplx else 0)).astype(DT[t])
            for _ in range(2))
    X, Y = dev(torch, x), dev(torch, y)
    off = shift * x.itemsize
    for n in sorted({0, 1, K, 32 * K - 1, 32 * K, 1024 * K, 1024 * K + 1, 4095, 4096, 4097, 4096 * K - 1, 4096 * K,
                     4097 * K - 1, 4097 * K, top}):
        a, b = (v[shift:shift + n].astype(complex if cplx else float) for v in (x, y))
        px, py = X.data_ptr() + off, Y.data_ptr() + off
        for op in ("dot2", "dot"):
            o = red_ptr(ctx, op, t, n, px, py)
            w = np.sum(np.conj(a) * b)
            assert o[0] == w.real and (not cplx or o[1] == w.imag), (op, n)
        o = red_ptr(ctx, "sum2", t, n, px)
        assert o[0] == np.sum(a).real and (not cplx or o[1] == np.sum(a).imag), n
        for op in ("asum2", "asum"):
            assert red_ptr(ctx, op, t, n, px)[0] == np.sum(np.abs(a.real) + np.abs(a.imag)), (op, n)
        for op in ("nrm2", "nrm2plain"):
            w = np.sqrt(np.sum(a.real ** 2 + a.imag ** 2))
            assert any(abs(q - w) <= 4e-16 * w for q in red_ptr(ctx, op, t, n, px)[:3]), (op, n)
        out = torch.zeros(4, dtype=torch.float64, device="cuda")  # the result left on the device
        ctx.check(getattr(_lib.lib, f"hpb_dot2_{t}")(ctx.h, n, px, py, out.data_ptr()), "dot2")
        assert out[0].item() == np.sum(np.conj(a) * b).real
