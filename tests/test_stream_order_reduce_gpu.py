"""A reduction directly behind the call that writes its input, in every element
type: vectors that one block reduces (up to 4096 packs of 16 bytes) and longer
ones, aligned and not.  The entries are small integers, so every sum is exact
and a value read before the update has finished shows."""
import numpy as np
import pytest

from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib

pytestmark = pytest.mark.gpu
NP = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}
PACK = {"f32": 4, "f64": 2, "c64": 2, "c128": 1}


@pytest.mark.parametrize("t", ["f32", "f64", "c64", "c128"])
@pytest.mark.parametrize("packs,shift", [(40, 0), (2048, 0), (4096, 0), (4097, 0), (200000, 0), (900, 1), (200000, 1)])
def test_reduction_after_update(gpu, t, packs, shift):
    ctx, torch = gpu
    L = _lib.lib
    n = packs * PACK[t] + 1
    rng = np.random.default_rng(packs)
    cplx = t in ("c64", "c128")
    draw = lambda: rng.integers(-3, 4, n + shift) + (1j * rng.integers(-3, 4, n + shift) if cplx else 0)  # noqa: E731
    x, y = draw(), draw()
    dx, dy = dev(torch, x.astype(NP[t])), dev(torch, y.astype(NP[t]))
    size = np.dtype(NP[t]).itemsize
    px, py = dx.data_ptr() + size * shift, dy.data_ptr() + size * shift
    got = torch.zeros(8, 4, 4, dtype=torch.float64, device="cuda")
    a = _lib.scalar(t, -1.0)
    call = lambda op, *args: ctx.check(getattr(L, f"hpb_{op}_{t}")(ctx.h, n, *args), op)  # noqa: E731
    for k in range(8):  # x <- y - x: alternates between two vectors
        call("axpby", _lib.scalar(t, 1.0), py, a, px)
        call("dot2", px, py, got[k, 0].data_ptr())
        call("axpby", _lib.scalar(t, 1.0), py, a, px)
        call("nrm2", px, got[k, 1].data_ptr())
        call("axpby", _lib.scalar(t, 1.0), py, a, px)
        call("sum2", px, got[k, 2].data_ptr())
        call("axpby", _lib.scalar(t, 1.0), py, a, px)
        call("asum2", px, got[k, 3].data_ptr())
    torch.cuda.synchronize()
    got = host(got)
    x, y = x[shift:], y[shift:]
    z = y - x
    dot, total = np.vdot(z, y), z.sum()
    for k in range(8):
        assert (got[k, 0, 0], got[k, 0, 1] if cplx else 0.0) == (dot.real, dot.imag if cplx else 0.0)
        # the norm's square is an integer
        assert abs(got[k, 1, 0] ** 2 - np.vdot(x, x).real) < 0.25
        assert (got[k, 2, 0], got[k, 2, 1] if cplx else 0.0) == (total.real, total.imag if cplx else 0.0)
        assert got[k, 3, 0] == np.abs(x.real).sum() + np.abs(x.imag).sum()
