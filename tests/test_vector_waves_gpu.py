"""Elementwise updates around the sizes at which their grid changes (16 and 32
blocks of 256 packs an SM), in every type, aligned and one element past a
16-byte boundary.  Small integers: every result is exact."""
import numpy as np
import pytest

from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib

pytestmark = pytest.mark.gpu
NP = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}
PACK = {"f32": 4, "f64": 2, "c64": 2, "c128": 1}


@pytest.mark.parametrize("t", ["f32", "f64", "c64", "c128"])
@pytest.mark.parametrize("per_sm", [8, 16, 32])
@pytest.mark.parametrize("more,shift", [(-1, 0), (0, 0), (1, 0), (1, 1)])
def test_grid_edges(gpu, t, per_sm, more, shift):
    ctx, torch = gpu
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = per_sm * sms * 256 * (1 if shift else PACK[t]) + more
    rng = np.random.default_rng(per_sm)
    cplx = t in ("c64", "c128")
    v = [(rng.integers(-3, 4, n + shift) + (1j * rng.integers(-3, 4, n + shift) if cplx else 0)).astype(NP[t])
         for _ in range(3)]
    d = [dev(torch, a) for a in v]
    at = np.dtype(NP[t]).itemsize * shift
    c = [_lib.scalar(t, k) for k in (2.0, -1.0, 3.0)]
    args = [x for k in range(3) for x in (c[k], d[k].data_ptr() + at)]
    for _ in range(2):
        ctx.check(getattr(_lib.lib, f"hpb_axpbypcz_{t}")(ctx.h, n, *args), "axpbypcz")
    torch.cuda.synchronize()
    x, y, z = (a[shift:] for a in v)
    want = 2 * x - y + 3 * (2 * x - y + 3 * z)
    got = host(d[2])
    assert np.array_equal(got[shift:], want) and np.array_equal(got[:shift], v[2][:shift])
