"""Triangular solves of rows with more dependencies than the four that every
row's lane holds: up to fourteen are taken in before the warp's turn, the rest
during it.  Lengths on both sides of both, in tiles of their own and across
tiles, bit for bit against the CPU restatement."""
import ctypes as C

import numpy as np
import pytest

import oracle
from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib

pytestmark = pytest.mark.gpu
DT = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}


@pytest.mark.parametrize("t", ["f64", "f32", "c128", "c64"])
@pytest.mark.parametrize("most", [5, 13, 14, 15, 31])
@pytest.mark.parametrize("n,reach", [(40, 39), (3000, 60), (17000, 9000)])
def test_long_rows(gpu, n, reach, most, t):
    ctx, torch = gpu
    rng = np.random.default_rng(most + n)
    per = np.where(rng.random(n) < 0.3, most, rng.integers(0, most + 1, n))
    rows, cols = [np.arange(n)], [np.arange(n)]
    for k in range(most):  # to the left and, mirrored, to the right
        i = np.nonzero(per > k)[0]
        j = i - rng.integers(1, reach + 1, len(i))
        ok = j >= 0
        rows += [i[ok], n - 1 - i[ok]]
        cols += [j[ok], n - 1 - j[ok]]
    key = np.unique(np.concatenate(rows).astype(np.int64) * n + np.concatenate(cols))
    r, c = (key // n), (key % n).astype(np.int32)
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(r, minlength=n))
    cplx = t in ("c64", "c128")
    val = rng.uniform(-1, 1, len(c)) / most + (1j * rng.uniform(-1, 1, len(c)) / most if cplx else 0)
    val = np.where(r == c, 2.0 + val, val).astype(DT[t])
    b = (rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)).astype(DT[t])
    d = [dev(torch, a) for a in (rp, c, val, b)]
    x = torch.zeros_like(d[3])
    for upper in (0, 1):
        h = C.c_void_p()
        ctx.check(_lib.lib.hpb_csr_tri_create(ctx.h, upper, n, len(c), d[0].data_ptr(), d[1].data_ptr(), C.byref(h)), "create")
        try:
            for unit in (0, 1):
                ctx.check(getattr(_lib.lib, f"hpb_csr_trsv_{t}")(
                    ctx.h, h, unit, d[2].data_ptr(), _lib.scalar(t, 1.0), d[3].data_ptr(), x.data_ptr()), "trsv")
                want = oracle.csr_trsv(rp, c, val, b, bool(upper), bool(unit), 1.0)
                assert np.array_equal(host(x), want), (upper, unit)
        finally:
            _lib.lib.hpb_csr_tri_destroy(h)
