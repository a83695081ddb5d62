"""Triangular solves and ILU(0) where the solve's chunks end with a level and
where they do not, bit for bit against the CPU restatement: grids whose
levels hold 2 to 82 rows of a tile, a chain (a level a row) and rows without
dependencies (one level)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib

pytestmark = pytest.mark.gpu
DT = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}


def grid(n, nx, t):
    """5-point pattern on rows of nx (nx = 1: a chain, 0: the diagonal alone)."""
    rng = np.random.default_rng(nx)
    i = np.arange(n, dtype=np.int64)
    keys = [i * n + i]
    for d in ((1, nx) if nx > 1 else (1,) if nx else ()):
        a = i[d:] if d == nx or nx == 1 else i[i % nx > 0]
        keys += [a * n + a - d, (a - d) * n + a]
    key = np.unique(np.concatenate(keys))
    r, c = key // n, key % n
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(r, minlength=n))
    val = rng.uniform(-1, 1, len(c))
    b = rng.standard_normal(n)
    if t in ("c64", "c128"):
        val, b = val + 1j * rng.uniform(-1, 1, len(c)), b + 1j * rng.standard_normal(n)
    return rp, c.astype(np.int32), np.where(r == c, 6.0 + val, val).astype(DT[t]), b.astype(DT[t])


@pytest.mark.parametrize("t", ["f64", "f32", "c128", "c64"])
@pytest.mark.parametrize("n,nx", [(20001, 4096), (16384, 1024), (17000, 900), (16385, 256), (9000, 250), (20000, 100),
                                  (8193, 1), (9000, 0), (33, 8)])
def test_chunks(gpu, n, nx, t):
    ctx, torch = gpu
    L = _lib.lib
    rp, ci, val, b = grid(n, nx, t)
    rpd, cid, vd, bd = (dev(torch, a) for a in (rp, ci, val, b))
    xd = torch.zeros_like(bd)
    for upper in (0, 1):
        h = C.c_void_p()
        ctx.check(L.hpb_csr_tri_create(ctx.h, upper, n, len(ci), rpd.data_ptr(), cid.data_ptr(), C.byref(h)), "create")
        try:
            for unit in (0, 1):
                f = getattr(L, f"hpb_csr_trsv_{t}")
                ctx.check(f(ctx.h, h, unit, vd.data_ptr(), _lib.scalar(t, 1.0), bd.data_ptr(), xd.data_ptr()), "trsv")
                with np.errstate(all="ignore"):
                    want = oracle.csr_trsv(rp, ci, val, b, bool(upper), bool(unit), 1.0)
                assert np.array_equal(host(xd), want, equal_nan=True), (upper, unit)
            if not upper:
                lu = vd.clone()
                ctx.check(getattr(L, f"hpb_csr_ilu0_{t}")(ctx.h, h, lu.data_ptr()), "ilu0")
                assert np.array_equal(host(lu), oracle.csr_ilu0(rp, ci, val)[0])
        finally:
            L.hpb_csr_tri_destroy(h)
