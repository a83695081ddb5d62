"""The triangular solve's chunks of 32 positions and its prepared division,
bit for bit against the CPU restatement: lengths around a chunk, a round of
the block's 15 warps and a tile, levels narrower and wider than a chunk, and
diagonals and right-hand sides inside and outside the exponents for which the
division is prepared (the plain division takes the others)."""
import ctypes as C

import numpy as np
import pytest

import oracle
from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib, problems

pytestmark = pytest.mark.gpu
DT = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}


def lower_upper(n, reach, rng):
    """Square pattern with up to two entries each side of the diagonal, at most `reach` away."""
    rows = [np.arange(n)]
    cols = [np.arange(n)]
    for d in (reach, max(1, reach // 3)):
        if d < n:
            i = np.arange(d, n)
            keep = rng.random(n - d) < 0.9
            rows += [i[keep], i[keep] - d]
            cols += [i[keep] - d, i[keep]]
    key = np.unique(np.concatenate(rows).astype(np.int64) * n + np.concatenate(cols))
    r, c = key // n, key % n
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(r, minlength=n))
    return problems.CSR(n, rp, c.astype(np.int32), np.zeros(len(c))), r == c


@pytest.mark.parametrize("t", ["f64", "f32", "c128", "c64"])
@pytest.mark.parametrize("n,reach", [(1, 1), (31, 1), (33, 1), (481, 1), (700, 31), (700, 33), (8193, 40), (16385, 97)])
def test_trsv_chunks_and_division(gpu, n, reach, t):
    ctx, torch = gpu
    rng = np.random.default_rng(n + reach)
    A, diag = lower_upper(n, reach, rng)
    val = rng.uniform(-0.3, 0.3, A.nnz)
    wide = 110 if t in ("f64", "c128") else 34
    if t in ("c64", "c128"):  # |d|^2 is the divisor: half the exponent
        wide //= 2
        val = val + 1j * rng.uniform(-0.3, 0.3, A.nnz)
    # a tenth of the diagonal well outside the prepared range, on both sides
    e = np.where(rng.random(A.nnz) < 0.1, rng.choice([-wide, wide], A.nnz), rng.integers(-2, 3, A.nnz))
    val = np.where(diag, (1.0 + val) * 2.0 ** e, val).astype(DT[t])
    b = rng.standard_normal(n) * np.where(rng.random(n) < 0.1, 0.0, 1.0)
    b = (b + 1j * rng.standard_normal(n) if t in ("c64", "c128") else b).astype(DT[t])
    rp, ci, vd, bd = (dev(torch, a) for a in (A.row_ptr, A.col_ind, val, b))
    xd = torch.zeros_like(bd)
    for upper in (0, 1):
        h = C.c_void_p()
        ctx.check(_lib.lib.hpb_csr_tri_create(ctx.h, upper, n, A.nnz, rp.data_ptr(), ci.data_ptr(), C.byref(h)), "create")
        try:
            for unit in (0, 1):
                f = getattr(_lib.lib, f"hpb_csr_trsv_{t}")
                ctx.check(f(ctx.h, h, unit, vd.data_ptr(), _lib.scalar(t, 1.0), bd.data_ptr(), xd.data_ptr()), "trsv")
                with np.errstate(all="ignore"):
                    want = oracle.csr_trsv(A.row_ptr, A.col_ind, val, b, bool(upper), bool(unit), 1.0)
                got = host(xd)
                assert np.array_equal(got, want, equal_nan=True), (upper, unit)
        finally:
            _lib.lib.hpb_csr_tri_destroy(h)
