"""ILU(0) by the diagonal recurrence and by the general kernel, bit for bit
against the CPU restatement, on patterns on both sides of the rule between
them: no triangle in the graph (a grid, with entries missing on one side of
the diagonal), one triangle among a million, rows with more than four
dependencies; a zero pivot and a non-finite one."""
import ctypes as C

import numpy as np
import pytest

import oracle
from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib, problems

pytestmark = pytest.mark.gpu
DT = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}


def csr(n, pairs):
    key = np.unique(np.concatenate([np.asarray(r, np.int64) * n + np.asarray(c, np.int64) for r, c in pairs]))
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return rp, (key % n).astype(np.int32)


def pattern(kind, rng):
    nx, n = 131, 131 * 127  # two tiles and a part
    i = np.arange(n)
    pairs = [(i, i)]
    for d in (1, nx):
        a = i[d:] if d > 1 else i[(i % nx) > 0]
        pairs += [(a, a - d), (a - d, a)]
    if kind == "one-sided":  # a third of the upper entries missing: no a_ki there
        pairs = [pairs[0]] + [(r[k], c[k]) for r, c in pairs[1:] for k in [(r > c) | (rng.random(len(r)) < 0.66)]]
    elif kind == "one-triangle":
        pairs += [([9000 + nx], [9001]), ([9001], [9000 + nx])]
    elif kind == "wide":  # five dependencies, no triangle among them
        pairs = [(i, i)] + [(i[d:], i[d:] - d) for d in (1, 10, 100, 1000, 5000)]
    return n, csr(n, pairs)


def factor(ctx, torch, t, n, rp, ci, val):
    rpd, cid, lu = dev(torch, rp), dev(torch, ci), dev(torch, val)
    h = C.c_void_p()
    ctx.check(_lib.lib.hpb_csr_tri_create(ctx.h, 0, n, len(ci), rpd.data_ptr(), cid.data_ptr(), C.byref(h)), "create")
    try:
        st = getattr(_lib.lib, f"hpb_csr_ilu0_{t}")(ctx.h, h, lu.data_ptr())
        torch.cuda.synchronize()
        return st, host(lu)
    finally:
        _lib.lib.hpb_csr_tri_destroy(h)


@pytest.mark.parametrize("t", ["f64", "f32", "c128", "c64"])
@pytest.mark.parametrize("kind", ["grid", "one-sided", "one-triangle", "wide"])
def test_ilu0_kinds(gpu, kind, t):
    ctx, torch = gpu
    rng = np.random.default_rng(5)
    n, (rp, ci) = pattern(kind, rng)
    on = ci == np.repeat(np.arange(n), np.diff(rp))
    val = rng.uniform(-1, 1, len(ci)) + (1j * rng.uniform(-1, 1, len(ci)) if t in ("c64", "c128") else 0)
    val = np.where(on, 6.0 + val, val).astype(DT[t])
    st, got = factor(ctx, torch, t, n, rp, ci, val)
    want, zero_row = oracle.csr_ilu0(rp, ci, val)
    assert st == 0 and zero_row == -1
    assert np.array_equal(got, want)


@pytest.mark.parametrize("bad", [0.0, np.nan, np.inf])
def test_ilu0_bad_pivot(gpu, bad):
    """A zero pivot (row 40 of zeros) is reported with its row; others go through."""
    ctx, torch = gpu
    A = problems.convdiff2d(64)
    val = A.val.copy()
    rows = np.repeat(np.arange(A.n), np.diff(A.row_ptr))
    if bad == 0.0:
        val[rows == 40] = 0.0
    else:
        val[(rows == 40) & (A.col_ind == 40)] = bad
    st, got = factor(ctx, torch, "f64", A.n, A.row_ptr, A.col_ind, val)
    with np.errstate(all="ignore"):
        want, _ = oracle.csr_ilu0(A.row_ptr, A.col_ind, val)
    if bad == 0.0:
        assert st == -5 and "row 40" in _lib.lib.hpb_last_error(ctx.h).decode()
    else:
        assert st == 0
        assert np.array_equal(got, want, equal_nan=True)
