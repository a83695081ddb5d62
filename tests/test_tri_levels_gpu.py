"""The analysis' level schedule at its edges -- rows without dependencies, long
chains, rows with more than four dependents in the tile (the general list) and
tiles with too many dependencies for it (the sweeps), several tiles -- by the
levels it reports and by the solve that runs on it, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import oracle
from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib

pytestmark = pytest.mark.gpu
TILE = 8192


def pattern(kind, n, rng):
    """(row_ptr, col_ind) of a symmetric pattern with its diagonal."""
    if kind == "diagonal":
        lower = []
    elif kind == "chain":
        lower = [(np.arange(1, n), np.arange(n - 1))]
    elif kind == "fan":  # every row depends on the last multiple of 50 before it
        i = np.arange(1, n)
        lower = [(i, (i - 1) // 50 * 50)]
    elif kind == "band":  # 9 dependencies a row: past the general list's room in a full tile
        lower = [(np.arange(d, n), np.arange(n - d)) for d in range(1, 10)]
    else:  # shuffled long and short reaches
        lower = [(np.arange(d, n), np.arange(n - d)) for d in (7, 1000, 9001) if d < n]
        lower = [(i[k], j[k]) for i, j in lower for k in [rng.random(len(i)) < 0.8]]
    r = np.concatenate([np.arange(n)] + [x for i, j in lower for x in (i, j)])
    c = np.concatenate([np.arange(n)] + [x for i, j in lower for x in (j, i)])
    key = np.unique(r.astype(np.int64) * n + c)
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(key // n, minlength=n))
    return rp, (key % n).astype(np.int32)


def levels(rp, ci, upper):
    n = len(rp) - 1
    lev = [0] * n
    for i in (range(n - 1, -1, -1) if upper else range(n)):
        deps = [c for c in ci[rp[i]:rp[i + 1]] if (c > i if upper else c < i)]
        lev[i] = max((lev[c] + 1 for c in deps), default=0)
    return np.array(lev)


@pytest.mark.parametrize("kind", ["diagonal", "chain", "fan", "band", "mixed"])
@pytest.mark.parametrize("n", [1, 1000, TILE, 2 * TILE + 37])
def test_levels(gpu, kind, n):
    ctx, torch = gpu
    rng = np.random.default_rng(n)
    rp, ci = pattern(kind, n, rng)
    rows = np.repeat(np.arange(n), np.diff(rp))
    val = np.where(ci == rows, 2.0 + rng.random(len(ci)), rng.uniform(-0.1, 0.1, len(ci)))
    b = rng.standard_normal(n)
    rpd, cid, vd, bd = (dev(torch, a) for a in (rp, ci, val, b))
    xd = torch.zeros_like(bd)
    for upper in (0, 1):
        h = C.c_void_p()
        ctx.check(_lib.lib.hpb_csr_tri_create(ctx.h, upper, n, len(ci), rpd.data_ptr(), cid.data_ptr(), C.byref(h)),
                  "create")
        try:
            lev = levels(rp, ci, upper)
            per_tile = [len(np.unique(lev[t:t + TILE])) for t in range(0, n, TILE)]
            t, m, s, d = C.c_int32(), C.c_int32(), C.c_int64(), C.c_int()
            assert _lib.lib.hpb_csr_tri_info(h, C.byref(t), C.byref(m), C.byref(s), C.byref(d)) == 0
            assert (t.value, m.value, s.value, d.value) == (len(per_tile), max(per_tile), sum(per_tile), 1)
            ctx.check(_lib.lib.hpb_csr_trsv_f64(ctx.h, h, 0, vd.data_ptr(), 1.0, bd.data_ptr(), xd.data_ptr()), "trsv")
            ctx.check(_lib.lib.hpb_csr_tri_check(ctx.h, h), "check")
            assert np.array_equal(host(xd), oracle.csr_trsv(rp, ci, val, b, bool(upper), False, 1.0))
        finally:
            _lib.lib.hpb_csr_tri_destroy(h)
