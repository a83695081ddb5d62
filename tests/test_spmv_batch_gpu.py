"""SpMV rows around the batch of entries whose loads are issued together: row
lengths 0 to 16 in every order, and a matrix well above L2 on both sides of
the rule that keeps the plain loop.  Small integers: every result is exact."""
import numpy as np
import pytest

from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib

pytestmark = pytest.mark.gpu
DT = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}


def ints(rng, n, t):
    return (rng.integers(-3, 4, n) + (1j * rng.integers(-3, 4, n) if t[0] == "c" else 0)).astype(DT[t])


def run(ctx, torch, t, rows, cols, rp, ci, val, x, y, alpha, beta):
    d = [dev(torch, a) for a in (rp, ci, val, x, y)]
    ctx.check(getattr(_lib.lib, f"hpb_csr_spmv_{t}")(
        ctx.h, rows, cols, len(val), d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), _lib.scalar(t, alpha),
        d[3].data_ptr(), _lib.scalar(t, beta), d[4].data_ptr()), "spmv")
    torch.cuda.synchronize()
    return host(d[4])


@pytest.mark.parametrize("t", ["f32", "f64", "c64", "c128"])
@pytest.mark.parametrize("rows", [1, 255, 257, 5000])
@pytest.mark.parametrize("beta", [0.0, -2.0])
def test_row_lengths(gpu, t, rows, beta):
    ctx, torch = gpu
    rng = np.random.default_rng(rows)
    ln = rng.integers(0, 17, rows)
    rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
    cols = 700
    ci = rng.integers(0, cols, rp[-1]).astype(np.int32)
    val, x, y = ints(rng, rp[-1], t), ints(rng, cols, t), ints(rng, rows, t)
    want = np.zeros(rows, complex)
    np.add.at(want, np.repeat(np.arange(rows), ln), (val * x[ci]).astype(complex))
    got = run(ctx, torch, t, rows, cols, rp, ci, val, x, y, 3.0, beta)
    assert np.array_equal(got.astype(complex), 3 * want + beta * y)


@pytest.mark.parametrize("per_row", [5, 6])
def test_above_l2(gpu, per_row):
    ctx, torch = gpu
    l2 = torch.cuda.get_device_properties(0).L2_cache_size
    rows = int(1.5 * l2) // (per_row * 12) + 1001
    rng = np.random.default_rng(per_row)
    rp = np.arange(0, per_row * rows + 1, per_row).astype(np.int32)
    ci = ((np.arange(rows)[:, None] + np.arange(per_row) * 37) % rows).astype(np.int32)
    val, x, y = ints(rng, per_row * rows, "f64"), ints(rng, rows, "f64"), ints(rng, rows, "f64")
    got = run(ctx, torch, "f64", rows, rows, rp, ci.ravel(), val, x, y, 1.0, 0.0)
    assert np.array_equal(got, (val.reshape(rows, per_row) * x[ci]).sum(1))
