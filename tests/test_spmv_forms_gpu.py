"""Both sides of the mean row lengths at which the SpMV changes its form (three
and eight entries), in every type, with and without beta, on rows around a
block and more than the grid takes at once, and from unaligned arrays.  Small
integers: every result is exact."""
import numpy as np
import pytest

from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib

pytestmark = pytest.mark.gpu
DT = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}


def ints(rng, n, t):
    return (rng.integers(-3, 4, n) + (1j * rng.integers(-3, 4, n) if t[0] == "c" else 0)).astype(DT[t])


@pytest.mark.parametrize("t", ["f32", "f64", "c64", "c128"])
@pytest.mark.parametrize("per_row", [1, 3, 4, 8, 9, 27])
@pytest.mark.parametrize("rows,shift", [(3, 0), (255, 0), (700001, 0), (5001, 1)])
def test_forms(gpu, t, per_row, rows, shift):
    ctx, torch = gpu
    rng = np.random.default_rng(per_row)
    # the last row is one entry longer: the mean lies just above per_row, the lengths differ
    ln = np.full(rows, per_row)
    ln[rng.permutation(rows)[: rows // 3]] += 1
    ln[rng.permutation(np.nonzero(ln == per_row)[0])[: rows // 3]] -= 1
    for extra in (0, 1):
        ln[-1] += extra
        rp = np.concatenate([[0], np.cumsum(ln)]).astype(np.int32)
        ci = rng.integers(0, rows, rp[-1]).astype(np.int32)
        val, x, y = ints(rng, rp[-1] + shift, t), ints(rng, rows + shift, t), ints(rng, rows + shift, t)
        d = [dev(torch, a) for a in (rp, ci, val, x)]
        size = np.dtype(DT[t]).itemsize // (2 if t[0] == "c" else 1) * shift
        if shift and t[0] == "c":  # half an element past the pair's boundary
            val, x = (a.view(a.real.dtype)[1:-1].view(a.dtype) for a in (val, x))
        elif shift:
            val, x = val[1:], x[1:]
        want = np.zeros(rows, complex)
        np.add.at(want, np.repeat(np.arange(rows), ln), (val[: rp[-1]] * x[ci]).astype(complex))
        for beta in (0.0, -2.0):
            dy = dev(torch, y)
            ctx.check(getattr(_lib.lib, f"hpb_csr_spmv_{t}")(
                ctx.h, rows, rows, int(rp[-1]), d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr() + size,
                _lib.scalar(t, 3.0), d[3].data_ptr() + size, _lib.scalar(t, beta), dy.data_ptr()), "spmv")
            torch.cuda.synchronize()
            assert np.array_equal(host(dy)[:rows].astype(complex), 3 * want + beta * y[:rows])
