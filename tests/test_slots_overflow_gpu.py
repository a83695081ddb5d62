"""Binary32 solves that leave binary32's range: with the matrix in slot form
(operands rounded in binary64) they end as with it in CSR form -- the same
status, and a solution that is not finite or is the same."""
import ctypes as C

import numpy as np
import pytest

from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib
from test_slots_forms_gpu import has_slots, matrix
from test_slots_gpu import DT, csr, with_zeros

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", ["f32", "c64"])
@pytest.mark.parametrize("scale", [1e30, 1e36, 3e37])
@pytest.mark.parametrize("l", [1, 2])
def test_divergence(gpu, t, scale, l):
    torch = gpu[1]
    rng = np.random.default_rng(l)
    n, cplx = 1500, t == "c64"
    r, c, v = matrix("five", n, rng, cplx)
    b = (rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)) * 1e3
    ends = []
    for A in (csr(n, r, c, v), with_zeros(n, r, c, v)):
        assert has_slots(A) == (not ends)
        d = [dev(torch, a) for a in (A.row_ptr, A.col_ind, (A.val * scale).astype(DT[t]), b.astype(DT[t]), np.zeros(n, DT[t]))]
        p = _lib.solver_params("bicgstabl", l, rel_tol=1e-6, max_iters=40, fused=True)
        rep = _lib.hpb_solver_report()
        st = getattr(_lib.lib, f"hpb_csr_solve_{t}")(C.byref(p), n, A.nnz, *[x.data_ptr() for x in d], C.byref(rep), None, 0)
        ends.append((st, host(d[4])))
    (s0, x0), (s1, x1) = ends
    assert s0 == s1
    assert np.all(np.isfinite(x0)) == np.all(np.isfinite(x1))
    if np.all(np.isfinite(x1)):
        assert np.linalg.norm((x0 - x1) * scale) <= 1e-3 * np.linalg.norm(x1 * scale)
