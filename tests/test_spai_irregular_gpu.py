"""Systems that hold nothing outside the slots and still have no slot form: a
row whose entries run backwards, a row that holds an entry twice."""
import numpy as np
import pytest

from gpu_utils import host
from high_precision_blas1_b200 import problems, spai
from test_spai_slots_gpu import box, check

pytestmark = pytest.mark.gpu


def test_backward_rows(gpu):
    A, offs = box(7, 6, 8, seed=9)
    ci, val = A.col_ind.copy(), A.val.copy()
    for r in (0, 100, A.n - 1):
        s = slice(A.row_ptr[r], A.row_ptr[r + 1])
        ci[s], val[s] = ci[s][::-1].copy(), val[s][::-1].copy()
    check(gpu[1], problems.CSR(A.n, A.row_ptr, ci, val), offs, 2, 7)


def test_entry_twice(gpu):
    """M as without the second entry, but for that row's diagonal, which sums over the row's entries."""
    torch = gpu[1]
    A, offs = box(7, 6, 8, seed=9)
    row = 100
    at = A.row_ptr[row]
    rp = A.row_ptr.copy()
    rp[row + 1:] += 1
    B = problems.CSR(A.n, rp, np.insert(A.col_ind, at, A.col_ind[at]), np.insert(A.val, at, A.val[at]))
    net = spai.SpaiNet(offs, offs.index(0), seed=1)
    net.set_weights((np.random.default_rng(3).standard_normal(spai.NUM_PARAMS) * 0.2).astype(np.float32))
    m, n = (host(net.assemble(torch, spai.DeviceCSR(torch, s))).astype(np.float64) for s in (A, B))
    net.close()
    assert n[at] == n[at + 1]
    n = np.delete(n, at)
    keep = np.ones(A.nnz, bool)
    keep[A.row_ptr[row]:A.row_ptr[row + 1]] &= A.col_ind[A.row_ptr[row]:A.row_ptr[row + 1]] != row
    assert np.max(np.abs(m - n)[keep]) <= 1e-4 * np.max(np.abs(m))
