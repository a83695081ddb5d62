"""Threads that build preconditioners with one network at the same time, some
of them for systems that the slot form does not take: each build gives what it
gives alone."""
import threading

import numpy as np
import pytest

from gpu_utils import host
from high_precision_blas1_b200 import problems, spai

pytestmark = pytest.mark.gpu


def outside(A):
    """A with one symmetric pair of zero entries at an offset that is no slot."""
    rows = np.repeat(np.arange(A.n), np.diff(A.row_ptr))
    r, c, v = np.append(rows, [10, 13]), np.append(A.col_ind, [13, 10]), np.append(A.val, [0.0, 0.0])
    order = np.lexsort((c, r))
    rp = np.zeros(A.n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(r, minlength=A.n))
    return problems.CSR(A.n, rp, c[order].astype(np.int32), v[order])


def test_builds_side_by_side(gpu):
    torch = gpu[1]
    offs, dslot = spai.stencil7(12)
    net = spai.SpaiNet(offs, dslot, seed=1)
    net.set_weights((np.random.default_rng(0).standard_normal(spai.NUM_PARAMS) * 0.2).astype(np.float32))
    A = [problems.diffusion3d_lognormal(12, seed=s, sigma=1.0, corr=2.0) for s in range(4)]
    D = [spai.DeviceCSR(torch, outside(a) if k % 2 else a) for k, a in enumerate(A)]
    want = [host(net.assemble(torch, d)) for d in D]
    wrong = []

    def build(k):
        for _ in range(60):
            m = host(net.assemble(torch, D[k]))
            if not np.array_equal(m, want[k]):
                wrong.append(k)

    threads = [threading.Thread(target=build, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    net.close()
    assert not wrong, wrong
