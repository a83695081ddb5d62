"""Solves on matrices that do have a slot form -- four offsets (held as five),
five, six (the last of seven never loaded) and seven -- against the same
matrices with explicit zeros that take it from them (test_slots_gpu.py, whose
tolerances hold here too), and a refined GMRES whose CSR preconditioner is in
slot form, with A's own structure and with another."""
import ctypes as C

import numpy as np
import pytest

from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib
from test_slots_gpu import csr, solve, with_zeros

pytestmark = pytest.mark.gpu
OFFSETS = {"four": ([-40, -3, 2], 1.0), "five": ([-37, -1, 1, 37], 0.9), "six": ([-61, -9, -1, 1, 61], 0.95),
           "seven": ([-61, -9, -1, 1, 9, 61], 0.9)}


def matrix(kind, n, rng, cplx):
    offs, fill = OFFSETS[kind]
    i = np.arange(n)
    r, c = [i], [i]
    for d in offs:
        k = (i + d >= 0) & (i + d < n) & (rng.random(n) < fill)
        r.append(i[k])
        c.append(i[k] + d)
    r, c = np.concatenate(r), np.concatenate(c)
    v = rng.uniform(-1, 1, len(r)) + (1j * rng.uniform(-1, 1, len(r)) if cplx else 0)
    v[:n] += 8
    return r, c, v


def has_slots(A):
    """The rule of csrc/hpb_slots.cuh."""
    rows = np.repeat(np.arange(A.n), np.diff(A.row_ptr))
    ns = len(np.unique(A.col_ind - rows))
    return ns <= 7 and max(ns, 5) * A.n <= A.nnz + A.nnz // 3


@pytest.mark.parametrize("t", ["f64", "f32", "c128", "c64"])
@pytest.mark.parametrize("kind,n,l,jacobi", [("four", 5000, 4, True), ("four", 769, 1, False), ("six", 4099, 2, True),
                                             ("six", 257, 3, False), ("five", 3001, 2, True), ("seven", 2000, 1, True)])
@pytest.mark.parametrize("gmres", [False, True])
def test_solves(gpu, kind, n, l, jacobi, t, gmres):
    torch = gpu[1]
    rng = np.random.default_rng(n + l)
    cplx = t in ("c64", "c128")
    r, c, v = matrix(kind, n, rng, cplx)
    b = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)
    A, B = csr(n, r, c, v), with_zeros(n, r, c, v)
    assert has_slots(A) and not has_slots(B)
    m = 3 * l if gmres else l
    x, y = (solve(torch, M, b, t, m, jacobi, 2 * m, gmres) for M in (A, B))
    if t in ("f64", "c128") and not gmres:
        assert np.linalg.norm(x - y) <= 1e-13 * np.linalg.norm(y)
        assert np.mean(x == y) > 0.99
    else:
        assert np.linalg.norm(x - y) <= (1e-4 if t in ("f32", "c64") else 1e-10) * np.linalg.norm(y)


@pytest.mark.parametrize("structure", ["A's", "its own"])
@pytest.mark.parametrize("t", ["f64", "c128"])
def test_preconditioner_in_slot_form(gpu, structure, t):
    torch = gpu[1]
    n, rng, cplx = 4001, np.random.default_rng(5), t == "c128"
    A = csr(n, *matrix("seven", n, rng, cplx))
    if structure == "A's":
        M = csr(n, *matrix("seven", n, np.random.default_rng(5), cplx))
        assert np.array_equal(M.col_ind, A.col_ind)
    else:
        M = csr(n, *matrix("four", n, rng, cplx))
    r, c = np.repeat(np.arange(n), np.diff(M.row_ptr)), M.col_ind
    v = np.where(r == c, 1 / 8, -0.1 * M.val / 64)
    M, Z = csr(n, r, c, v), with_zeros(n, r, c, v)
    assert has_slots(A) and has_slots(M) and not has_slots(Z)
    dt, lo = (np.complex128, np.complex64) if cplx else (np.float64, np.float32)
    b = dev(torch, (rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)).astype(dt))
    a = [dev(torch, w) for w in (A.row_ptr, A.col_ind, A.val.astype(dt))]

    def run(P, like):
        m = [dev(torch, w) for w in (P.row_ptr, P.col_ind, P.val.astype(lo))]
        rp, ci = (a[0], a[1]) if like else (m[0], m[1])
        x = torch.zeros_like(b)
        p = _lib.ir_params("gmres", 6, inner_rel_tol=0.0, inner_max_iters=0, rel_tol=1e-30, max_refinements=3,
                           precond="matrix")
        rep = _lib.hpb_ir_report()
        st = getattr(_lib.lib, f"hpb_ir_solve_{t}")(
            C.byref(p), n, A.nnz, *[w.data_ptr() for w in a], None, rp.data_ptr(), ci.data_ptr(), m[2].data_ptr(),
            P.nnz, b.data_ptr(), x.data_ptr(), C.byref(rep), None, 0)
        assert st in (0, -7), st
        return host(x)

    # the product's operations and their order are the CSR kernel's: the same bits
    assert np.array_equal(run(M, structure == "A's"), run(Z, False))
