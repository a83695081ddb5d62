"""The slot form of the device-resident solvers' matrices against their CSR
form: the same matrix is solved as it is (slots) and with explicit zeros at
enough further offsets in a few rows that it has no slot form.  A zero entry
adds 0 * x to its row's sum, which changes nothing, so for binary64 storage
every iterate has to agree to the last bit; binary32 storage too, except that
the reductions run over other grids and binary64 scalars may then differ in
their last bits: two solves that agree to 1e-4 after a few cycles."""
import ctypes as C

import numpy as np
import pytest

from gpu_utils import dev, host
from high_precision_blas1_b200 import _lib, problems

pytestmark = pytest.mark.gpu
DT = {"f32": np.float32, "f64": np.float64, "c64": np.complex64, "c128": np.complex128}


def matrix(kind, n, rng, cplx):
    """Diagonally dominant matrix with the kind's column offsets, a tenth of the off-diagonal entries missing."""
    offs = {"tri": [-1, 1], "five": [-37, -1, 1, 37], "seven": [-61, -9, -1, 1, 9, 61], "one-sided": [-40, -3, 2]}[kind]
    i = np.arange(n)
    r, c = [i], [i]
    for d in offs:
        k = (i + d >= 0) & (i + d < n) & (rng.random(n) < 0.9)
        r.append(i[k])
        c.append(i[k] + d)
    r, c = np.concatenate(r), np.concatenate(c)
    v = rng.uniform(-1, 1, len(r)) + (1j * rng.uniform(-1, 1, len(r)) if cplx else 0)
    v[:n] += 8
    return r, c, v


def csr(n, r, c, v):
    o = np.lexsort((c, r))
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(r, minlength=n))
    return problems.CSR(n, rp, c[o].astype(np.int32), v[o])


def with_zeros(n, r, c, v):
    """Explicit zeros on up to twelve further offsets, one row each."""
    have = set((c - r).tolist())
    er, ec = [], []
    for d in range(2, n):
        if len(er) == 12:
            break
        if d not in have:
            er.append(len(er) % max(1, n - d))
            ec.append(er[-1] + d)
    return csr(n, np.append(r, er).astype(int), np.append(c, ec).astype(int), np.append(v, np.zeros(len(er))))


def solve(torch, A, b, t, l, jacobi, iters, gmres=False):
    val = A.val.astype(DT[t])
    d = [dev(torch, a) for a in (A.row_ptr, A.col_ind, val, b.astype(DT[t]), np.zeros(A.n, DT[t]))]
    p = _lib.solver_params("gmres" if gmres else "bicgstabl", l, rel_tol=1e-30, max_iters=iters,
                           precond="jacobi" if jacobi else "none", fused=True)
    rep = _lib.hpb_solver_report()
    st = getattr(_lib.lib, f"hpb_csr_solve_{t}")(C.byref(p), A.n, A.nnz, *[x.data_ptr() for x in d], C.byref(rep), None, 0)
    assert st in (0, -7, -5), st
    return host(d[4])


def compare(torch, kind, n, t, l, jacobi, iters, gmres=False):
    rng = np.random.default_rng(n + l)
    cplx = t in ("c64", "c128")
    r, c, v = matrix(kind, n, rng, cplx)
    b = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cplx else 0)
    x = solve(torch, csr(n, r, c, v), b, t, l, jacobi, iters, gmres)
    y = solve(torch, with_zeros(n, r, c, v), b, t, l, jacobi, iters, gmres)
    if t in ("f64", "c128") and not gmres:
        # (the inner products over the two kernels' grids may round differently once in a great while)
        assert np.linalg.norm(x - y) <= 1e-13 * np.linalg.norm(y)
        assert np.mean(x == y) > 0.99
    else:
        assert np.linalg.norm(x - y) <= (1e-4 if t in ("f32", "c64") else 1e-10) * np.linalg.norm(y)


@pytest.mark.parametrize("t", ["f64", "f32", "c128", "c64"])
@pytest.mark.parametrize("kind,n,l,jacobi", [("five", 255, 1, False), ("five", 4097, 2, True), ("seven", 257, 4, False),
                                             ("seven", 9000, 2, False), ("one-sided", 5000, 4, True), ("tri", 3001, 3, False)])
def test_bicgstabl_slots(gpu, kind, n, l, jacobi, t):
    compare(gpu[1], kind, n, t, l, jacobi, 2 * l)


@pytest.mark.parametrize("kind", ["unsorted", "sparse fill", "eight offsets", "repeated column"])
def test_matrices_without_a_slot_form(gpu, kind):
    """Outside the rule: the CSR kernels solve them as before."""
    ctx, torch = gpu
    rng = np.random.default_rng(3)
    n = 3000
    r, c, v = matrix("five", n, rng, False)
    if kind == "sparse fill":  # five more offsets with few entries would leave most slots empty
        keep = (rng.random(len(r)) < 0.4) | (r == c)
        r, c, v = r[keep], c[keep], v[keep]
    elif kind == "eight offsets":
        i = np.arange(0, n - 300)
        for d in (100, 200, 300):
            r, c, v = np.append(r, i), np.append(c, i + d), np.append(v, 0.1 * rng.standard_normal(len(i)))
    elif kind == "repeated column":
        r, c, v = np.append(r, [5]), np.append(c, [5]), np.append(v, [1.0])
    A = csr(n, r, c, v)
    if kind == "unsorted":
        for k in range(n):  # each row backwards
            s = slice(A.row_ptr[k], A.row_ptr[k + 1])
            A.col_ind[s], A.val[s] = A.col_ind[s][::-1].copy(), A.val[s][::-1].copy()
    b = rng.standard_normal(n)
    x = solve(torch, A, b, "f64", 2, False, 60)
    dense = np.zeros((n, n))
    np.add.at(dense, (np.repeat(np.arange(n), np.diff(A.row_ptr)), A.col_ind), A.val)
    assert np.linalg.norm(dense @ x - b) <= 1e-9 * np.linalg.norm(b)


@pytest.mark.parametrize("t", ["f64", "f32", "c128", "c64"])
@pytest.mark.parametrize("kind,n,m,jacobi", [("five", 255, 3, False), ("seven", 9000, 10, False), ("one-sided", 5000, 8, True),
                                             ("tri", 3001, 5, True)])
def test_gmres_slots(gpu, kind, n, m, jacobi, t):
    compare(gpu[1], kind, n, t, m, jacobi, 2 * m, gmres=True)


@pytest.mark.parametrize("packs", [1, 2, 4, 7, 9])
def test_gmres_binary32_reduction(gpu, packs):
    """One cycle of binary32 GMRES against binary64 GMRES with `packs` packs a
    thread (more than the kernel takes at once for 9), the last pass ragged.
    Binary32 rounding moves a few steps on a matrix of condition below 2 by
    some 1e-6; an inner product without its last block moves them by 1e-3."""
    ctx, torch = gpu
    wave = 256 * 2 * torch.cuda.get_device_properties(0).multi_processor_count
    n = 4 * (wave * (packs - 1) + 5)
    rng = np.random.default_rng(packs)
    A = csr(n, *matrix("tri", n, rng, False))
    A.val = A.val.astype(np.float32).astype(np.float64)
    b = rng.standard_normal(n).astype(np.float32).astype(np.float64)
    x, y = (solve(torch, A, b, t, 4, False, 4, gmres=True) for t in ("f32", "f64"))
    assert np.linalg.norm(x - y) <= 1e-4 * np.linalg.norm(y)
