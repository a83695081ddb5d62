"""Calls that use memory where there is some -- slot forms of a solver's
matrices, the diagonal recurrence of ILU(0), the slot form of a training system
-- when there is not: they run as they would without it.  The rest of the
device's memory is held by one allocation meanwhile."""
import ctypes as C

import numpy as np
import pytest

from gpu_utils import host
from high_precision_blas1_b200 import _lib, problems, spai

pytestmark = pytest.mark.gpu
L = _lib.lib
MB = 1 << 20
N, STEP = 1 << 22, 2048


class Scarce:
    """Within: `leave` bytes of device memory are free, nothing kept in the library's pools."""

    def __init__(self, torch, leave):
        self.torch, self.leave = torch, leave

    def __enter__(self):
        self.torch.cuda.synchronize()
        L.hpb_solver_memory_release()
        self.torch.cuda.empty_cache()
        free = self.torch.cuda.mem_get_info()[0]
        self.held = self.torch.empty(free - self.leave, dtype=self.torch.uint8, device="cuda")

    def __exit__(self, *exc):
        self.torch.cuda.synchronize()
        del self.held
        self.torch.cuda.empty_cache()
        L.hpb_solver_memory_release()


def five_point(torch):
    """A diagonally dominant five-point operator on a grid of N points, on the device."""
    i = torch.arange(N, device="cuda")
    offs = [-STEP, -1, 0, 1, STEP]
    has = torch.stack([(i + d >= 0) & (i + d < N) for d in offs], 1)
    has[:, 1] &= i % STEP != 0
    has[:, 3] &= i % STEP != STEP - 1
    cols = (i[:, None] + torch.tensor(offs, device="cuda"))[has].to(torch.int32)
    g = torch.Generator(device="cuda").manual_seed(1)
    val = -torch.rand(N, 5, generator=g, device="cuda", dtype=torch.float64)
    val[:, 2] = 6
    rp = torch.zeros(N + 1, dtype=torch.int32, device="cuda")
    rp[1:] = torch.cumsum(has.sum(1), 0).to(torch.int32)
    b = torch.rand(N, generator=g, device="cuda", dtype=torch.float64)
    out = rp, cols.contiguous(), val[has].contiguous(), b
    torch.cuda.synchronize()
    return out


def solve(torch, A, method, basis, iters):
    rp, ci, val, b = A
    x = torch.zeros_like(b)
    p = _lib.solver_params(method, basis, rel_tol=1e-30, max_iters=iters, fused=True)
    rep = _lib.hpb_solver_report()
    st = L.hpb_csr_solve_f64(C.byref(p), N, len(ci), rp.data_ptr(), ci.data_ptr(), val.data_ptr(), b.data_ptr(),
                             x.data_ptr(), C.byref(rep), None, 0)
    return st, x


# vectors each solve cannot do without; 100 MB beyond them are too few for the slots (41 bytes a row: 172 MB)
@pytest.mark.parametrize("method,basis,vectors", [("bicgstabl", 2, 8), ("gmres", 8, 11)])
def test_solve_without_memory_for_slots(gpu, method, basis, vectors):
    ctx, torch = gpu
    A = five_point(torch)
    st0, want = solve(torch, A, method, basis, 8)
    with Scarce(torch, vectors * 8 * N + 32 * MB + 100 * MB):  # x: 32 MB
        st, x = solve(torch, A, method, basis, 8)
    assert (st0, st) == (-7, -7)
    assert torch.linalg.vector_norm(x - want) <= 1e-12 * torch.linalg.vector_norm(want)


def analysis(ctx, A, upper):
    h = C.c_void_p()
    ctx.check(L.hpb_csr_tri_create(ctx.h, upper, N, len(A[1]), A[0].data_ptr(), A[1].data_ptr(), C.byref(h)), "tri_create")
    return h


def test_ilu0_without_scratch(gpu):
    """24 bytes a row (100 MB) of scratch for the recurrence, 60 MB left: the general factorisation's bits are the same."""
    ctx, torch = gpu
    A = five_point(torch)
    h = analysis(ctx, A, 0)
    want, got = A[2].clone(), A[2].clone()
    ctx.check(L.hpb_csr_ilu0_f64(ctx.h, h, want.data_ptr()), "ilu0")
    with Scarce(torch, 60 * MB):
        st = L.hpb_csr_ilu0_f64(ctx.h, h, got.data_ptr())
    L.hpb_csr_tri_destroy(h)
    assert st == 0
    assert torch.equal(got.view(torch.int64), want.view(torch.int64))


def test_analysis_after_a_solve(gpu):
    """What a solve's workspace keeps in its pool is there for an analysis when nothing else is."""
    ctx, torch = gpu
    A = five_point(torch)
    with Scarce(torch, 700 * MB):
        assert solve(torch, A, "gmres", 10, 10)[0] == -7  # its pool keeps some 420 MB or more
        h = [analysis(ctx, A, k) for k in (0, 1)]  # 58 bytes a row each: 480 MB, and 50 MB for a while
    for k in h:
        L.hpb_csr_tri_destroy(k)


def test_training_system_outside_the_slot_form(gpu):
    """It needs the general workspace; the slot form's, tried before, does not stand in its way."""
    torch = gpu[1]
    n = 64
    A = problems.diffusion3d_lognormal(n, seed=1, sigma=1.0, corr=2.0)
    rows = np.repeat(np.arange(A.n), np.diff(A.row_ptr))
    r, c, v = np.append(rows, [10, 13]), np.append(A.col_ind, [13, 10]), np.append(A.val, [0.0, 0.0])
    order = np.lexsort((c, r))
    rp = np.zeros(A.n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(r, minlength=A.n))
    D = spai.DeviceCSR(torch, problems.CSR(A.n, rp, c[order].astype(np.int32), v[order]))
    offs, dslot = spai.stencil7(n)
    want = spai.SpaiNet(offs, dslot, seed=1)
    loss, g = want.loss_grad(D, want_grad=True)
    want.close()
    net = spai.SpaiNet(offs, dslot, seed=1)
    with Scarce(torch, int(1.5 * 900 * A.n)):  # each workspace takes 800 to 900 bytes a row
        got, h = net.loss_grad(D, want_grad=True)
    net.close()
    assert np.array_equal(got, loss) and np.array_equal(h, g)
