"""The learned SPAI's slot form against its CSR path and the binary64 oracle:
the stencils it has kernels for, a general slot count, rows around a block and
a tile, zero to four samples; and systems that it must leave to the CSR path
(an entry outside the slots, an entry twice, five samples), where the results
have to be the CSR path's.  Tolerances as in test_spai_gpu.py: M 1e-4 of its
largest entry, losses 1e-4, gradient 2e-3 (binary32 kernels)."""
import numpy as np
import pytest

from gpu_utils import host
from high_precision_blas1_b200 import problems, spai

pytestmark = pytest.mark.gpu


def box(nx, ny, nz, seed, dims=3):
    """Diffusion on a box by the repository's family, cut from a cube, with its offsets."""
    N = max(nx, ny, nz)
    A = problems.diffusion3d_lognormal(N, seed=seed, sigma=1.0, corr=2.0)
    i = np.arange(A.n)
    x, y, z = i % N, (i // N) % N, i // (N * N)
    keep = (x < nx) & (y < ny) & (z < nz)
    new = np.cumsum(keep) - 1
    rows = np.repeat(i, np.diff(A.row_ptr))
    use = keep[rows] & keep[A.col_ind]
    r, c, v = new[rows[use]], new[A.col_ind[use]], A.val[use]
    n = int(keep.sum())
    rp = np.zeros(n + 1, np.int32)
    rp[1:] = np.cumsum(np.bincount(r, minlength=n))
    offs = [-nx * ny, -nx, -1, 0, 1, nx, nx * ny] if dims == 3 else [-nx, -1, 0, 1, nx]
    if dims == 1:
        offs = [-1, 0, 1]
    return problems.CSR(n, rp, c.astype(np.int32), v), offs


def check(torch, A, offs, nres, seed):
    from oracle import spai_ref
    rng = np.random.default_rng(seed)
    net = spai.SpaiNet(offs, offs.index(0), seed=1)
    w = (rng.standard_normal(spai.NUM_PARAMS) * 0.2).astype(np.float32)
    net.set_weights(w)
    D = spai.DeviceCSR(torch, A)
    res = rng.standard_normal((nres, A.n)).astype(np.float32)
    if nres:
        D.res, D.nres = torch.from_numpy(res).cuda(), nres
    m = host(net.assemble(torch, D)).astype(np.float64)
    X, diag = spai_ref.features(A, offs, offs.index(0))
    _, _, out = spai_ref.forward(w, X)
    want = spai_ref.assemble(A, offs, offs.index(0), out, diag)
    assert np.max(np.abs(m - want)) <= 1e-4 * np.max(np.abs(want))
    loss, g = net.loss_grad(D, 1.0, 0.5, want_grad=True)
    only = net.loss(D, 1.0, 0.5)
    _, lf, lr, gref = spai_ref.loss_and_grad(A, offs, offs.index(0), w, list(res), 1.0, 0.5)
    assert loss[1] == pytest.approx(lf, rel=1e-4) and loss[2] == pytest.approx(lr, rel=1e-4, abs=1e-12)
    assert np.allclose(only, loss, rtol=1e-12)
    assert np.linalg.norm(g - gref) <= 2e-3 * np.linalg.norm(gref)
    net.close()
    return loss, g


@pytest.mark.parametrize("shape,nres", [((6, 6, 6), 0), ((7, 6, 9), 1), ((8, 8, 2), 3), ((12, 11, 10), 4)])
def test_slots_7(gpu, shape, nres):
    A, offs = box(*shape, seed=3)
    check(gpu[1], A, offs, nres, 5)


@pytest.mark.parametrize("dims,shape", [(2, (9, 15, 1)), (1, (127, 1, 1)), (1, (129, 1, 1))])
def test_other_stencils(gpu, dims, shape):
    if dims == 1:  # a tridiagonal system: three slots
        n = shape[0]
        rows = [[c for c in (r - 1, r, r + 1) if 0 <= c < n] for r in range(n)]
        rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
        ci = np.concatenate(rows).astype(np.int32)
        d = 2.0 + 0.1 * np.sin(np.arange(n))
        val = np.where(ci == np.repeat(np.arange(n), np.diff(rp)), d[np.repeat(np.arange(n), np.diff(rp))], -0.9)
        A, offs = problems.CSR(n, rp, ci, val), [-1, 0, 1]
    else:
        A, offs = box(*shape, seed=4, dims=dims)
    check(gpu[1], A, offs, 2, 6)


@pytest.mark.parametrize("kind", ["outside", "five samples"])
def test_left_to_the_csr_path(gpu, kind):
    A, offs = box(7, 7, 7, seed=9)
    nres = 5 if kind == "five samples" else 2
    if kind == "outside":  # one symmetric pair of entries at an offset that is no slot
        rows = np.repeat(np.arange(A.n), np.diff(A.row_ptr))
        r = np.append(rows, [10, 13])
        c = np.append(A.col_ind, [13, 10])
        v = np.append(A.val, [0.0, 0.0])
        order = np.lexsort((c, r))
        rp = np.zeros(A.n + 1, np.int32)
        rp[1:] = np.cumsum(np.bincount(r, minlength=A.n))
        A = problems.CSR(A.n, rp, c[order].astype(np.int32), v[order])
    check(gpu[1], A, offs, nres, 7)
