"""Timed cases of the library, through its C ABI as ctypes callers use it.

Eight families, each a group of calls that programs built on the library make:

* reduce -- one compensated reduction (dot2, sum2, asum2, nrm2), its result
            left on the device or returned by value, in the four element types;
* vector -- one update of the axpy family;
* spmv   -- one CSR product y = alpha A x + beta y, or the product fused with
            the Dot2 that consumes it;
* ilu0   -- the set-up of an ILU(0) preconditioner for a new matrix: the
            analyses of both triangles and the factorisation;
* trsv   -- one application of ILU(0) factors, (L U)^-1 b, by two exact
            triangular solves on kept analyses;
* bicg   -- the device-resident BiCGStab(l) for a bounded number of iterations;
* refine -- a mixed-precision solve (binary32 inner iterations with Dot2 in a
            binary64 refinement loop) to a tight tolerance;
* spai   -- the learned sparse approximate inverse: its build for a new
            matrix, or its loss and parameter gradient on a training system.

The matrices are the 5- and 7-point grid operators of the benchmark
configurations on boxes of any side lengths, made on the GPU.
"""
import ctypes
import math

import numpy as np
import torch

from high_precision_blas1_b200 import Context, _lib, spai

L = _lib.lib
BYTES = {"f32": 4, "f64": 8, "c64": 8, "c128": 16}
TORCH = {"f32": torch.float32, "f64": torch.float64, "c64": torch.complex64, "c128": torch.complex128}
NOT_CONVERGED = -7  # a solve that ran its bounded number of iterations


def listed():
    return [
        # a scalar product returned to the host, as the drop-in's scalar_prod
        # makes between the steps of a host-driven solver: the smallest call
        dict(name="dot2_value_small", family="reduce", op="dot2", dtype="f64", n=5003, by_value=True, cond=False,
             shift=0),
        # the ill-conditioned scalar product of the benchmark, left on the device
        dict(name="dot2_f64_1m", family="reduce", op="dot2", dtype="f64", n=1048576, by_value=False, cond=True,
             shift=0),
        # a norm of a long complex vector of odd length
        dict(name="nrm2_c64_large", family="reduce", op="nrm2", dtype="c64", n=33554393, by_value=False, cond=False,
             shift=0),
        # a three-term update of long vectors of odd length
        dict(name="axpbypcz_f32_large", family="vector", op="axpbypcz", dtype="f32", n=40000003),
        # the product with the benchmark's convection-diffusion matrix
        dict(name="spmv_f64_convdiff", family="spmv", grid="convdiff", nx=1024, ny=1024, nz=1, dtype="f64",
             beta=False, dot=False),
        # a new 5-point matrix's ILU(0), as every solve with that preconditioner begins
        dict(name="ilu0_setup_convdiff", family="ilu0", grid="convdiff", nx=1024, ny=1024, nz=1, dtype="f64"),
        # one application of those factors, as in every iteration
        dict(name="trsv_ilu0_convdiff", family="trsv", grid="convdiff", nx=1024, ny=1024, nz=1, dtype="f64"),
        # the headline solver, 100 of its cycles
        dict(name="bicgstab4_convdiff", family="bicg", grid="convdiff", nx=1024, ny=1024, nz=1, dtype="f64", l=4,
             jacobi=False, iters=400),
        # the precision form: GMRES(50) on the anisotropic Poisson operator
        dict(name="gmres50_refined_poisson", family="refine", grid="poisson", nx=128, ny=128, nz=128, basis=50,
             tol=1e-11),
        # the complex precision form: BiCGStab(2) on the damped Helmholtz operator
        dict(name="bicgstab2_refined_helm", family="refine", grid="helmholtz", nx=2048, ny=2048, nz=1, basis=2,
             tol=1e-11),
        # the learned preconditioner for a new matrix
        dict(name="spai_build_96", family="spai", nx=96, ny=96, nz=96, train=False),
        # one training system's loss and gradient
        dict(name="spai_train_24", family="spai", nx=24, ny=24, nz=24, train=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["reduce", "reduce", "vector", "spmv", "ilu0", "trsv", "bicg", "refine", "spai"])
    if family == "reduce":
        op = rng.choice(["dot2", "dot2", "sum2", "asum2", "nrm2"])
        t = rng.choice(["f32", "f64", "c64", "c128"])
        # a third of them one element past a 16-byte boundary, as a slice of a longer array is
        return dict(family=family, op=op, dtype=t, n=_log(rng, 2000, 50000000), by_value=rng.random() < 0.4,
                    cond=False, shift=rng.choice([0, 0, 1]))
    if family == "vector":
        op = rng.choice(["axpy", "axpby", "axpbypcz", "axpbypcwpdz", "lincomb4", "scal", "mul_pointwise"])
        return dict(family=family, op=op, dtype=rng.choice(["f32", "f64", "c64", "c128"]),
                    n=_log(rng, 2000, 40000000))
    if family == "spmv":
        grid = rng.choice(["convdiff", "poisson", "helmholtz", "lognormal"])
        two = grid in ("convdiff", "helmholtz")
        side = (40, 2000) if two else (16, 150)
        return dict(family=family, grid=grid, nx=_log(rng, *side), ny=_log(rng, *side),
                    nz=1 if two else _log(rng, *side),
                    dtype=rng.choice(["c64", "c128"] if grid == "helmholtz" else ["f32", "f64"]),
                    beta=rng.random() < 0.3, dot=rng.random() < 0.3)
    if family in ("ilu0", "trsv"):
        grid = rng.choice(["convdiff", "poisson", "helmholtz", "lognormal"])
        two = grid in ("convdiff", "helmholtz")
        side = (40, 1000) if two else (12, 96)
        return dict(family=family, grid=grid, nx=_log(rng, *side), ny=_log(rng, *side),
                    nz=1 if two else _log(rng, *side),
                    dtype=rng.choice(["c64", "c128"] if grid == "helmholtz" else ["f32", "f64"]))
    if family == "bicg":
        grid = rng.choice(["convdiff", "poisson", "helmholtz"])
        two = grid != "poisson"
        side = (48, 1100) if two else (16, 110)
        l = rng.choice([1, 2, 4, 4])
        return dict(family=family, grid=grid, nx=_log(rng, *side), ny=_log(rng, *side),
                    nz=1 if two else _log(rng, *side), dtype="c128" if grid == "helmholtz" else "f64", l=l,
                    jacobi=rng.random() < 0.3, iters=l * rng.randint(8, 40))
    if family == "refine":
        if rng.random() < 0.5:
            return dict(family=family, grid="poisson", nx=_log(rng, 16, 112), ny=_log(rng, 16, 112),
                        nz=_log(rng, 16, 112), basis=rng.choice([30, 50]), tol=1e-11)
        return dict(family=family, grid="helmholtz", nx=_log(rng, 64, 2000), ny=_log(rng, 64, 2000), nz=1, basis=2,
                    tol=1e-11)
    train = rng.random() < 0.5
    side = (12, 36) if train else (16, 110)
    return dict(family=family, nx=_log(rng, *side), ny=_log(rng, *side), nz=_log(rng, *side), train=train)


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(n, dtype, g):
    """n entries uniform in [-1, 1] (complex: each part)."""
    r = torch.float32 if dtype in ("f32", "c64") else torch.float64
    if dtype in ("f32", "f64"):
        return torch.rand(n, generator=g, device="cuda", dtype=r) * 2 - 1
    return torch.view_as_complex(torch.rand(n, 2, generator=g, device="cuda", dtype=r) * 2 - 1)


class Grid:
    """A 5- or 7-point operator on an nx x ny x nz box (x fastest, Dirichlet
    boundaries): offs[s] the column offset of slot s, val[s][i] the entry of
    row i there, has[s][i] whether the row stores it."""

    def __init__(self, case, seed):
        nx, ny, nz = case["nx"], case["ny"], case["nz"]
        kind = case.get("grid", "lognormal")
        n = self.n = nx * ny * nz
        self.shape = (nz, ny, nx)
        dim = 3 if nz > 1 else 2
        step = [1, nx, nx * ny][:dim]
        self.offs = [-s for s in reversed(step)] + [0] + step
        self.dslot = dim
        i = torch.arange(n, device="cuda")
        at = [i % nx, (i // nx) % ny, i // (nx * ny)][:dim]
        side = [nx, ny, nz][:dim]
        ones = torch.ones(n, dtype=torch.bool, device="cuda")
        self.has = torch.stack([at[d] > 0 for d in reversed(range(dim))] + [ones]
                               + [at[d] < side[d] - 1 for d in range(dim)])
        if kind == "lognormal":
            lo, hi, diag = self._diffusion(seed)
        else:
            h = 1.0 / (max(side) + 1)
            if kind == "convdiff":  # a . grad u - lap u / Re, upwind, a = (1, 1) / sqrt 2, Re = 50, times h^2
                a, d = h / math.sqrt(2.0), 1.0 / 50.0
                lo, hi, diag = [-a - d] * dim, [-d] * dim, dim * a + 2 * dim * d
            elif kind == "poisson":
                e = [1.0, 1e-2, 1e-4][:dim]
                lo, hi, diag = [-v for v in e], [-v for v in e], 2 * sum(e)
            else:  # damped Helmholtz, ten points a wavelength
                kh = 2.0 * math.pi / 10.0
                lo, hi, diag = [-1.0] * dim, [-1.0] * dim, 2.0 * dim + complex(-kh * kh, 0.5 * kh * kh)
        self.const = None if kind == "lognormal" else (lo, hi, diag)
        t = torch.complex128 if kind == "helmholtz" else torch.float64
        self.val = torch.empty(len(self.offs), n, dtype=t, device="cuda")
        for s, v in enumerate(list(reversed(lo)) + [diag] + list(hi)):
            self.val[s] = v
        if case["family"] in ("ilu0", "trsv"):  # a reaction term that changes with the system
            self.val[dim] *= 1 + 0.1 * torch.rand(n, generator=_gen(seed + 2), device="cuda", dtype=torch.float64)
        self.val *= self.has

    def _diffusion(self, seed):
        """-div(kappa grad u): lognormal kappa of log-deviation 2.3, correlation length 8 cells."""
        g = torch.randn(self.shape, generator=_gen(seed), device="cuda", dtype=torch.float64)
        f = torch.fft.fftn(g)
        for ax, m in enumerate(self.shape):
            k = torch.fft.fftfreq(m, device="cuda", dtype=torch.float64)
            w = torch.exp(-0.5 * (2 * math.pi * k * 8.0) ** 2)
            f = f * w.reshape([-1 if j == ax else 1 for j in range(3)])
        g = torch.fft.ifftn(f).real
        kap = torch.exp((g - g.mean()) / g.std() * 2.3)
        lo, hi, diag = [], [], 0.0
        for ax in (2, 1, 0):
            m = self.shape[ax]
            a, b = kap.narrow(ax, 0, m - 1), kap.narrow(ax, 1, m - 1)
            face = 2 * a * b / (a + b)
            below = torch.cat([kap.narrow(ax, 0, 1), face], ax).reshape(-1)
            above = torch.cat([face, kap.narrow(ax, m - 1, 1)], ax).reshape(-1)
            lo.append(-below)
            hi.append(-above)
            diag = diag + below + above
        return lo, hi, diag

    def csr(self, dtype):
        """(row_ptr, col_ind, val) on the device."""
        has = self.has.t()
        rp = torch.zeros(self.n + 1, dtype=torch.int32, device="cuda")
        rp[1:] = torch.cumsum(has.sum(1), 0).to(torch.int32)
        cols = torch.arange(self.n, device="cuda", dtype=torch.int32)[:, None] \
            + torch.tensor(self.offs, device="cuda", dtype=torch.int32)[None, :]
        return rp, cols[has].contiguous(), self.val.t()[has].to(TORCH[dtype]).contiguous()

    def rounded(self, dtype):
        """The slots' values as an operator of that type holds them, in 64 bits."""
        return self.val.to(TORCH[dtype]).to(self.val.dtype)


def _apply(offs, val, x):
    """A x in the slot form."""
    return sum(v * torch.roll(x, -o) for o, v in zip(offs, val))


def _residuals(G, seed):
    """Residuals of the damped Jacobi iteration at steps 2, 8 and 32, normalised: what the learned part trains on."""
    val = G.rounded("f32")
    r = _uniform(G.n, "f64", _gen(seed + 7))
    out = []
    for it in range(33):
        if it in (2, 8, 32):
            out.append(r / torch.linalg.vector_norm(r))
        r = r - (2.0 / 3.0) * _apply(G.offs, val, r / val[G.dslot])
    return torch.stack(out).to(torch.float32).contiguous()


def _vectors(case, seed):
    """x, y of a reduction (y only for dot2)."""
    g, n, t = _gen(seed), case["n"], case["dtype"]
    if not case["cond"]:
        v = [_uniform(n + case["shift"], t, g)[case["shift"]:] for _ in range(2 if case["op"] == "dot2" else 1)]
        return v if len(v) == 2 else [v[0], None]
    # products over 48 binary orders whose sum cancels up to a tail of a thousand terms near 1
    half = (n - 1000) // 2
    x, y = (_uniform(n, "f64", g) for _ in range(2))
    for v in (x, y):
        v[:half] *= 2.0 ** torch.randint(0, 25, (half,), generator=g, device="cuda")
    at = half + torch.randperm(half, generator=g, device="cuda")
    x[at] = x[:half].clone()
    y[at] = -y[:half].clone()
    return [x, y]


VECTOR_INPUTS = {"axpy": 1, "axpby": 1, "axpbypcz": 2, "axpbypcwpdz": 3, "lincomb4": 4, "scal": 1, "mul_pointwise": 2}
COEF = (0.75, -0.5, 0.25, 0.125)


def _vec_inputs(case, seed):
    g = _gen(seed)
    return [_uniform(case["n"], case["dtype"], g) for _ in range(VECTOR_INPUTS[case["op"]] + 1)]


def _solver_params(case):
    return _lib.solver_params("bicgstabl", case["l"], rel_tol=1e-14, max_iters=case["iters"],
                              precond="jacobi" if case["jacobi"] else "none", fused=True)


def _refine_params(case):
    if case["grid"] == "poisson":
        return _lib.ir_params("gmres", case["basis"], inner_rel_tol=0.0, inner_max_iters=0, rel_tol=case["tol"],
                              max_refinements=400)
    return _lib.ir_params("bicgstabl", case["basis"], inner_rel_tol=1e-5, inner_max_iters=5000, rel_tol=case["tol"])


def _ok(st, *also):
    if st != 0 and st not in also:
        raise _lib.HpbError(st, "call failed")


def prepare(case, seed):
    f = case["family"]
    ctx = Context(0, torch.cuda.current_stream().cuda_stream)
    s = {"case": case, "ctx": ctx}
    if f == "reduce":
        s["x"], s["y"] = _vectors(case, seed)
        s["host"] = np.zeros(4)
        s["dev"] = torch.zeros(4, dtype=torch.float64, device="cuda")
        name = "hpb_%s_%s%s" % (case["op"], case["dtype"], "_host" if case["by_value"] else "")
        out = s["host"].ctypes.data if case["by_value"] else s["dev"].data_ptr()
        args = [ctx.h, case["n"], s["x"].data_ptr()] + ([s["y"].data_ptr()] if s["y"] is not None else []) + [out]
        s["call"], s["args"] = getattr(L, name), args
        wide = case["dtype"] in ("c64", "c128") and case["op"] in ("dot2", "sum2")
        k = 4 if wide else 3 if case["op"] == "nrm2" else 2
        s["out"] = s["host"][:k] if case["by_value"] else s["dev"][:k]
    elif f == "vector":
        v = s["v"] = _vec_inputs(case, seed)
        c = [_lib.scalar(case["dtype"], z) for z in COEF]
        args = [ctx.h, case["n"]]
        if case["op"] == "axpy":
            args += [c[0], v[0].data_ptr(), v[1].data_ptr()]
        elif case["op"] == "scal":
            args += [c[0], v[0].data_ptr(), v[1].data_ptr()]
        elif case["op"] in ("lincomb4", "mul_pointwise"):  # the result in a vector of its own
            for k in range(VECTOR_INPUTS[case["op"]]):
                args += [c[k], v[k].data_ptr()]
            args.append(v[-1].data_ptr())
        else:
            for k in range(len(v)):
                args += [c[k], v[k].data_ptr()]
        s["call"], s["args"], s["out"] = getattr(L, "hpb_%s_%s" % (case["op"], case["dtype"])), args, v[-1]
    elif f == "spai":
        G = Grid(case, seed)
        rp, ci, val = s["csr"] = G.csr("f32")
        s["net"] = spai.SpaiNet(G.offs, G.dslot)
        s["net"].set_weights(np.load(spai.WEIGHTS_FILE))
        s["res"] = _residuals(G, seed) if case["train"] else None
        s["sys"] = _lib.hpb_spai_system(G.n, len(ci), rp.data_ptr(), ci.data_ptr(), val.data_ptr(),
                                        3 if case["train"] else 0, s["res"].data_ptr() if case["train"] else None)
        s["loss"], s["grad"] = np.zeros(3), np.zeros(spai.NUM_PARAMS, dtype=np.float32)
        s["m"] = torch.empty(len(ci), dtype=torch.float32, device="cuda")
    else:
        G = Grid(case, seed)
        t = case.get("dtype") or ("c128" if case["grid"] == "helmholtz" else "f64")
        rp, ci, val = s["csr"] = G.csr(t)
        s["n"], s["nnz"], s["t"] = G.n, len(ci), t
        s["ptr"] = [rp.data_ptr(), ci.data_ptr(), val.data_ptr()]
        s["b"] = _uniform(G.n, t, _gen(seed))
        s["x"] = torch.zeros_like(s["b"])
        if f == "spmv":
            s["w"] = _uniform(G.n, t, _gen(seed + 1))
            s["dev"] = torch.zeros(4 if case["grid"] == "helmholtz" else 2, dtype=torch.float64, device="cuda")
        elif f in ("ilu0", "trsv"):
            s["lu"] = torch.empty_like(val)
            s["call"] = getattr(L, "hpb_csr_%s_%s" % (f, t))
            if f == "trsv":
                s["lu"].copy_(val)
                s["tri"] = [_analysis(s, k) for k in (0, 1)]
                _ok(getattr(L, "hpb_csr_ilu0_%s" % t)(ctx.h, s["tri"][0], s["lu"].data_ptr()))
                s["mid"] = torch.empty_like(s["b"])
        elif f == "bicg":
            s["p"], s["rep"] = _solver_params(case), _lib.hpb_solver_report()
            s["call"] = getattr(L, "hpb_csr_solve_%s" % t)
        else:
            s["p"], s["rep"] = _refine_params(case), _lib.hpb_ir_report()
            s["call"] = getattr(L, "hpb_ir_solve_%s" % t)
    return s


def _analysis(s, upper):
    h = ctypes.c_void_p()
    _ok(L.hpb_csr_tri_create(s["ctx"].h, upper, s["n"], s["nnz"], s["ptr"][0], s["ptr"][1], ctypes.byref(h)))
    return Analysis(h)


class Analysis(ctypes.c_void_p):
    """A triangle's analysis, released with the program's last reference to it."""

    def __init__(self, h):
        super().__init__(h.value)

    def __del__(self):
        if self.value:
            L.hpb_csr_tri_destroy(self)
            self.value = None


def run(s):
    case, f = s["case"], s["case"]["family"]
    if f in ("reduce", "vector"):
        _ok(s["call"](*s["args"]))
        return s["out"]
    if f == "spai":
        if case["train"]:
            _ok(L.hpb_spai_loss_grad(s["net"].h, ctypes.byref(s["sys"]), 1.0, 1.0, s["loss"].ctypes.data,
                                     s["grad"].ctypes.data))
            return s["loss"], s["grad"]
        _ok(L.hpb_spai_assemble(s["net"].h, ctypes.byref(s["sys"]), s["m"].data_ptr()))
        return s["m"]
    n, nnz, ptr, t = s["n"], s["nnz"], s["ptr"], s["t"]
    if f == "spmv":
        if case["dot"]:
            _ok(getattr(L, "hpb_csr_spmv_dot2_" + t)(s["ctx"].h, n, n, nnz, *ptr, s["b"].data_ptr(),
                                                     s["x"].data_ptr(), s["w"].data_ptr(), s["dev"].data_ptr()))
            return s["x"], s["dev"]
        beta = _lib.scalar(t, 0.5 if case["beta"] else 0.0)
        _ok(getattr(L, "hpb_csr_spmv_" + t)(s["ctx"].h, n, n, nnz, *ptr, _lib.scalar(t, 1.0), s["b"].data_ptr(),
                                            beta, s["x"].data_ptr()))
        return s["x"]
    if f == "ilu0":
        s["lu"].copy_(s["csr"][2])
        s["tri"] = [_analysis(s, k) for k in (0, 1)]
        _ok(s["call"](s["ctx"].h, s["tri"][0], s["lu"].data_ptr()))
        return s["lu"]
    if f == "trsv":
        one = _lib.scalar(t, 1.0)
        _ok(s["call"](s["ctx"].h, s["tri"][0], 1, s["lu"].data_ptr(), one, s["b"].data_ptr(), s["mid"].data_ptr()))
        _ok(s["call"](s["ctx"].h, s["tri"][1], 0, s["lu"].data_ptr(), one, s["mid"].data_ptr(), s["x"].data_ptr()))
        return s["x"]
    s["x"].zero_()
    if f == "bicg":
        _ok(s["call"](ctypes.byref(s["p"]), n, nnz, *ptr, s["b"].data_ptr(), s["x"].data_ptr(),
                      ctypes.byref(s["rep"]), None, 0), NOT_CONVERGED)
        return s["x"], s["rep"].true_resid_norm
    _ok(s["call"](ctypes.byref(s["p"]), n, nnz, *ptr, None, None, None, None, 0, s["b"].data_ptr(),
                  s["x"].data_ptr(), ctypes.byref(s["rep"]), None, 0))
    return s["x"]


# ---------------------------------------------------------------- work
def _nnz(case):
    n, side = case["nx"] * case["ny"] * case["nz"], [case["nx"], case["ny"]] + ([case["nz"]] if case["nz"] > 1 else [])
    return n, n + 2 * sum(n - n // m for m in side)


def work(case):
    f = case["family"]
    if f == "reduce":
        v = case["n"] * (2 if case["op"] == "dot2" else 1)
        flops = {"f32": 10, "f64": 10, "c64": 40, "c128": 40}[case["dtype"]] * case["n"]
        return {"bytes": v * BYTES[case["dtype"]], "flops": flops}
    if f == "vector":
        k = VECTOR_INPUTS[case["op"]]
        moved = k + 1 if case["op"] in ("lincomb4", "mul_pointwise", "scal") else k + 2
        return {"bytes": moved * case["n"] * BYTES[case["dtype"]], "flops": 2 * k * case["n"]}
    n, nnz = _nnz(case)
    if f == "spai":
        b = nnz * 8 + 4 * n + (n * 12 if case["train"] else nnz * 4)
        return {"bytes": b, "flops": n * 2 * (16 * 64 + 64 * 64 + 64 * 8) * (3 if case["train"] else 1)}
    t = case.get("dtype") or ("c128" if case["grid"] == "helmholtz" else "f64")
    V = BYTES[t]
    m = 4 if t in ("c64", "c128") else 1
    matrix = nnz * (V + 4) + 4 * (n + 1)
    if f == "spmv":
        return {"bytes": matrix + V * n * (2 + case["beta"] + case["dot"]), "flops": 2 * m * nnz}
    if f == "ilu0":
        return {"bytes": matrix + V * nnz, "flops": 2 * m * nnz}
    if f == "trsv":
        return {"bytes": matrix + 2 * V * n, "flops": 2 * m * nnz}
    if f == "bicg":  # per iteration two products, per cycle one pass over the cycle's vectors
        cycles = -(-case["iters"] // case["l"])
        per = 2 * case["l"] * (matrix + 2 * V * n) + (2 * case["l"] + 6) * V * n
        return {"bytes": cycles * per, "flops": cycles * 2 * case["l"] * 2 * m * nnz}
    # the iterations of a refined solve depend on the system: those measured on
    # the listed sizes, scaled with the side for the Poisson operator
    h = V // 2
    low = nnz * (h + 4) + 4 * (n + 1)
    if case["grid"] == "poisson":
        steps = 13 * max(case["nx"], case["ny"], case["nz"])
        per = low + 2 * h * n + 2 * (case["basis"] / 2) * h * n
    else:
        steps = 120
        per = 2 * (low + 2 * h * n) + (2 * case["basis"] + 6) * h * n / case["basis"]
    return {"bytes": steps * per, "flops": steps * 2 * m * nnz}


# ---------------------------------------------------------------- exact
def _wide(v):
    return v.to(torch.complex128 if v.is_complex() else torch.float64)


def _exact_reduce(case, seed):
    x, y = _vectors(case, seed)
    if case["cond"]:
        p = x * y

        def halves(v):  # Veltkamp's splitting
            c = 134217729.0 * v
            hi = c - (c - v)
            return hi, v - hi

        (xh, xl), (yh, yl) = halves(x), halves(y)
        e = xl * yl - (((p - xh * yh) - xl * yh) - xh * yl)
        return np.array([math.fsum(p.tolist() + e.tolist()), 0.0])
    x = _wide(x)
    if case["op"] == "dot2":
        v = (x.conj() * _wide(y)).sum()
    elif case["op"] == "sum2":
        v = x.sum()
    elif case["op"] == "asum2":
        v = (x.real.abs() + x.imag.abs()).sum() if x.is_complex() else x.abs().sum()
    else:
        v = (x.real.square() + x.imag.square()).sum() if x.is_complex() else x.square().sum()
        return np.array([math.sqrt(float(v)), float(v), 0.0])
    if v.is_complex():
        return np.array([float(v.real), float(v.imag), 0.0, 0.0])
    return np.array([float(v), 0.0])


def _exact_vector(case, seed):
    v = [_wide(z) for z in _vec_inputs(case, seed)]
    op = case["op"]
    if op == "mul_pointwise":
        return COEF[0] * v[0] * COEF[1] * v[1]
    if op == "axpy":
        return COEF[0] * v[0] + v[1]
    used = v[:-1] if op in ("lincomb4", "scal") else v
    return sum(c * z for c, z in zip(COEF, used))


def _levels(G):
    nz, ny, nx = G.shape
    i = np.arange(G.n)
    lev = i % nx + (i // nx) % ny + i // (nx * ny)
    order = np.argsort(lev, kind="stable")
    return np.split(order, np.cumsum(np.bincount(lev))[:-1])


def _exact_ilu0(G, dtype):
    """ILU(0) of a grid operator: only the diagonal is updated beside the lower entries' division."""
    val, has = G.rounded(dtype).cpu().numpy().copy(), G.has.cpu().numpy()
    d, k = G.dslot, len(G.offs)
    for at in _levels(G):
        for s in range(d):
            m = at[has[s, at]]
            j = m + G.offs[s]
            val[s, m] = val[s, m] / val[d, j]
            val[d, m] -= val[s, m] * val[k - 1 - s, j]
    return val


def _exact_trsv(G, case, seed):
    val, has = _exact_ilu0(G, case["dtype"]), G.has.cpu().numpy()
    d, k = G.dslot, len(G.offs)
    x = _wide(_uniform(G.n, case["dtype"], _gen(seed))).cpu().numpy().astype(val.dtype)
    levels = _levels(G)
    for at in levels:
        for s in range(d):
            m = at[has[s, at]]
            x[m] -= val[s, m] * x[m + G.offs[s]]
    for at in reversed(levels):
        for s in range(d + 1, k):
            m = at[has[s, at]]
            x[m] -= val[s, m] * x[m + G.offs[s]]
        x[at] /= val[d, at]
    return torch.from_numpy(x)


def _sine(v, ax):
    """Sum over j of v_j sin(pi (j+1) (k+1) / (m+1)) along one axis."""
    m = v.shape[ax]
    z = torch.zeros_like(v.narrow(ax, 0, 1))
    odd = torch.cat([z, v, z, -v.flip(ax)], ax)
    f = torch.fft.fft(odd, dim=ax).narrow(ax, 1, m)
    return f * 0.5j


def _exact_solve(G, b):
    """A^-1 b for constant symmetric coefficients, by the sine transform of each axis."""
    lo, _, diag = G.const
    v = b.reshape(G.shape).to(torch.complex128)
    lam = torch.zeros((1, 1, 1), dtype=torch.complex128, device=b.device) + diag
    for d in range(len(lo)):
        ax = 2 - d
        m = G.shape[ax]
        k = torch.arange(1, m + 1, device=b.device, dtype=torch.float64)
        c = 2 * lo[d] * torch.cos(math.pi * k / (m + 1))
        lam = lam + c.reshape([-1 if j == ax else 1 for j in range(3)])
        v = _sine(v, ax)
    v = v / lam
    for d in range(len(lo)):
        v = _sine(v, 2 - d) * (2.0 / (G.shape[2 - d] + 1))
    v = v.reshape(-1)
    return v if b.is_complex() else v.real.contiguous()


def _bf16_weights():
    w = torch.from_numpy(np.load(spai.WEIGHTS_FILE)).cuda()
    return w.to(torch.bfloat16).to(torch.float64)


def _exact_spai(case, seed):
    G = Grid(case, seed)
    val, has, offs, d = G.rounded("f32"), G.has, G.offs, G.dslot
    k = len(offs)
    diag = val[d]

    def nb(v, s):  # the neighbour's value in slot s
        return torch.roll(v, -offs[s], -1)

    w = _bf16_weights().requires_grad_(case["train"])
    w1, b1, w2, b2, w3, b3 = torch.split(w, [16 * 64, 64, 64 * 64, 64, 64 * 8, 8])
    off = [s for s in range(k) if s != d]
    ah = torch.stack([torch.where(has[s], val[s] / torch.sqrt((diag * nb(diag, s)).abs()), 0.0) for s in range(k)])
    logs = torch.log(diag.abs())
    zero = torch.zeros_like(diag)
    feat = [ah[s] for s in off] + [torch.where(has[s], nb(logs, s) - logs, 0.0) for s in off]
    feat += [logs - logs.mean(), torch.ones_like(diag)]
    x = torch.stack(feat + [zero] * (16 - len(feat)), 1)
    h = torch.relu(x @ w1.reshape(16, 64) + b1)
    h = torch.relu(h @ w2.reshape(64, 64) + b2)
    t = torch.tanh(h @ w3.reshape(64, 8) + b3).t()
    S = [0.25 * torch.where(has[s], t[s] + nb(t[k - 1 - s], s), zero) for s in range(k)]
    mh = [S[s] if s != d else 1 + 0.5 * t[d] + sum(S[q].abs() for q in off) for s in range(k)]
    if not case["train"]:
        m = [mh[s] / torch.sqrt((diag * nb(diag, s)).abs()) for s in range(k)]
        return torch.stack(m).t()[has.t()]
    g = {}
    for p in range(k):
        for q in range(k):
            o = offs[p] + offs[q]
            g[o] = g.get(o, 0.0) + ah[p] * nb(mh[q], p)
    frob = sum((v - (1.0 if o == 0 else 0.0)).square().sum() for o, v in g.items()) / G.n
    resid = 0.0
    for r in _residuals(G, seed).to(torch.float64):
        rh = r / torch.sqrt(diag.abs())
        z = _apply(offs, ah, _apply(offs, mh, rh)) - rh
        resid = resid + z.square().sum() / rh.square().sum() / 3
    (frob + resid).backward()
    return np.array([float(frob + resid), float(frob), float(resid)]), w.grad


def exact(case, seed):
    f = case["family"]
    if f == "reduce":
        return _exact_reduce(case, seed)
    if f == "vector":
        return _exact_vector(case, seed)
    if f == "spai":
        return _exact_spai(case, seed)
    if f == "bicg":
        return None  # where a bounded number of iterations ends is no value of its own
    G = Grid(case, seed)
    if f == "refine":
        b = _uniform(G.n, "c128" if case["grid"] == "helmholtz" else "f64", _gen(seed))
        return _exact_solve(G, b)
    if f == "ilu0":
        return torch.from_numpy(_exact_ilu0(G, case["dtype"])).t()[G.has.cpu().t()]
    if f == "trsv":
        return _exact_trsv(G, case, seed)
    x = _wide(_uniform(G.n, case["dtype"], _gen(seed)))
    y = _apply(G.offs, G.rounded(case["dtype"]), x)
    if not case["dot"]:
        return y
    w = _wide(_uniform(G.n, case["dtype"], _gen(seed + 1)))
    v = (w.conj() * y).sum()
    return y, np.array([float(v.real), float(v.imag), 0.0, 0.0] if v.is_complex() else [float(v), 0.0])
