"""round_f32 (csrc/hpb_fused.cuh) is the conversion to binary32 and back for
every value that stays within binary32's range (a zero's sign apart), and no
arithmetic in it overflows an int: its source, compiled for the host with the
intrinsics restated, against the compiler's conversions."""
import subprocess
import sys

import numpy as np

from conftest import ROOT

SHIM = r"""
#include <cstdint>
#include <cstring>
#include <algorithm>
using std::max;
static inline uint64_t bits(double v) { uint64_t u; memcpy(&u, &v, 8); return u; }
static inline double from(uint64_t u) { double v; memcpy(&v, &u, 8); return v; }
static inline int __double2hiint(double v) { return int(uint32_t(bits(v) >> 32)); }
static inline int __double2loint(double v) { return int(uint32_t(bits(v))); }
static inline double __hiloint2double(int h, int l) { return from(uint64_t(uint32_t(h)) << 32 | uint32_t(l)); }
static inline float __double2float_rn(double v) { return float(v); }
static inline double add_rn(double a, double b) { volatile double s = a + b; return s; }
static inline double sub_rn(double a, double b) { volatile double s = a - b; return s; }
#define __device__
#define __forceinline__ static inline
"""


def test_round_f32(tmp_path):
    text = (ROOT / "high_precision_blas1_b200" / "csrc" / "hpb_fused.cuh").read_text()
    at = text.index("__device__ __forceinline__ double round_f32")
    body = text[at:text.index("\n}\n", at) + 3]
    src = tmp_path / "r.cpp"
    src.write_text(SHIM + body + 'extern "C" void run(long n, const double* a, double* o) '
                   "{ for (long i = 0; i < n; ++i) o[i] = round_f32(a[i]); }\n")
    lib = tmp_path / "r.so"
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-fsanitize=signed-integer-overflow",
                    "-fsanitize-undefined-trap-on-error", "-shared", "-fPIC", str(src), "-o", str(lib)], check=True)
    rng = np.random.default_rng(1)
    # every exponent, with mantissas at, next to and between binary32's values, of both signs
    exps = np.repeat(np.arange(0, 2048, dtype=np.uint64), 400)
    top = rng.integers(0, 2 ** 23, exps.size, dtype=np.uint64)
    top[::7], top[1::7] = 0, 2 ** 23 - 1
    low = rng.choice(np.array([0, 1, 2 ** 28 - 1, 2 ** 28, 2 ** 28 + 1, 2 ** 29 - 1], dtype=np.uint64), exps.size)
    low[::3] = rng.integers(0, 2 ** 29, len(low[::3]), dtype=np.uint64)
    sign = rng.integers(0, 2, exps.size, dtype=np.uint64)
    v = np.ascontiguousarray((sign << np.uint64(63) | exps << np.uint64(52) | top << np.uint64(29) | low).view(np.float64))
    v = np.concatenate([v, [0.0, -0.0, np.inf, -np.inf, np.nan, 2.0 ** 128, 2.0 ** 128 - 2.0 ** 103, -1e-46, 1e-45]])
    values = tmp_path / "v.npy"
    np.save(values, v)
    # a process of its own: an overflow ends it
    code = ("import ctypes, numpy as np, sys; v = np.load(sys.argv[1]); o = np.empty_like(v); "
            "ctypes.CDLL(sys.argv[2]).run(ctypes.c_long(len(v)), *(ctypes.c_void_p(a.ctypes.data) for a in (v, o))); "
            "np.save(sys.argv[1], o)")
    subprocess.run([sys.executable, "-c", code, str(values), str(lib)], check=True)
    got = np.load(values)
    with np.errstate(all="ignore"):
        want = v.astype(np.float32).astype(np.float64)
    within = np.isfinite(want)
    assert np.array_equal(got[within], want[within])
    assert np.all(np.isnan(got[np.isnan(v)]))
    huge = np.isfinite(v) & ~within & (np.abs(v) < 2.0 ** 994)
    assert np.all(np.abs(got[huge]) >= 2.0 ** 128 - 2.0 ** 104)
