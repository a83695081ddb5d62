// The products of the device-resident BiCGStab(l) on a matrix in slot form:
// k_spmv_dot and k_spmv_upd of hpb_fused_bicgstabl.cu (what they compute, and
// why the updates run inside them, is said there) with the row's entries from
// SlotRow.  Bound by memory latency: what made them faster than the CSR
// products is less the fewer bytes (1.22 instead of 1.42 GB a BiCGStab(4)
// cycle) than that all loads of a row are in flight at once -- with the slots'
// loads behind the row's mask they were no faster (k_spmv_upd_slots<double, 3>
// 50 us, 31 us as it is; CSR 42).
// Measured on B200: f64, 1024^2 5-point, BiCGStab(4): 250 us a cycle against
// 324 us; complex<binary32>, 2048^2, BiCGStab(2) in refinement: 60 ms a solve
// against 80 ms, of which 5 ms come from rounding in binary64 (round_s) instead
// of converting back and forth.  Three blocks an SM where the registers allow
// it (25.2 against 25.8 and 26.0 ms for 100 cycles at two and four); six blocks
// an SM of the product with the Dot2 (four, eight: 26.5, 26.9 ms); contiguous
// rows per block were slower for complex data (62.5 against 60.3 ms).
#include <algorithm>

#include "hpb_bcg.cuh"

namespace hpb {
namespace fused {
namespace {

template <class E, int NS>
__global__ void __launch_bounds__(kThreads)
k_spmv_dot_slots(int32_t rows, SlotMat<E> A, const E* __restrict__ diag, const E* __restrict__ u, E* __restrict__ y,
                 const E* __restrict__ w, typename acc_of<typename scalar_of<E>::type>::type* partials,
                 unsigned int* ticket, int* badflag, EpiArgs<typename scalar_of<E>::type> ea, const E* __restrict__ rr) {
    using S = typename scalar_of<E>::type;
    using AC = typename acc_of<S>::type;
    typename pacc_of<E>::type pacc;
    const S nb = s_neg(ea.st->beta);
    constexpr int XL = LM_ALIGNED;
    const int32_t stride = gridDim.x * kThreads;
    for (int32_t r = blockIdx.x * kThreads + threadIdx.x; r < rows; r += stride) {
        SlotRow<E, NS, SlotFma<E>> row;
        const E we = ldE(w, r);
        row.load(A, rows, r, [&](int32_t c) { return SlotFma<E>{ld_x<XL>(u, c), ld_x<XL>(rr, c), nb}; });
        S acc = row.sum(s_zero(S{}));
        if (diag) acc = s_div(acc, to_s(ldE(diag, r)));
        const E out = from_s<E>(acc);
        stE(y, r, out);
        pdot_add(pacc, we, out);
    }
    AC dacc[1] = {widen_acc(pacc)};
    grid_finish<1>(dacc, false, partials, ticket, badflag, [&](const S* v, bool bad) { run_epi(ea, v, bad); });
}

template <class E, int J, bool MR, int NS>
__global__ void __launch_bounds__(kThreads, J <= 3 ? 3 : 1)
k_spmv_upd_slots(int32_t rows, SlotMat<E> A, const E* __restrict__ diag, Vecs<E> V, E* __restrict__ x,
                 const E* __restrict__ w, BcgState<typename scalar_of<E>::type>* st,
                 typename acc_of<typename scalar_of<E>::type>::type* partials, unsigned int* ticket, int* badflag,
                 EpiArgs<typename scalar_of<E>::type> ea) {
    using S = typename scalar_of<E>::type;
    using AC = typename acc_of<S>::type;
    constexpr int ND = MR ? J + 2 : 1, XL = LM_ALIGNED;
    const S nb = s_neg(st->beta), al = st->alpha, nal = s_neg(st->alpha), nalp = s_neg(st->alpha_prev);
    const E* __restrict__ rj = V.r[J];
    const E* __restrict__ uj1 = V.u[J + 1];
    E* y = V.r[J + 1];
    typename pacc_of<E>::type pacc[ND];
    const int32_t stride = gridDim.x * kThreads;
    for (int32_t q = blockIdx.x * kThreads + threadIdx.x; q < rows; q += stride) {
        // every load of the row first
        SlotRow<E, NS, SlotFma<E>> row;
        row.load(A, rows, q, [&](int32_t c) { return SlotFma<E>{ld_x<XL>(uj1, c), ld_x<XL>(rj, c), nal}; });
        S r[J + 1], u[J + 1];
        E rv[J + 1];
#pragma unroll
        for (int i = 0; i <= J; ++i) {
            r[i] = to_s(ldE(V.r[i], q));
            u[i] = to_s(ldE(V.u[i], q));
        }
        const E xq = ldE(x, q);
        E uq{}, wq{};
        if (MR) uq = ldE(uj1, q);
        if (!MR) wq = ldE(w, q);
        S acc = row.sum(s_zero(S{}));
        // each vector is rounded to storage where a separate update would store it
        if (J >= 1) r[J - 1] = round_s<E>(s_fma(nalp, u[J], r[J - 1]));
#pragma unroll
        for (int i = 0; i <= J; ++i) {
            u[i] = round_s<E>(s_fma(nb, u[i], r[i]));
            stE(V.u[i], q, from_s<E>(u[i]));
        }
#pragma unroll
        for (int i = 0; i < J; ++i) {
            rv[i] = from_s<E>(s_fma(nal, u[i + 1], r[i]));
            stE(V.r[i], q, rv[i]);
        }
        if (MR) rv[J] = from_s<E>(s_fma(nal, to_s(uq), r[J]));
        stE(x, q, from_s<E>(s_fma(al, u[0], to_s(xq))));
        if (diag) acc = s_div(acc, to_s(ldE(diag, q)));
        const E out = from_s<E>(acc);
        stE(y, q, out);
        if constexpr (MR) {
            const E r1 = J >= 1 ? rv[J >= 1 ? 1 : 0] : out;
            pdot_add(pacc[0], r1, r1);
            pdot_add(pacc[1], r1, rv[0]);
#pragma unroll
            for (int i = 2; i < ND; ++i) pdot_add(pacc[i], r1, i <= J ? rv[i <= J ? i : 0] : out);
        } else {
            pdot_add(pacc[0], wq, out);
        }
    }
    AC dacc[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d) dacc[d] = widen_acc(pacc[d]);
    if constexpr (MR) {
        __shared__ AC sh[ND * 32];
        block_merge<ND>(dacc, sh);
        if (threadIdx.x == 0)
#pragma unroll
            for (int d = 0; d < ND; ++d) partials[size_t(d) * gridDim.x + blockIdx.x] = dacc[d];
    } else {
        grid_finish<1>(dacc, false, partials, ticket, badflag, [&](const S* v, bool bad) { run_epi(ea, v, bad); });
    }
}

// f(NS) for the compile-time slot count that holds ns
template <class F>
void with_slots(int ns, F f) {
    if (ns <= 5)
        f(std::integral_constant<int, 5>{});
    else
        f(std::integral_constant<int, 7>{});
}
template <class F>
void with_step(int j, F f) {
    switch (j) {
#define HPB_J(JJ) case JJ: f(std::integral_constant<int, JJ>{}); break;
        HPB_J(0) HPB_J(1) HPB_J(2) HPB_J(3) HPB_J(4) HPB_J(5) HPB_J(6) HPB_J(7)
#undef HPB_J
        default: break;
    }
}

}  // namespace

template <class E>
void launch_spmv_dot_slots(const SlotMat<E>& A, int grid, cudaStream_t s, int32_t rows, const E* diag, const E* u, E* y,
                           const E* w, typename acc_of<typename scalar_of<E>::type>::type* partials,
                           unsigned int* ticket, int* badflag, EpiArgs<typename scalar_of<E>::type> ea, const E* r) {
    with_slots(A.ns, [&](auto nsc) {
        constexpr int NS = decltype(nsc)::value;
        k_spmv_dot_slots<E, NS><<<grid, kThreads, 0, s>>>(rows, A, diag, u, y, w, partials, ticket, badflag, ea, r);
    });
}

template <class E>
void launch_spmv_upd_slots(const SlotMat<E>& A, int j, int L, int grid, cudaStream_t s, int32_t rows, const E* diag,
                           const Vecs<E>& V, E* x, const E* w, BcgState<typename scalar_of<E>::type>* st,
                           typename acc_of<typename scalar_of<E>::type>::type* partials, unsigned int* ticket,
                           int* badflag, EpiArgs<typename scalar_of<E>::type> ea) {
    with_slots(A.ns, [&](auto nsc) {
        with_step(j, [&](auto jc) {
            constexpr int NS = decltype(nsc)::value, J = decltype(jc)::value;
            if (J + 1 == L)
                k_spmv_upd_slots<E, J, true, NS><<<grid, kThreads, 0, s>>>(rows, A, diag, V, x, w, st, partials, ticket,
                                                                          badflag, ea);
            else
                k_spmv_upd_slots<E, J, false, NS><<<grid, kThreads, 0, s>>>(rows, A, diag, V, x, w, st, partials, ticket,
                                                                           badflag, ea);
        });
    });
}

template <class E>
int spmv_upd_slots_occupancy(int ns, int j, int L) {
    int occ = 1;
    with_slots(ns, [&](auto nsc) {
        with_step(j, [&](auto jc) {
            constexpr int NS = decltype(nsc)::value, J = decltype(jc)::value;
            const void* f = J + 1 == L ? reinterpret_cast<const void*>(k_spmv_upd_slots<E, J, true, NS>)
                                       : reinterpret_cast<const void*>(k_spmv_upd_slots<E, J, false, NS>);
            int o = 0;
            occ = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, f, kThreads, 0) == cudaSuccess && o > 0 ? o : 1;
        });
    });
    return occ;
}

#define HPB_BCG_SLOTS(E)                                                                                                 \
    template void launch_spmv_dot_slots<E>(const SlotMat<E>&, int, cudaStream_t, int32_t, const E*, const E*, E*,       \
                                           const E*, acc_of<scalar_of<E>::type>::type*, unsigned int*, int*,            \
                                           EpiArgs<scalar_of<E>::type>, const E*);                                      \
    template void launch_spmv_upd_slots<E>(const SlotMat<E>&, int, int, int, cudaStream_t, int32_t, const E*,           \
                                           const Vecs<E>&, E*, const E*, BcgState<scalar_of<E>::type>*,                 \
                                           acc_of<scalar_of<E>::type>::type*, unsigned int*, int*,                      \
                                           EpiArgs<scalar_of<E>::type>);                                                \
    template int spmv_upd_slots_occupancy<E>(int, int, int);
HPB_BCG_SLOTS(float)
HPB_BCG_SLOTS(double)
HPB_BCG_SLOTS(cf)
HPB_BCG_SLOTS(cd)
#undef HPB_BCG_SLOTS

}  // namespace fused
}  // namespace hpb
