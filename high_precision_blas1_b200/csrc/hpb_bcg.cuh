// Scalars, vectors and epilogues shared by the kernels of the device-resident
// BiCGStab(l): hpb_fused_bicgstabl.cu (CSR matrices, the cycle) and
// hpb_bcg_slots.cu (matrices in slot form).
#pragma once
#include <type_traits>

#include "hpb_fused.cuh"
#include "hpb_slots.cuh"

namespace hpb {
namespace fused {

constexpr int kMaxL = 8;
constexpr int kThreads = 256;

template <class S>
struct BcgState {
    S rho, alpha, omega, beta;
    S alpha_prev;  // alpha of the previous inner step (its deferred r update)
    S tau[kMaxL + 1][kMaxL + 1];
    S sigma[kMaxL + 1], gam[kMaxL + 1], gam1[kMaxL + 1], gam2[kMaxL + 1];
    S last[2];
};

struct Report {
    double rnorm;   // ||r_0|| (compensated)
    int breakdown;  // rho == 0 met
    int nonfinite;  // x held a non-finite entry
};

// The monitor of the device-side cycle loop (default_monitor semantics, one
// test per cycle): the host sets tol / max_iters / iters once per solve and
// chunk_left / hl before each launch of the loop graph.
constexpr int kLoopChunk = 128;  // cycles one launch of the loop graph runs at most
struct MonState {
    double tol;
    double rn;
    int max_iters;
    int iters;
    int chunk_left;
    int hl;          // history entries written in this launch
    int finished, conv, valid, breakdown;
};

template <class E>
struct Vecs {
    E* r[kMaxL + 1];
    E* u[kMaxL + 1];
};

enum Epi { EPI_NONE = 0, EPI_ALPHA, EPI_BETA, EPI_STEP, EPI_FINAL };

template <class S>
struct EpiArgs {
    BcgState<S>* st;
    Report* rep;
    int kind, k, j, L;
    // EPI_FINAL inside the loop graph: the monitor's test and the loop's
    // condition (monitor_step) after the cycle's report is complete
    MonState* mon = nullptr;
    double* hist = nullptr;
    cudaGraphConditionalHandle cond = 0;
};

// End of a cycle inside the loop graph: the host loop's test, then the
// loop's condition.  Every path reaches the one cudaGraphSetConditional
// call, and the loop stops after chunk_left cycles whatever the test says,
// so one launch of the graph always ends.
__device__ inline void monitor_step(MonState* M, const Report* rep, double* hist, int L, cudaGraphConditionalHandle h) {
    const int it = M->iters + L;
    M->iters = it;
    int fin;
    if (rep->breakdown) {
        M->breakdown = 1;
        fin = 1;
    } else {
        const double rn = rep->rnorm;
        const int valid = !rep->nonfinite && isfinite(rn);
        const int conv = valid && rn <= M->tol;
        M->rn = rn;
        M->valid = valid;
        M->conv = conv;
        const int k = M->hl;
        if (k < kLoopChunk) {
            hist[2 * k] = double(it);
            hist[2 * k + 1] = rn;
            M->hl = k + 1;
        }
        fin = !valid || conv || it >= M->max_iters;
    }
    M->finished = fin;
    const int left = M->chunk_left - 1;
    M->chunk_left = left;
    cudaGraphSetConditional(h, (fin || left <= 0) ? 0u : 1u);
}

template <class S>
__device__ void run_epi(const EpiArgs<S>& a, const S* v, bool bad) {
    BcgState<S>& st = *a.st;
    switch (a.kind) {
        case EPI_ALPHA:  // alpha = rho / <rt, u_{j+1}>
            st.alpha_prev = st.alpha;
            st.alpha = s_div(st.rho, v[0]);
            break;
        case EPI_BETA:  // rho1 = <rt, r_j>; beta = alpha rho1 / rho; rho = rho1
            if (s_is_zero(st.rho)) a.rep->breakdown = 1;
            st.beta = s_div(s_mul(st.alpha, v[0]), st.rho);
            st.rho = v[0];
            break;
        case EPI_STEP: {  // sweep k: v = (<r_k, r_k>, <r_k, r_0>, <r_k, r_{k+1}>, ..., <r_k, r_L>)
            const int k = a.k, L = a.L;
            st.sigma[k] = v[0];
            st.gam1[k] = s_div(v[1], v[0]);
            for (int j = k + 1; j <= L; ++j) st.tau[k][j] = s_div(v[1 + j - k], v[0]);
            if (k == L) {  // gamma = T^{-1} gamma', gamma'' (the MR part of bicgstabl.h)
                st.gam[L] = st.gam1[L];
                st.omega = st.gam[L];
                for (int jj = L - 1; jj >= 1; --jj) {
                    S g = st.gam1[jj];
                    for (int i = jj + 1; i <= L; ++i) g = s_sub(g, s_mul(st.tau[jj][i], st.gam[i]));
                    st.gam[jj] = g;
                }
                for (int jj = 1; jj < L; ++jj) {
                    S g = st.gam[jj + 1];
                    for (int i = jj + 1; i < L; ++i) g = s_add(g, s_mul(st.tau[jj][i], st.gam[i + 1]));
                    st.gam2[jj] = g;
                }
            }
            break;
        }
        case EPI_FINAL: {  // v[0] = <rt, r_0>, v[1] = <r_0, r_0>
            a.rep->rnorm = norm_sqrt(s_real(v[1]));
            a.rep->nonfinite = bad ? 1 : 0;
            st.rho = s_neg(s_mul(st.omega, st.rho));  // next cycle: rho = -omega rho
            if (s_is_zero(st.rho)) a.rep->breakdown = 1;
            st.beta = s_div(s_mul(st.alpha, v[0]), st.rho);
            st.rho = v[0];
            if (a.mon) monitor_step(a.mon, a.rep, a.hist, a.L, a.cond);
            break;
        }
        default:
            break;
    }
    st.last[0] = v[0];
}

// The slot-form products (hpb_bcg_slots.cu): k_spmv_dot and k_spmv_upd of
// hpb_fused_bicgstabl.cu with the matrix as slots, element by element the same
// operations.  The first: y = A (r - beta u) and <w, y>, then the epilogue.
template <class E>
void launch_spmv_dot_slots(const SlotMat<E>& A, int grid, cudaStream_t s, int32_t rows, const E* diag, const E* u, E* y,
                           const E* w, typename acc_of<typename scalar_of<E>::type>::type* partials,
                           unsigned int* ticket, int* badflag, EpiArgs<typename scalar_of<E>::type> ea, const E* r);
template <class E>
void launch_spmv_upd_slots(const SlotMat<E>& A, int j, int L, int grid, cudaStream_t s, int32_t rows, const E* diag,
                           const Vecs<E>& V, E* x, const E* w, BcgState<typename scalar_of<E>::type>* st,
                           typename acc_of<typename scalar_of<E>::type>::type* partials, unsigned int* ticket,
                           int* badflag, EpiArgs<typename scalar_of<E>::type> ea);
// resident blocks per SM of the second for step j of l, with ns slots
template <class E>
int spmv_upd_slots_occupancy(int ns, int j, int L);

}  // namespace fused
}  // namespace hpb
