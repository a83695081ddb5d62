// Matrices in slot form, for the plans of the device-resident solvers.
//
// Where every row's columns lie at a few fixed offsets from the row -- every
// 5- and 7-point stencil operator -- the entry of row i at offset off[s] is
// kept at val[s * rows + i], with bit s of mask[i] telling whether row i stores
// it.  A product then reads no column indices and no row pointers (41 bytes a
// row instead of 64 for a binary64 5-point row) and consecutive threads read
// consecutive words everywhere, where a thread of the CSR kernels steps
// through its row's 40 to 112 bytes.  The entries of a row are taken in CSR
// order (increasing columns), absent ones are left out, so every sum has the
// CSR kernels' operations in their order and the same bits.
#pragma once
#include "hpb_fused.cuh"

namespace hpb {
namespace fused {

constexpr int kMaxSlots = 7;

template <class E>
struct SlotMat {
    const E* val = nullptr;
    const uint8_t* mask = nullptr;
    int ns = 0;  // 0: no slot form
    int off[kMaxSlots] = {};  // (with fewer than five slots val holds five: the others empty)
};

// Distinct offsets col - row of a whole matrix (kNoOffset where free); bad: more
// than kMaxSlots, or a row whose columns do not increase within [0, rows).
struct OffsetTable {
    int off[kMaxSlots];
    int bad;
};

// The slot form of a CSR matrix if it has one, in two steps that both leave
// their work on the workspace's stream: find_slots fills *host (pinned), which
// may be read once the stream has been waited for; make_slots then fills the
// slots in workspace memory (ns > 0 on return).  A plan makes its slots after
// all it cannot do without is allocated: without memory for them the matrix
// stays CSR.
// Rule: at most kMaxSlots distinct offsets, columns increasing in every row
// and within [0, rows), and no more than a quarter of the slots empty (a
// matrix that fills its slots less would move more bytes than its CSR).
// `like`: a slot form of a matrix with the same row pointers and column
// indices, whose offsets are taken over (no find_slots then, host unused).
int find_slots(SolverWorkspace& ws, int32_t rows, int64_t nnz, const int32_t* rp, const int32_t* ci, OffsetTable* host);
template <class E>
int make_slots(SolverWorkspace& ws, int32_t rows, int64_t nnz, const int32_t* rp, const int32_t* ci, const E* val,
               const OffsetTable* host, SlotMat<E>* out, const SlotMat<E>* like = nullptr);

// y_i = sum_s a_{i,s} x(i + off[s]) over the slots row i stores, in slot order;
// X: (column) -> operand.  Every load is issued whether the row stores the slot
// or not (columns clamped into the matrix), so none waits for the mask or for
// another: a row costs one memory latency, not the CSR kernels' three (row
// pointers, indices, operand).  NS >= ns, known at compile time.
template <class E, int NS, class O>
struct SlotRow {
    E v[NS];
    O x[NS];
    unsigned m;
    template <class X>
    __device__ __forceinline__ void load(const SlotMat<E>& A, int32_t rows, int32_t i, X op) {
        m = __ldg(A.mask + i);
#pragma unroll
        for (int s = 0; s < NS; ++s) {
            if (NS > 5 && s >= A.ns) continue;  // the same for every thread
            v[s] = ld_val<LM_ALIGNED | LM_CACHED>(A.val, int64_t(s) * rows + i);
            x[s] = op(min(max(i + A.off[s], 0), rows - 1));
        }
    }
    template <class S>
    __device__ __forceinline__ S sum(S acc) const {
#pragma unroll
        for (int s = 0; s < NS; ++s)
            if ((m >> s) & 1u) acc = s_fma(to_s(v[s]), x[s].value(), acc);
        return acc;
    }
};

// Operands of a SlotRow: a vector's entry; x - b r formed as the BiCG updates
// form it (one rounding to the storage type).
template <class E>
struct SlotX {
    E v;
    __device__ __forceinline__ typename scalar_of<E>::type value() const { return to_s(v); }
};
template <class E>
struct SlotFma {
    E u, r;
    typename scalar_of<E>::type f;
    __device__ __forceinline__ typename scalar_of<E>::type value() const {
        return round_s<E>(s_fma(f, to_s(u), to_s(r)));
    }
};

}  // namespace fused
}  // namespace hpb
