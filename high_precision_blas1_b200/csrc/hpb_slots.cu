// Finding and filling the slot form of a CSR matrix (hpb_slots.cuh).
#include <algorithm>
#include <climits>

#include "hpb_slots.cuh"

namespace hpb {
namespace fused {
namespace {

constexpr int kFindThreads = 256;
constexpr int kNoOffset = INT_MIN;

// Distinct offsets col - row of the whole matrix.  Each block collects its own in
// shared memory.
__global__ void k_slots_init(OffsetTable* t) {
    if (threadIdx.x < kMaxSlots) t->off[threadIdx.x] = kNoOffset;
    if (threadIdx.x == kMaxSlots) t->bad = 0;
}
__device__ __forceinline__ bool insert_offset(int* table, int d) {
    for (int q = 0; q < kMaxSlots; ++q) {
        const int have = *reinterpret_cast<volatile int*>(table + q);
        if (have == d) return true;
        if (have == kNoOffset) {
            const int was = atomicCAS(table + q, kNoOffset, d);
            if (was == kNoOffset || was == d) return true;
        }
    }
    return false;
}
__global__ void __launch_bounds__(kFindThreads)
k_slots_find(int32_t rows, int64_t nnz, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, OffsetTable* t) {
    __shared__ int table[kMaxSlots];
    if (threadIdx.x < kMaxSlots) table[threadIdx.x] = kNoOffset;
    __syncthreads();
    bool bad = false;
    for (int64_t i = int64_t(blockIdx.x) * kFindThreads + threadIdx.x; i < rows && !bad;
         i += int64_t(gridDim.x) * kFindThreads) {
        const int32_t b = __ldg(rp + i), e = __ldg(rp + i + 1);
        if (b < 0 || e < b || e - b > kMaxSlots || int64_t(e) > nnz) {
            bad = true;
            break;
        }
        int32_t prev = -1;
        for (int32_t k = b; k < e; ++k) {
            const int32_t c = __ldg(ci + k);
            bad |= c <= prev || c >= rows || !insert_offset(table, c - int32_t(i));
            prev = c;
        }
    }
    if (__syncthreads_or(bad)) {
        if (threadIdx.x == 0) t->bad = 1;
        return;
    }
    if (threadIdx.x < kMaxSlots && table[threadIdx.x] != kNoOffset && !insert_offset(t->off, table[threadIdx.x]))
        t->bad = 1;
}

template <class E>
struct SlotTarget {
    E* val;
    uint8_t* mask;
    int ns, held;
    int off[kMaxSlots];
};
template <class E>
__global__ void __launch_bounds__(kFindThreads)
k_slots_fill(int32_t rows, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci, const E* __restrict__ val,
             SlotTarget<E> t) {
    const int32_t i = blockIdx.x * kFindThreads + threadIdx.x;
    if (i >= rows) return;
    int32_t k = __ldg(rp + i);
    const int32_t e = __ldg(rp + i + 1);
    unsigned m = 0;
#pragma unroll
    for (int s = 0; s < kMaxSlots; ++s)
        if (s < t.held) {
            E v{};
            if (s < t.ns && k < e && __ldg(ci + k) - i == t.off[s]) {
                v = ldE(val, k);
                m |= 1u << s;
                ++k;
            }
            t.val[int64_t(s) * rows + i] = v;
        }
    t.mask[i] = uint8_t(m);
}

}  // namespace

int find_slots(SolverWorkspace& ws, int32_t rows, int64_t nnz, const int32_t* rp, const int32_t* ci, OffsetTable* host) {
    host->bad = 1;
    // at least nnz / rows offsets: a matrix with longer rows has no slot form
    if (rows <= 0 || nnz <= 0 || nnz > int64_t(rows) * kMaxSlots) return HPB_SUCCESS;
    cudaStream_t s = ws.stream;
    OffsetTable* t = static_cast<OffsetTable*>(ws.alloc(sizeof(OffsetTable)));
    if (t == nullptr) return HPB_SUCCESS;
    k_slots_init<<<1, 32, 0, s>>>(t);
    k_slots_find<<<int(std::min<int64_t>((int64_t(rows) + kFindThreads - 1) / kFindThreads, 148 * 8)), kFindThreads, 0, s>>>(
        rows, nnz, rp, ci, t);
    count_launch(2);
    return cudaMemcpyAsync(host, t, sizeof(*t), cudaMemcpyDeviceToHost, s) == cudaSuccess ? HPB_SUCCESS : HPB_ERROR_CUDA;
}

template <class E>
int make_slots(SolverWorkspace& ws, int32_t rows, int64_t nnz, const int32_t* rp, const int32_t* ci, const E* val,
               const OffsetTable* host, SlotMat<E>* out, const SlotMat<E>* like) {
    *out = SlotMat<E>{};
    SlotMat<E> A;
    if (like != nullptr) {
        if (like->ns == 0) return HPB_SUCCESS;
        A = *like;
    } else {
        if (host->bad) return HPB_SUCCESS;
        for (int q = 0; q < kMaxSlots; ++q)
            if (host->off[q] != kNoOffset) A.off[A.ns++] = host->off[q];
        std::sort(A.off, A.off + A.ns);
        if (A.ns == 0 || int64_t(std::max(A.ns, 5)) * rows > nnz + nnz / 3) return HPB_SUCCESS;
    }
    const int held = std::max(A.ns, 5);  // kernels read at least five slots
    E* v = static_cast<E*>(ws.alloc(size_t(held) * size_t(rows) * sizeof(E)));
    if (v == nullptr) return HPB_SUCCESS;
    uint8_t* mask = static_cast<uint8_t*>(ws.alloc(size_t(rows)));
    if (mask == nullptr) {
        ws.free_last();
        return HPB_SUCCESS;
    }
    SlotTarget<E> t{v, mask, A.ns, held, {}};
    for (int q = 0; q < kMaxSlots; ++q) t.off[q] = A.off[q];
    k_slots_fill<E><<<int((int64_t(rows) + kFindThreads - 1) / kFindThreads), kFindThreads, 0, ws.stream>>>(rows, rp, ci, val, t);
    count_launch();
    if (cudaGetLastError() != cudaSuccess) return HPB_ERROR_CUDA;
    A.val = v;
    A.mask = mask;
    *out = A;
    return HPB_SUCCESS;
}

#define HPB_SLOTS_INST(E)                                                                                       \
    template int make_slots<E>(SolverWorkspace&, int32_t, int64_t, const int32_t*, const int32_t*, const E*, \
                               const OffsetTable*, SlotMat<E>*, const SlotMat<E>*);
HPB_SLOTS_INST(float)
HPB_SLOTS_INST(double)
HPB_SLOTS_INST(cf)
HPB_SLOTS_INST(cd)
#undef HPB_SLOTS_INST

}  // namespace fused
}  // namespace hpb
