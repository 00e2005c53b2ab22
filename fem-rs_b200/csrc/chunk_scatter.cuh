// chunk_scatter.cuh -- device side of the chunked gather and deterministic
// scatter of the unstructured operators (plan: chunk_plan.h).
//
// Gather: chunk_load_x reads the chunk's DOFs of x once, in ascending runs, into
// shared memory (zero on the essential DOFs of a constrained call); the elements
// take their values from there through 16-bit positions.  Reading x per element
// through a 32-bit map instead (the form before) issued 27 scattered loads per
// Q2 element, each its own 16 to 32 sectors a warp, for 11 DOFs per element of a
// 128-element chunk.
//
// Scatter: the element results lie in shared memory as ys[i * CE + e_local];
// per DOF of the list its slots are summed in the listed order, owned DOFs are
// stored and shared ones leave a partial, which chunk_shared_kernel adds in chunk
// order.  The slot lists (16 bits throughout, 16-byte aligned per chunk) are
// copied to shared memory with cp.async while the elements are computed.  On
// essential DOFs of a constrained call the identity row: y_d (+)= x_d (apply) or 1
// (diagonal).
#pragma once
#include <cstdint>

#include "fg_common.cuh"

namespace fg {

struct ChunkLists {
    const int32_t *cu_off, *cu_n, *cu_own, *cu_part, *cu_s0, *cu_ns;  // per chunk (ChunkPlan)
    const int32_t *cu_dof;     // DOF, sign bit: essential
    const uint16_t *cu_soff, *cu_slots;
    const uint16_t *lmap;      // [nl][E] position in the chunk's list
    void *part;                // partial sums of shared DOFs (the apply's precision)
    const int32_t *sh_dof, *sh_off, *sh_idx;
    int64_t n_shared;
    int max_nu;                // longest chunk DOF list
};

// Bytes of shared memory of a chunk's slot lists: soff [max_nu], slots [nl * CE],
// each padded to 16 bytes.
__host__ __device__ inline int chunk_soff_bytes(int max_nu) { return (2 * max_nu + 15) & ~15; }
__host__ __device__ inline int chunk_list_smem(int nl, int CE, int max_nu) {
    return chunk_soff_bytes(max_nu) + ((2 * nl * CE + 15) & ~15);
}

struct ChunkStage {
    const uint16_t *soff, *slot;  // in shared memory
    int u0, nu, own, part0, ns;
};

__device__ __forceinline__ void chunk_cp16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// Block-wide (BT threads): start the copy of chunk c's slot lists into `stage`
// (chunk_list_smem bytes).  The caller waits (chunk_wait) and places a barrier
// before chunk_sums.
template <int BT>
__device__ __forceinline__ ChunkStage chunk_stage_lists(const ChunkLists &L, int c, unsigned char *stage) {
    ChunkStage S;
    S.u0 = __ldg(L.cu_off + c);
    S.nu = __ldg(L.cu_n + c);
    S.own = __ldg(L.cu_own + c);
    S.part0 = __ldg(L.cu_part + c);
    const int s0 = __ldg(L.cu_s0 + c);
    S.ns = __ldg(L.cu_ns + c);
    uint16_t *soff = reinterpret_cast<uint16_t *>(stage);
    uint16_t *slot = reinterpret_cast<uint16_t *>(stage + chunk_soff_bytes(L.max_nu));
    for (int k = threadIdx.x; k < (S.nu + 7) / 8; k += BT) chunk_cp16(soff + 8 * k, L.cu_soff + S.u0 + 8 * k);
    for (int k = threadIdx.x; k < (S.ns + 7) / 8; k += BT) chunk_cp16(slot + 8 * k, L.cu_slots + s0 + 8 * k);
    asm volatile("cp.async.commit_group;" ::: "memory");
    S.soff = soff;
    S.slot = slot;
    return S;
}
__device__ __forceinline__ void chunk_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Block-wide: the chunk's values of x into xu (the caller places the barrier).
// Eight DOFs of a thread at a time, so a chunk waits for its list and for x once
// or twice instead of once per DOF of a thread.  x may be written by the kernel ahead
// of a dependent launch, so it is read by ordinary loads (pdl_wait, fg_common.cuh).
template <typename T, int BT>
__device__ __forceinline__ void chunk_load_x(const ChunkLists &L, int c, const T *x, T *xu, int constrained) {
    const int u0 = __ldg(L.cu_off + c), nu = __ldg(L.cu_n + c);
    for (int k0 = threadIdx.x; k0 < nu; k0 += 8 * BT) {
        int32_t d[8];
        T v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) d[u] = k0 + u * BT < nu ? __ldg(L.cu_dof + u0 + k0 + u * BT) : 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = k0 + u * BT < nu ? x[d[u] & INT32_MAX] : T(0);
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (k0 + u * BT < nu) xu[k0 + u * BT] = constrained && d[u] < 0 ? T(0) : v[u];
    }
}

// Block-wide (BT threads), after a barrier that follows both the element phase
// (ys complete) and chunk_wait: per DOF of the chunk the sum of its slots in
// the listed order, stored (owned) or as the partial (shared).
template <typename T, int BT>
__device__ __forceinline__ void chunk_sums(const ChunkLists &L, const ChunkStage &S, const T *ys, const T *x, T *y,
                                           int accumulate, int constrained, int diag) {
    T *part = reinterpret_cast<T *>(L.part);
    for (int k = threadIdx.x; k < S.nu; k += BT) {
        T s = T(0);
        const int j1 = k + 1 < S.nu ? S.soff[k + 1] : S.ns;
        for (int j = S.soff[k]; j < j1; ++j) s += ys[S.slot[j]];
        if (k >= S.own) {
            part[S.part0 + k - S.own] = s;
        } else {
            const int32_t f = __ldg(L.cu_dof + S.u0 + k), d = f & INT32_MAX;
            if (constrained && f < 0) s = diag ? T(1) : x[d];
            y[d] = accumulate ? y[d] + s : s;
        }
    }
}

// DOFs not owned by a single chunk: the partials of their chunks in chunk order
template <typename T>
__global__ void chunk_shared_kernel(const ChunkLists L, const T *x, T *y, int accumulate,
                                    int constrained, int diag, const int *skip) {
    pdl_wait();
    if (skip && *skip) return;
    const T *part = reinterpret_cast<const T *>(L.part);
    for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < L.n_shared;
         k += (int64_t)gridDim.x * blockDim.x) {
        const int32_t f = L.sh_dof[k], d = f & INT32_MAX;
        T s = T(0);
#pragma unroll 4
        for (int j = L.sh_off[k]; j < L.sh_off[k + 1]; ++j) s += part[L.sh_idx[j]];
        if (constrained && f < 0) s = diag ? T(1) : x[d];
        y[d] = accumulate ? y[d] + s : s;
    }
}

}  // namespace fg
