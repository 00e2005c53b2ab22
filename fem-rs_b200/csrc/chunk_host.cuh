// chunk_host.cuh -- device copies of a chunk plan (chunk_plan.h), owned by an
// unstructured operator's handle.
#pragma once
#include "chunk_plan.h"
#include "chunk_scatter.cuh"

struct ChunkBufs {
    int32_t *cu_off = nullptr, *cu_n = nullptr, *cu_own = nullptr, *cu_part = nullptr, *cu_s0 = nullptr,
            *cu_ns = nullptr, *cu_dof = nullptr, *sh_dof = nullptr, *sh_off = nullptr, *sh_idx = nullptr;
    uint16_t *cu_soff = nullptr, *cu_slots = nullptr, *lmap = nullptr;
    int64_t n_shared = 0;
    int max_nu = 0;

    template <typename V> static int up(V **dst, const std::vector<V> &v) {
        CK(cudaMalloc(dst, sizeof(V) * std::max<size_t>(v.size(), 1)));
        if (!v.empty()) CK(cudaMemcpy(*dst, v.data(), sizeof(V) * v.size(), cudaMemcpyHostToDevice));
        return FG_OK;
    }
    int upload(const fg::ChunkPlan &P) {
        n_shared = (int64_t)P.sh_dof.size();
        max_nu = P.max_nu;
        int rc;
        if ((rc = up(&cu_off, P.cu_off)) || (rc = up(&cu_n, P.cu_n)) || (rc = up(&cu_own, P.cu_own)) ||
            (rc = up(&cu_part, P.cu_part)) || (rc = up(&cu_s0, P.cu_s0)) || (rc = up(&cu_ns, P.cu_ns)) ||
            (rc = up(&cu_dof, P.cu_dof)) || (rc = up(&sh_dof, P.sh_dof)) || (rc = up(&sh_off, P.sh_off)) ||
            (rc = up(&sh_idx, P.sh_idx)) || (rc = up(&cu_soff, P.cu_soff)) || (rc = up(&cu_slots, P.cu_slots)) ||
            (rc = up(&lmap, P.lmap)))
            return rc;
        FG_LEGACY_FENCE();
        return FG_OK;
    }
    void release() {
        void *p[] = {cu_off, cu_n, cu_own, cu_part, cu_s0, cu_ns, cu_dof, sh_dof, sh_off, sh_idx, cu_soff, cu_slots, lmap};
        for (void *q : p)
            if (q) cudaFree(q);
        *this = ChunkBufs{};
    }
    fg::ChunkLists device(void *part) const {
        return fg::ChunkLists{cu_off, cu_n, cu_own, cu_part, cu_s0, cu_ns, cu_dof, cu_soff, cu_slots, lmap,
                              part, sh_dof, sh_off, sh_idx, n_shared, max_nu};
    }
};
