// chunk_plan.h -- host-side plan of the chunked gather and deterministic
// scatter shared by the unstructured operators (tetrahedra, Hex8).
//
// The elements are put in a Morton order of their centroids and cut into
// chunks of CE consecutive elements, one CTA each.  Per chunk the plan lists
// the DOFs its elements touch, each with its element-local slots
// i * CE + e_local (ascending), and marks a DOF *owned* when all of its elements
// lie in that chunk; the owned DOFs come first, both parts ascending.  Every
// other DOF -- touched by several chunks, or by none -- gets one partial per
// touching chunk: a chunk's partials are contiguous, in the order of its list,
// and chunk_shared_kernel (chunk_scatter.cuh) adds a DOF's partials in chunk
// order through an index list.  The element map is stored as positions in the
// chunk's list (16 bits), so the apply reads each DOF of the chunk once and the
// elements take their values from shared memory.
#pragma once
#include <algorithm>
#include <cstdint>
#include <vector>

namespace fg {

// Morton key of a point in the box [lo, lo + ext): 21 bits per axis, interleaved
inline uint64_t morton_key(const double *p, const double *lo, const double *ext) {
    uint64_t key = 0;
    uint32_t v[3];
    for (int a = 0; a < 3; ++a) {
        double f = ext[a] > 0.0 ? (p[a] - lo[a]) / ext[a] : 0.0;
        f = std::min(std::max(f, 0.0), 1.0);
        v[a] = (uint32_t)std::min<double>(f * 2097152.0, 2097151.0);
    }
    for (int b = 20; b >= 0; --b)
        for (int a = 0; a < 3; ++a) key = (key << 1) | ((v[a] >> b) & 1u);
    return key;
}

// perm[n] = the element at position n of the Morton order of the centroids
// cen[E][3] (stable: ties keep the caller's order)
inline void morton_order(const std::vector<double> &cen, int64_t E, std::vector<int32_t> &perm) {
    double lo[3] = {1e300, 1e300, 1e300}, hi[3] = {-1e300, -1e300, -1e300};
    for (int64_t e = 0; e < E; ++e)
        for (int a = 0; a < 3; ++a) {
            lo[a] = std::min(lo[a], cen[3 * e + a]);
            hi[a] = std::max(hi[a], cen[3 * e + a]);
        }
    const double ext[3] = {hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]};
    std::vector<uint64_t> key(E);
    for (int64_t e = 0; e < E; ++e) key[e] = morton_key(&cen[3 * e], lo, ext);
    perm.resize(E);
    for (int64_t e = 0; e < E; ++e) perm[e] = (int32_t)e;
    std::stable_sort(perm.begin(), perm.end(), [&](int32_t a, int32_t b) { return key[a] < key[b]; });
}

constexpr int32_t CHUNK_ESS = INT32_MIN;  // sign bit of a listed DOF: essential

struct ChunkPlan {
    std::vector<int32_t> cu_off;   // [n_chunks + 1] start of each chunk's list, multiples of 8
    std::vector<int32_t> cu_n;     // [n_chunks] DOFs of the chunk
    std::vector<int32_t> cu_own;   // [n_chunks] owned ones (the first of the list)
    std::vector<int32_t> cu_part;  // [n_chunks] first partial of the chunk
    std::vector<int32_t> cu_s0;    // [n_chunks] start of each chunk's slots, multiples of 8
    std::vector<int32_t> cu_ns;    // [n_chunks] slots of the chunk
    std::vector<int32_t> cu_dof;   // DOFs (sign bit: essential); padding between chunks 0
    std::vector<uint16_t> cu_soff; // per listed DOF the start of its slots, relative to the chunk's
    std::vector<uint16_t> cu_slots;
    std::vector<uint16_t> lmap;    // [nl][Es] position of the element's DOF in its chunk's list (0 for padding elements)
    std::vector<int32_t> sh_dof, sh_off, sh_idx;  // shared DOFs, their ranges in sh_idx, partials in chunk order
    int max_nu = 0;
    int64_t n_chunks = 0, n_part = 0;
};

// smap: element map [Es][nl] in chunk order (an entry < 0: padding, no DOF);
// ess: essential-DOF mask [N] or null; requires nl * CE <= 65536 (16-bit local slots).
inline void plan_chunk_lists(const std::vector<int32_t> &smap, int64_t Es, int64_t N, int nl, int CE,
                             const uint8_t *ess, ChunkPlan &P) {
    const int64_t nch = (Es + CE - 1) / CE;
    P = ChunkPlan{};
    P.n_chunks = nch;
    // (DOF, slot) keys of every chunk, sorted; how many chunks touch each DOF
    std::vector<uint64_t> key((size_t)Es * nl);
    std::vector<int64_t> k0(nch + 1, 0);
    std::vector<int32_t> nchk(N, 0);
    for (int64_t c = 0; c < nch; ++c) {
        const int64_t e0 = c * CE;
        const int ne = (int)std::min<int64_t>(CE, Es - e0);
        int64_t n = k0[c];
        for (int el = 0; el < ne; ++el)
            for (int i = 0; i < nl; ++i) {
                const int32_t d = smap[(size_t)(e0 + el) * nl + i];
                if (d >= 0) key[n++] = ((uint64_t)d << 16) | (uint32_t)(i * CE + el);
            }
        std::sort(key.begin() + k0[c], key.begin() + n);
        for (int64_t k = k0[c]; k < n; ++k)
            if (k == k0[c] || key[k] >> 16 != key[k - 1] >> 16) ++nchk[key[k] >> 16];
        k0[c + 1] = n;
    }
    P.cu_off.assign(1, 0);
    P.lmap.assign((size_t)Es * nl, 0);
    P.cu_slots.reserve((size_t)Es * nl + 8 * nch);
    std::vector<int32_t> shared_of;  // DOF of each partial
    for (int64_t c = 0; c < nch; ++c) {
        const size_t d0 = P.cu_dof.size(), s0 = P.cu_slots.size();
        P.cu_part.push_back((int32_t)shared_of.size());
        P.cu_s0.push_back((int32_t)s0);
        for (int pass = 0; pass < 2; ++pass) {
            for (int64_t k = k0[c]; k < k0[c + 1];) {
                const int32_t d = (int32_t)(key[k] >> 16);
                int64_t k1 = k + 1;
                while (k1 < k0[c + 1] && (int32_t)(key[k1] >> 16) == d) ++k1;
                if ((nchk[d] == 1) == (pass == 0)) {
                    const uint16_t pos = (uint16_t)(P.cu_dof.size() - d0);
                    P.cu_soff.push_back((uint16_t)(P.cu_slots.size() - s0));
                    P.cu_dof.push_back(d | (ess && ess[d] ? CHUNK_ESS : 0));
                    if (pass) shared_of.push_back(d);
                    for (; k < k1; ++k) {
                        const int slot = (int)(key[k] & 0xffff);
                        P.cu_slots.push_back((uint16_t)slot);
                        P.lmap[(size_t)(slot / CE) * Es + c * CE + slot % CE] = pos;
                    }
                }
                k = k1;
            }
            if (!pass) P.cu_own.push_back((int32_t)(P.cu_dof.size() - d0));
        }
        const int nu = (int)(P.cu_dof.size() - d0);
        P.cu_n.push_back(nu);
        P.max_nu = std::max(P.max_nu, nu);
        P.cu_ns.push_back((int32_t)(P.cu_slots.size() - s0));
        while (P.cu_dof.size() % 8) P.cu_dof.push_back(0), P.cu_soff.push_back(0);
        while (P.cu_slots.size() % 8) P.cu_slots.push_back(0);
        P.cu_off.push_back((int32_t)P.cu_dof.size());
    }
    P.n_part = (int64_t)shared_of.size();
    std::vector<int32_t> base(N, -1);
    P.sh_off.assign(1, 0);
    for (int64_t d = 0; d < N; ++d)
        if (nchk[d] != 1) {
            base[d] = P.sh_off.back();
            P.sh_dof.push_back((int32_t)d | (ess && ess[d] ? CHUNK_ESS : 0));
            P.sh_off.push_back(P.sh_off.back() + nchk[d]);
        }
    P.sh_idx.resize((size_t)P.n_part);
    for (int64_t k = 0; k < P.n_part; ++k) P.sh_idx[(size_t)base[shared_of[(size_t)k]]++] = (int32_t)k;  // chunks in order
}

}  // namespace fg
