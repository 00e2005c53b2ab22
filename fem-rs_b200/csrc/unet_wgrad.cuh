// unet_wgrad.cuh -- weight and bias gradients of every convolution of the
// network in one launch (and one launch that adds the partial sums).
//
//   dW[co][tap][ci] = sum_v dY[v][co] X[v + off(tap)][ci],   db[co] = sum_v dY[v][co]
//
// as GEMMs whose K dimension is the voxels, on the BF16 tensor cores
// (mma.sync m16n8k16, FP32 accumulators).
//
// What bounds it: 3.5 GFLOP and 20 MB of activations on a 33^3 volume, all in
// L2, so the launch is bound by how many voxels are in flight, not by the
// tensor cores.  The per-fragment gathers of the form before this one (one
// thread per output-channel tile walking 4096 voxels through global memory
// with an index division and a bounds test per element) took 4.0 ms of a
// 5.0 ms pass.  Loss and gradients of one 33^3 sample, gradients copied to the
// host: 5.53 ms before, 1.06 ms with this kernel (0.79 ms with the batched convolution
// loads, the fused ReLU backward and the single copy that came later) (the bias gradients, 16 launches
// of 12 us, went with it).
//
// Split.  A block owns (layer, voxel split, tap plane dz, group of n-tiles).  It
// walks its share of the layer's voxel tiles (a patch of TX x TY voxels of one z
// plane): the patch of dY and the patch of X at z + dz with a one-voxel halo
// are copied to shared memory with 16-byte cp.async (zero-filled outside the
// volume), double buffered; all nine taps of the plane then read their operand
// from the same X patch by a row offset, so X is fetched three times in all (once
// per dz) instead of 27.  Both operands are stored voxel-major with channels
// contiguous, the transposed fragments come from ldmatrix.trans; the row pitch is
// an odd number of 16-byte units, so the eight rows of a fragment fall in
// different banks.  The accumulators (MT m-tiles of 16 output channels x NPW
// n-tiles of 8 (tap, input channel) columns per warp) stay in registers over all
// of the block's tiles.  The bias is one more column whose operand is the
// constant 1.  The partials of the splits are added in split order: the same sums
// every run.  A split is at most WG_CHAIN voxels, so that the FP32 accumulators of a large
// volume take no more steps than those of a small one: on 129^3 the error of the last
// layer's sums is 5.8e-7 (5.8e-6 with four blocks per SM over all layers), 16.4 -> 15.9 ms.
#pragma once
#include "unet_kernels.cuh"

namespace fg {

constexpr int WG_THREADS = 256, WG_NPW = 4, WG_MAXL = 9;
constexpr int WG_TILE = 144;  // voxels per patch (nine k16 steps)
constexpr int WG_CHAIN = 4096;  // voxels of one partial sum, at most

struct WgLayer {
    TView in, dy;
    Vol V;
    int cin, cout;
    int TX, TY, ntx, nty, ntiles;  // voxel patches: (batch, z, y tile, x tile), x fastest
    int groups, tpg;               // n-tile groups of one dz plane, n-tiles per group
    int splits, blk0;              // voxel splits; first block of the layer
    int64_t part0;                 // first float of the layer's partials [split][cout][27 cin + 1]
    float *gw, *gb;                // results: [cout][kp], [cout]
    int kp;
    int red0;                      // first element of the layer in the reduction
};
struct WgArgs {
    WgLayer L[WG_MAXL];
    int n;
    float *part;
};

__host__ __device__ inline int wg_c8(int cin) { return (cin + 7) / 8; }
__host__ __device__ inline int wg_pitch(int c8) { return c8 | 1; }  // 16-byte units, odd
__host__ __device__ inline int wg_co16(int cout) { return (cout + 15) / 16; }
// Shared memory (16-byte units) of one stage: X rows (+ one zero row), dY rows (+ one zero row)
__host__ __device__ inline int wg_stage_units(const WgLayer &l) {
    return ((l.TX + 2) * (l.TY + 2) + 1) * wg_pitch(wg_c8(l.cin)) + (l.TX * l.TY + 1) * wg_pitch(2 * wg_co16(l.cout));
}

__device__ __forceinline__ void wg_cp16(uint32_t dst, const void *src, bool ok) {
    const int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void wg_ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

// Eight channels c .. c+7 of voxel vox (ok: inside the volume) into shared
// memory; channels >= C are zero.
__device__ __forceinline__ void wg_load8(uint32_t dst, const TView &t, int64_t vox, int c, int C, bool ok, bool vec) {
    if (vec) {
        wg_cp16(dst, ok && c < C ? t.p + vox * t.cs + t.co + c : t.p, ok && c < C);
        return;
    }
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        w[k] = ok && c + 2 * k < C ? ld_bf16x2(t.p + vox * t.cs + t.co + c + 2 * k) : 0u;
    asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}

__global__ void __launch_bounds__(WG_THREADS, 2) conv3_wgrad_all_kernel(const __grid_constant__ WgArgs A) {
    extern __shared__ __align__(128) unsigned char wg_smem[];
    __shared__ uint16_t rowx[2][WG_TILE], rowd[2][WG_TILE];  // voxel of the patch -> row of X (tap 0,0), of dY
    __shared__ int kmax[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int li = 0;
    while (li + 1 < A.n && (int)blockIdx.x >= A.L[li + 1].blk0) ++li;
    const WgLayer &L = A.L[li];
    int rem = (int)blockIdx.x - L.blk0;
    const int split = rem / (3 * L.groups);
    rem -= split * 3 * L.groups;
    const int dz = rem / L.groups, group = rem - dz * L.groups;
    const int cin = L.cin, cout = L.cout, c8 = wg_c8(cin), MT = wg_co16(cout);
    const int px = wg_pitch(c8), pd = wg_pitch(2 * MT);
    const int TX = L.TX, TY = L.TY, RX = TX + 2, nxr = RX * (TY + 2);
    const Vol V = L.V;
    const uint32_t s0 = smem_u32(wg_smem);
    const uint32_t xbytes = (uint32_t)(nxr + 1) * px * 16, stage = xbytes + (uint32_t)(TX * TY + 1) * pd * 16;
    const bool vx = cin % 8 == 0 && L.in.cs % 8 == 0 && L.in.co % 8 == 0;
    const bool vd = cout % 8 == 0 && L.dy.cs % 8 == 0 && L.dy.co % 8 == 0;
    // zero rows (voxels beyond the patch)
    for (int s = 0; s < 2; ++s) {
        for (int k = tid; k < px; k += WG_THREADS)
            asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(s0 + s * stage + (nxr * px + k) * 16), "r"(0) : "memory");
        for (int k = tid; k < pd; k += WG_THREADS)
            asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};" ::"r"(s0 + s * stage + xbytes + (TX * TY * pd + k) * 16), "r"(0)
                         : "memory");
    }
    const int t0 = (int)((int64_t)L.ntiles * split / L.splits), t1 = (int)((int64_t)L.ntiles * (split + 1) / L.splits);
    auto load = [&](int t, int s) {
        const int tx = t % L.ntx, ty = (t / L.ntx) % L.nty, bz = t / (L.ntx * L.nty);
        const int z = bz % V.Z, b = bz / V.Z, x0 = tx * TX, y0 = ty * TY;
        const int ax = min(TX, V.X - x0), ay = min(TY, V.Y - y0);  // voxels of a ragged last patch
        const uint32_t sx = s0 + s * stage, sd = sx + xbytes;
        const int zz = z + dz - 1;
        const bool zok = zz >= 0 && zz < V.Z;
        for (int i = tid; i < nxr * c8; i += WG_THREADS) {
            const int r = i / c8, c = i - r * c8, ry = r / RX, rx = r - ry * RX;
            const int yy = y0 + ry - 1, xx = x0 + rx - 1;
            const bool ok = zok && yy >= 0 && yy < V.Y && xx >= 0 && xx < V.X;
            wg_load8(sx + (r * px + c) * 16, L.in, ok ? (((int64_t)b * V.Z + zz) * V.Y + yy) * V.X + xx : 0, c * 8, cin, ok, vx);
        }
        for (int i = tid; i < TX * TY * 2 * MT; i += WG_THREADS) {
            const int r = i / (2 * MT), c = i - r * 2 * MT, ry = r / TX, rx = r - ry * TX;
            const bool ok = ry < ay && rx < ax;
            wg_load8(sd + (r * pd + c) * 16, L.dy,
                     ok ? (((int64_t)b * V.Z + z) * V.Y + y0 + ry) * V.X + x0 + rx : 0, c * 8, cout, ok, vd);
        }
        for (int v = tid; v < WG_TILE; v += WG_THREADS) {
            const int ry = v / ax, rx = v - ry * ax;
            rowx[s][v] = (uint16_t)(ry < ay ? (ry + 1) * RX + rx + 1 : nxr);
            rowd[s][v] = (uint16_t)(ry < ay ? ry * TX + rx : TX * TY);
        }
        if (tid == 0) kmax[s] = (ax * ay + 15) / 16;
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // this warp's n-tiles: j = 9 taps x c8 channel blocks of the plane
    const int jb = group * L.tpg, jn = min(L.tpg, 9 * c8 - jb);
    int rofs[WG_NPW], cofs[WG_NPW];  // row offset of the tap, 16-byte unit of the channel block
#pragma unroll
    for (int i = 0; i < WG_NPW; ++i) {
        const int j = jb + min(warp + 8 * i, jn - 1), tap = j / c8;
        rofs[i] = (tap / 3 - 1) * RX + tap % 3 - 1;
        cofs[i] = j - tap * c8;
    }
    const bool bias = dz == 1 && group == 0 && warp == 7;
    float acc[4][WG_NPW][4], ab[4][4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
#pragma unroll
        for (int e = 0; e < 4; ++e) ab[m][e] = 0.f;
#pragma unroll
        for (int i = 0; i < WG_NPW; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[m][i][e] = 0.f;
    }
    const int nt = warp < jn ? (jn - warp + 7) / 8 : 0;  // n-tiles of this warp (<= WG_NPW)
    if (t0 < t1) load(t0, 0);
    for (int t = t0; t < t1; ++t) {
        const int s = (t - t0) & 1;
        if (t + 1 < t1) {
            load(t + 1, s ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint32_t sx = s0 + s * stage, sd = sx + xbytes;
        const int nk = kmax[s];
        for (int k = 0; k < nk; ++k) {
            // lane's row of the fragments: matrices (voxels 0-7, c 0-7), (0-7, 8-15), (8-15, 0-7), (8-15, 8-15) of dY
            // and (voxels 0-7, tile i), (8-15, tile i), (0-7, tile i+1), (8-15, tile i+1) of X
            const int rd = rowd[s][k * 16 + (lane >> 4) * 8 + (lane & 7)];
            const int rx = rowx[s][k * 16 + ((lane >> 3) & 1) * 8 + (lane & 7)];
            uint32_t a[4][4];
#pragma unroll
            for (int m = 0; m < 4; ++m)
                if (m < MT) wg_ldsm4t(a[m], sd + (rd * pd + 2 * m + ((lane >> 3) & 1)) * 16);
#pragma unroll
            for (int i = 0; i < WG_NPW; i += 2) {
                if (i < nt) {
                    const int h = i + (i + 1 < WG_NPW ? (lane >> 4) : 0);
                    const int ro = h == i ? rofs[i] : rofs[i + 1 < WG_NPW ? i + 1 : i];
                    const int cu = h == i ? cofs[i] : cofs[i + 1 < WG_NPW ? i + 1 : i];
                    const int row = rx == nxr ? nxr : rx + ro;
                    uint32_t b[4];
                    wg_ldsm4t(b, sx + (row * px + cu) * 16);
#pragma unroll
                    for (int m = 0; m < 4; ++m)
                        if (m < MT) {
                            mma_bf16_16816(acc[m][i], a[m], b[0], b[1]);
                            if (i + 1 < WG_NPW) mma_bf16_16816(acc[m][i + 1 < WG_NPW ? i + 1 : i], a[m], b[2], b[3]);
                        }
                }
            }
            if (bias)
#pragma unroll
                for (int m = 0; m < 4; ++m)
                    if (m < MT) mma_bf16_16816(ab[m], a[m], 0x3f803f80u, 0x3f803f80u);
        }
        __syncthreads();  // the stage is free for the load of the tile after the next
    }
    const int gid = lane >> 2, t4 = lane & 3, NC = 27 * cin + 1;
    float *pp = A.part + L.part0 + (int64_t)split * cout * NC;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        if (m >= MT) continue;
#pragma unroll
        for (int i = 0; i < WG_NPW; ++i) {
            if (i >= nt) continue;
            const int j = jb + warp + 8 * i, tap = j / c8, ci = (j - tap * c8) * 8 + 2 * t4;
            if (ci >= cin) continue;  // cin is even: the pair exists or does not
            float *q = pp + (dz * 9 + tap) * cin + ci;
            const int co = m * 16 + gid;
            if (co < cout) {
                q[(int64_t)co * NC] = acc[m][i][0];
                q[(int64_t)co * NC + 1] = acc[m][i][1];
            }
            if (co + 8 < cout) {
                q[(int64_t)(co + 8) * NC] = acc[m][i][2];
                q[(int64_t)(co + 8) * NC + 1] = acc[m][i][3];
            }
        }
        if (bias && t4 == 0) {
            const int co = m * 16 + gid;
            if (co < cout) pp[(int64_t)co * NC + NC - 1] = ab[m][0];
            if (co + 8 < cout) pp[(int64_t)(co + 8) * NC + NC - 1] = ab[m][2];
        }
    }
}

// gw / gb of every layer: the splits' partials in split order
__global__ void __launch_bounds__(256) conv3_wgrad_all_reduce(const __grid_constant__ WgArgs A, int total) {
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        int li = 0;
        while (li + 1 < A.n && e >= A.L[li + 1].red0) ++li;
        const WgLayer &L = A.L[li];
        const int NC = 27 * L.cin + 1, i = e - L.red0, co = i / NC, k = i - co * NC;
        const float *p = A.part + L.part0 + i;
        const int64_t step = (int64_t)L.cout * NC;
        float s = 0.f;
#pragma unroll 8
        for (int c = 0; c < L.splits; ++c) s += p[c * step];
        if (k < NC - 1) L.gw[(int64_t)co * L.kp + k] = s;
        else L.gb[co] = s;
    }
}

}  // namespace fg
