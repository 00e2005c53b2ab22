// tet_kernels.cuh -- partial-assembly operator on unstructured tetrahedra
// (TetP1 / TetP2 / TetP3), the element path of crates/assembly/src/partial.rs
// on Tet4.
//
// Per quadrature point the reference computes grad_phys = J^-T grad_ref and
// y_i += w |det J| kappa (grad u . grad phi_i); with the affine map this is
// y_i += (w kappa) grad_ref phi_i . G grad_ref u, G = |det J| J^-1 J^-T
// (constant per element), which the apply evaluates.
//
// Moment form (diffusion, P1 and P2).  The reference gradients of P1/P2 are
// affine in xi: grad_ref u(xi) = g0 + H xi (H symmetric, the Hessian of u; 0
// for P1).  With s_q = w_q kappa_q c_k the quadrature sum is then exactly
//   y_i = a_i . G M0 + sum_k B_i[:,k] . G M_k,   grad_ref phi_i = a_i + B_i xi,
//   M0 = S00 g0 + H s1,   M_k = s1_k g0 + H S2[:,k],
// with the per-element moments S00 = sum s_q, s1 = sum s_q xi_q and
// S2 = sum s_q xi_q xi_q^T (10 numbers, P1: S00 only), so the apply reads 10
// numbers per element instead of nq point scalars and does ~160 FMAs instead
// of ~70 nq.  The mass term, P3 and the diagonal use the point form.
//
// Layout (element-major structure of arrays in a locality order of the
// elements, one coalesced load per component across a warp):
//   G    [6][E]    |det J| J^-1 J^-T (xx xy xz yy yz zz)
//   Sm   [10][E]   diffusion moments (S00, s1, S2 as xx xy xz yy yz zz); P1: [6][E] S00 G
//   sk   [nq][E]   w_q kappa_q c_k          (diffusion, point form)
//   sm   [nq][E]   w_q |det J| rho_q c_m    (mass)
//   lmap [nl][E]   16-bit position of the local DOF in its chunk's DOF list
//
// Scatter without float atomics and without an element-result array in HBM:
// the elements, sorted along a Morton curve of their centroids, form chunks
// of CE elements, one CTA each.  A chunk computes its element results into
// shared memory and sums, per DOF of its list, the element-local slots of
// that DOF in increasing (local index, element) order.  A DOF whose elements all lie in the chunk is
// stored directly; a DOF shared with other chunks gets one partial sum per
// chunk, and chunk_shared_kernel adds the partials of each such DOF in
// increasing chunk order (chunk_plan.h, chunk_scatter.cuh).  The result is
// deterministic.
#pragma once
#include "chunk_scatter.cuh"
#include "fg_common.cuh"

namespace fg {

constexpr int TET_MAXQ = 35;  // Grundmann-Moller s = 3

struct TetRule {
    int nq;
    const double *phi;   // [nq][nl] basis values at the points
    const double *grad;  // [nq][nl][3] reference gradients
};

struct TetArgs {
    int64_t E, N;
    int kind;                  // bit 1 mass, bit 2 diffusion
    const int32_t *dofs;       // [nl][E] caller's element order
    const double *G;           // [6][E]
    const double *sk, *sm;     // [nq][E]
    TetRule R;
};

// Chunked apply: element data in the chunk order, chunk DOF lists.
struct TetChunk {
    int64_t E, N;
    int CE;                      // elements per chunk
    const double *G, *Sm;        // [6][E], [10][E] (P1: [6][E] S00 G)
    const double *sk, *sm;       // [nq][E]
    ChunkLists L;
};

// one thread per element: geometry and the per-point scalars
__global__ void tet_setup_kernel(TetArgs A, int nl, const double *__restrict__ coords,
                                 const double *__restrict__ qw, const double *__restrict__ kappa_q, double kappa_c,
                                 const double *__restrict__ rho_q, double rho_c, double c_m, double c_k,
                                 double *G, double *sk, double *sm, int *err) {
    const int64_t E = A.E;
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < E; e += (int64_t)gridDim.x * blockDim.x) {
        const double *x0 = coords + 3 * (int64_t)A.dofs[e];
        double J[3][3];
        for (int c = 0; c < 3; ++c) {
            const double *xc = coords + 3 * (int64_t)A.dofs[(int64_t)(c + 1) * E + e];
            for (int r = 0; r < 3; ++r) J[r][c] = xc[r] - x0[r];
        }
        const double det = J[0][0] * (J[1][1] * J[2][2] - J[1][2] * J[2][1]) -
                           J[0][1] * (J[1][0] * J[2][2] - J[1][2] * J[2][0]) +
                           J[0][2] * (J[1][0] * J[2][1] - J[1][1] * J[2][0]);
        if (!(fabs(det) > 0.0)) atomicOr(err, FG_DERR_BOUNDS);
        double inv[3][3];
        inv[0][0] = (J[1][1] * J[2][2] - J[1][2] * J[2][1]) / det;
        inv[0][1] = (J[0][2] * J[2][1] - J[0][1] * J[2][2]) / det;
        inv[0][2] = (J[0][1] * J[1][2] - J[0][2] * J[1][1]) / det;
        inv[1][0] = (J[1][2] * J[2][0] - J[1][0] * J[2][2]) / det;
        inv[1][1] = (J[0][0] * J[2][2] - J[0][2] * J[2][0]) / det;
        inv[1][2] = (J[0][2] * J[1][0] - J[0][0] * J[1][2]) / det;
        inv[2][0] = (J[1][0] * J[2][1] - J[1][1] * J[2][0]) / det;
        inv[2][1] = (J[0][1] * J[2][0] - J[0][0] * J[2][1]) / det;
        inv[2][2] = (J[0][0] * J[1][1] - J[0][1] * J[1][0]) / det;
        const double ad = fabs(det);
        const int mi[6] = {0, 0, 0, 1, 1, 2}, ni[6] = {0, 1, 2, 1, 2, 2};
        for (int k = 0; k < 6; ++k) {
            const int m = mi[k], n = ni[k];
            G[(int64_t)k * E + e] = ad * (inv[m][0] * inv[n][0] + inv[m][1] * inv[n][1] + inv[m][2] * inv[n][2]);
        }
        for (int q = 0; q < A.R.nq; ++q) {
            if (A.kind & 2) sk[(int64_t)q * E + e] = qw[q] * (kappa_q ? kappa_q[e * A.R.nq + q] : kappa_c) * c_k;
            if (A.kind & 1) sm[(int64_t)q * E + e] = qw[q] * ad * (rho_q ? rho_q[e * A.R.nq + q] : rho_c) * c_m;
        }
        (void)nl;
    }
}

// ---- point form on the FP64 tensor cores ------------------------------------
// The point form is two small GEMMs per element with the rule's tables as the
// fixed operand: values and reference gradients at the points, V = x T (K = the
// NL local DOFs), then, after the point scalars and G, y = W T^T (K = the points).
// mma.m8n8k4 (FP64, fused multiply-adds) takes eight elements as its rows: a lane
// holds element lane / 4, local DOFs 4 ks + lane % 4 of x as the first operand, and gets
// the points 8 t + 2 (lane % 4) + {0, 1} of each table in the same accumulator
// registers, so the point scalars apply without moving data.  The second product
// takes those registers as they are: k-step j of a block of eight points holds
// points 8 t + 2 (lane % 4) + j, and the table is stored in that order.
//
// What bounds it: the FP64 rate once enough warps are there.  One thread per
// element (the form before) ran 5,600 multiply-adds a P3 element behind indexed
// constant loads with 234 registers: 8 warps per SM, the pipe a quarter busy.
// 48,000 P3 tetrahedra, mass + diffusion, 35 points: 122 -> 46.7 us (chunks of 128
// elements; 256: 82, 64: 47); 280,000 P1, 15 points: 80.8 -> 44.7.  The error against
// 64-bit sums in another order is unchanged (1.7e-14).
//
// Tables in fragment order (tet_point_tables): TF [t][table][ks][lane] =
// table(point 8 t + lane / 4, DOF 4 ks + lane % 4) and TB [t][table][j][it][lane] =
// table(point 8 t + 2 (lane % 4) + j, DOF 8 it + lane / 4), zero beyond the rule and
// the element; tables: the gradient components (diffusion), then the values (mass).
template <int NL> struct TetPoint {
    static constexpr int KS = (NL + 3) / 4, IT = (NL + 7) / 8;
};

__device__ __forceinline__ void dmma_884(double (&c)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

// Diagonal of element e of the chunk order (a set-up kernel: one thread per element).
template <int NL>
__device__ __forceinline__ void tet_elem_diag(const TetChunk &C, int kind, int nq, const TetRule &R, int64_t e,
                                              double (&ye)[NL]) {
    const int64_t E = C.E;
#pragma unroll
    for (int i = 0; i < NL; ++i) ye[i] = 0.0;
    double g[6] = {0, 0, 0, 0, 0, 0};
    if (kind & 2)
#pragma unroll
        for (int k = 0; k < 6; ++k) g[k] = __ldg(C.G + (int64_t)k * E + e);
    for (int q = 0; q < nq; ++q) {
        const double *gr = R.grad + (int64_t)q * NL * 3, *ph = R.phi + (int64_t)q * NL;
        if (kind & 2) {
            const double s = __ldg(C.sk + (int64_t)q * E + e);
#pragma unroll
            for (int i = 0; i < NL; ++i) {
                const double a = __ldg(gr + 3 * i), b = __ldg(gr + 3 * i + 1), c = __ldg(gr + 3 * i + 2);
                ye[i] += s * (g[0] * a * a + g[3] * b * b + g[5] * c * c + 2.0 * (g[1] * a * b + g[2] * a * c + g[4] * b * c));
            }
        }
        if (kind & 1) {
            const double m = __ldg(C.sm + (int64_t)q * E + e);
#pragma unroll
            for (int i = 0; i < NL; ++i) ye[i] += m * __ldg(ph + i) * __ldg(ph + i);
        }
    }
}

// Element diffusion result by the moment form (P1: NL = 4, P2: NL = 10).
// Gradients of the TetP1/TetP2 bases of crates/element/src/lagrange/tet.rs in
// barycentric form (l1 = 1 - x - y - z): vertex i grad (4 l_i - 1) grad l_i,
// edge (i, j) grad 4 l_i l_j; their coefficients of 1, x, y, z give g0, H and
// the a_i, B_i below.
template <int NL> struct TetMom { static constexpr int n = NL == 4 ? 6 : 16; };

// The element's moment-form data: P1 the 6 entries of S00 G, P2 G (6) and the
// 10 moments.
template <int NL>
__device__ __forceinline__ void tet_load_moments(const TetChunk &C, int64_t e, double (&md)[TetMom<NL>::n]) {
    const int64_t E = C.E;
    if constexpr (NL == 4) {
#pragma unroll
        for (int k = 0; k < 6; ++k) md[k] = __ldg(C.Sm + (int64_t)k * E + e);
    } else {
#pragma unroll
        for (int k = 0; k < 6; ++k) md[k] = __ldg(C.G + (int64_t)k * E + e);
#pragma unroll
        for (int k = 0; k < 10; ++k) md[6 + k] = __ldg(C.Sm + (int64_t)k * E + e);
    }
}

template <int NL>
__device__ __forceinline__ void tet_elem_moments(const double (&md)[TetMom<NL>::n], const double (&u)[NL],
                                                 double (&y)[NL]) {
    const double *G = md;
    auto Gv = [&](const double (&m)[3], double (&v)[3]) {
        v[0] = G[0] * m[0] + G[1] * m[1] + G[2] * m[2];
        v[1] = G[1] * m[0] + G[3] * m[1] + G[4] * m[2];
        v[2] = G[2] * m[0] + G[4] * m[1] + G[5] * m[2];
    };
    if constexpr (NL == 4) {
        const double g[3] = {u[1] - u[0], u[2] - u[0], u[3] - u[0]};
        double v[3];
        Gv(g, v);  // G holds S00 G
        y[0] = -(v[0] + v[1] + v[2]);
        y[1] = v[0];
        y[2] = v[1];
        y[3] = v[2];
    } else {
        const double *S = md + 6;
        // g0 and the Hessian H (xx yy zz xy xz yz)
        const double t0 = 3.0 * u[0], f0 = 4.0 * u[0];
        const double g0[3] = {4.0 * u[4] - t0 - u[1], 4.0 * u[5] - t0 - u[2], 4.0 * u[6] - t0 - u[3]};
        const double hxx = 4.0 * (u[0] + u[1]) - 8.0 * u[4];
        const double hyy = 4.0 * (u[0] + u[2]) - 8.0 * u[5];
        const double hzz = 4.0 * (u[0] + u[3]) - 8.0 * u[6];
        const double hxy = f0 + 4.0 * (u[7] - u[4] - u[5]);
        const double hxz = f0 + 4.0 * (u[8] - u[4] - u[6]);
        const double hyz = f0 + 4.0 * (u[9] - u[5] - u[6]);
        auto Hv = [&](double a, double b, double c, double (&v)[3]) {
            v[0] = hxx * a + hxy * b + hxz * c;
            v[1] = hxy * a + hyy * b + hyz * c;
            v[2] = hxz * a + hyz * b + hzz * c;
        };
        // S = (S00, s1x, s1y, s1z, S2xx, S2xy, S2xz, S2yy, S2yz, S2zz)
        double m[3], v0[3], w[3][3];  // w[k] = G M_{k+1}
        Hv(S[1], S[2], S[3], m);
#pragma unroll
        for (int c = 0; c < 3; ++c) m[c] += S[0] * g0[c];
        Gv(m, v0);
        const double s2c[3][3] = {{S[4], S[5], S[6]}, {S[5], S[7], S[8]}, {S[6], S[8], S[9]}};
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            Hv(s2c[k][0], s2c[k][1], s2c[k][2], m);
#pragma unroll
            for (int c = 0; c < 3; ++c) m[c] += S[1 + k] * g0[c];
            Gv(m, w[k]);
        }
        // W[c][k] = w[k][c]; diagonal and symmetric off-diagonal sums
        const double d0 = w[0][0], d1 = w[1][1], d2 = w[2][2];
        const double o01 = w[1][0] + w[0][1], o02 = w[2][0] + w[0][2], o12 = w[2][1] + w[1][2];
        y[0] = -3.0 * (v0[0] + v0[1] + v0[2]) + 4.0 * (d0 + d1 + d2 + o01 + o02 + o12);
        y[1] = 4.0 * d0 - v0[0];
        y[2] = 4.0 * d1 - v0[1];
        y[3] = 4.0 * d2 - v0[2];
        y[4] = 4.0 * (v0[0] - 2.0 * d0 - o01 - o02);
        y[5] = 4.0 * (v0[1] - 2.0 * d1 - o01 - o12);
        y[6] = 4.0 * (v0[2] - 2.0 * d2 - o02 - o12);
        y[7] = 4.0 * o01;
        y[8] = 4.0 * o02;
        y[9] = 4.0 * o12;
    }
}

// Shared-memory plan of a chunk (bytes): element results, the chunk's slot
// lists, its values of x.
__host__ __device__ inline size_t tet_chunk_smem(int NL, int CE, int max_nu) {
    return sizeof(double) * ((size_t)NL * CE + max_nu) + chunk_list_smem(NL, CE, max_nu);
}

// One CTA (BT threads) per chunk; diffusion by the moment form (P1, P2).  The
// copies of the chunk's slot lists are started and its values of x read once into
// shared memory; then the element results are computed into shared memory, each element
// taking its values by its 16-bit positions.  After a barrier each DOF's slots are
// summed.  On essential DOFs of a constrained call the identity row: y_d (+)= x_d (apply)
// or 1 (diagonal).  40^3 x 6 P2 tetrahedra, new vectors each pass: 41.0 us with x gathered
// per element through a 32-bit map, 30.9 us this way (with dependent launches).
template <int NL, int BT>
__global__ void __launch_bounds__(BT, BT == 512 ? 2 : 3) tet_moment_kernel(const TetChunk C, const double *x, double *y,
                                                                         int accumulate, int constrained) {
    extern __shared__ __align__(16) unsigned char tsm_raw[];
    const int CE = C.CE;
    double *ys = reinterpret_cast<double *>(tsm_raw);  // [NL][CE] element results
    const ChunkStage S = chunk_stage_lists<BT>(C.L, blockIdx.x, tsm_raw + sizeof(double) * NL * CE);
    double *xu = reinterpret_cast<double *>(tsm_raw + sizeof(double) * NL * CE + chunk_list_smem(NL, CE, C.L.max_nu));
    const int64_t e0 = (int64_t)blockIdx.x * CE;
    const int ne = (int)(C.E - e0 < CE ? C.E - e0 : CE);
    pdl_wait();  // the slot lists do not depend on earlier kernels
    chunk_load_x<double, BT>(C.L, blockIdx.x, x, xu, constrained);
    __syncthreads();
    for (int el = threadIdx.x; el < ne; el += BT) {
        const int64_t e = e0 + el;
        double xe[NL], ye[NL], md[TetMom<NL>::n];
        tet_load_moments<NL>(C, e, md);
#pragma unroll
        for (int i = 0; i < NL; ++i) xe[i] = xu[__ldg(C.L.lmap + (int64_t)i * C.E + e)];
        tet_elem_moments<NL>(md, xe, ye);
#pragma unroll
        for (int i = 0; i < NL; ++i) ys[i * CE + el] = ye[i];
    }
    chunk_wait();
    __syncthreads();
    chunk_sums<double, BT>(C.L, S, ys, x, y, accumulate, constrained, 0);
}

// The same chunk scheme by the point form: a warp takes 16 elements (two
// eight-row tiles that share the table operand) at a time.
template <int NL, int KIND, int BT>
__global__ void __launch_bounds__(BT) tet_point_kernel(const TetChunk C, int nq, const double *__restrict__ TF,
                                                       const double *__restrict__ TB, const double *x, double *y,
                                                       int accumulate, int constrained) {
    constexpr bool HM = (KIND & 1) != 0, HK = (KIND & 2) != 0;
    constexpr int NC = (HK ? 3 : 0) + (HM ? 1 : 0), KS = TetPoint<NL>::KS, IT = TetPoint<NL>::IT;
    extern __shared__ __align__(16) unsigned char tsm_raw[];
    const int CE = C.CE;
    const int64_t E = C.E;
    double *ys = reinterpret_cast<double *>(tsm_raw);  // [NL][CE] element results
    const ChunkStage S = chunk_stage_lists<BT>(C.L, blockIdx.x, tsm_raw + sizeof(double) * NL * CE);
    double *xu = reinterpret_cast<double *>(tsm_raw + sizeof(double) * NL * CE + chunk_list_smem(NL, CE, C.L.max_nu));
    const int64_t e0 = (int64_t)blockIdx.x * CE;
    const int ne = (int)(E - e0 < CE ? E - e0 : CE);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r8 = lane >> 2, l4 = lane & 3;
    const int QT = (nq + 7) / 8;
    pdl_wait();
    chunk_load_x<double, BT>(C.L, blockIdx.x, x, xu, constrained);
    __syncthreads();
    for (int t16 = warp * 16; t16 < ne; t16 += BT / 2) {
        double xa[2][KS], G[2][6], Y[2][IT][2];
        bool ok[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int el = t16 + 8 * p + r8;
            ok[p] = el < ne;
            const int64_t e = e0 + (ok[p] ? el : 0);
#pragma unroll
            for (int ks = 0; ks < KS; ++ks) {
                const int i = 4 * ks + l4;
                xa[p][ks] = ok[p] && i < NL ? xu[__ldg(C.L.lmap + (int64_t)i * E + e)] : 0.0;
            }
            if (HK)
#pragma unroll
                for (int k = 0; k < 6; ++k) G[p][k] = __ldg(C.G + (int64_t)k * E + e);
#pragma unroll
            for (int it = 0; it < IT; ++it) Y[p][it][0] = Y[p][it][1] = 0.0;
        }
        for (int t = 0; t < QT; ++t) {
            double sc[2][2], mc[2][2];  // point scalars of this lane's points
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int q = 8 * t + 2 * l4 + j;
                    const bool v = ok[p] && q < nq;
                    const int64_t o = (int64_t)q * E + e0 + t16 + 8 * p + r8;
                    if (HK) sc[p][j] = v ? __ldg(C.sk + o) : 0.0;
                    if (HM) mc[p][j] = v ? __ldg(C.sm + o) : 0.0;
                }
            double V[2][NC][2];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
#pragma unroll
                for (int p = 0; p < 2; ++p) V[p][c][0] = V[p][c][1] = 0.0;
#pragma unroll
                for (int ks = 0; ks < KS; ++ks) {
                    const double b = __ldg(TF + (((int64_t)t * NC + c) * KS + ks) * 32 + lane);
#pragma unroll
                    for (int p = 0; p < 2; ++p) dmma_884(V[p][c], xa[p][ks], b);
                }
            }
#pragma unroll
            for (int p = 0; p < 2; ++p)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const bool v = 8 * t + 2 * l4 + j < nq;
                    if (HK) {
                        const double gx = V[p][0][j], gy = V[p][1][j], gz = V[p][2][j], s = sc[p][j];
                        V[p][0][j] = v ? s * (G[p][0] * gx + G[p][1] * gy + G[p][2] * gz) : 0.0;
                        V[p][1][j] = v ? s * (G[p][1] * gx + G[p][3] * gy + G[p][4] * gz) : 0.0;
                        V[p][2][j] = v ? s * (G[p][2] * gx + G[p][4] * gy + G[p][5] * gz) : 0.0;
                    }
                    if (HM) V[p][NC - 1][j] = v ? mc[p][j] * V[p][NC - 1][j] : 0.0;
                }
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int it = 0; it < IT; ++it) {
                        const double b = __ldg(TB + ((((int64_t)t * NC + c) * 2 + j) * IT + it) * 32 + lane);
#pragma unroll
                        for (int p = 0; p < 2; ++p) dmma_884(Y[p][it], V[p][c][j], b);
                    }
        }
#pragma unroll
        for (int p = 0; p < 2; ++p)
            if (ok[p])
#pragma unroll
                for (int it = 0; it < IT; ++it)
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int i = 8 * it + 2 * l4 + j;
                        if (i < NL) ys[i * CE + t16 + 8 * p + r8] = Y[p][it][j];
                    }
    }
    chunk_wait();
    __syncthreads();
    chunk_sums<double, BT>(C.L, S, ys, x, y, accumulate, constrained, 0);
}

// Jacobi diagonal, one thread per element (1 on essential DOFs of a constrained call).
template <int NL, int BT>
__global__ void __launch_bounds__(BT) tet_diag_kernel(const TetChunk C, int kind, int nq, const TetRule R,
                                                      double *__restrict__ y, int constrained) {
    extern __shared__ __align__(16) unsigned char tsm_raw[];
    const int CE = C.CE;
    double *ys = reinterpret_cast<double *>(tsm_raw);
    const ChunkStage S = chunk_stage_lists<BT>(C.L, blockIdx.x, tsm_raw + sizeof(double) * NL * CE);
    const int64_t e0 = (int64_t)blockIdx.x * CE;
    const int ne = (int)(C.E - e0 < CE ? C.E - e0 : CE);
    for (int el = threadIdx.x; el < ne; el += BT) {
        double ye[NL];
        tet_elem_diag<NL>(C, kind, nq, R, e0 + el, ye);
#pragma unroll
        for (int i = 0; i < NL; ++i) ys[i * CE + el] = ye[i];
    }
    chunk_wait();
    __syncthreads();
    chunk_sums<double, BT>(C.L, S, ys, nullptr, y, 0, constrained, 1);
}

// Reorder the per-element data into the chunk order and form the diffusion
// moments from the point scalars (nmom = 10 for P2; 6 for P1, where the only
// moment S00 is stored multiplied into G; 0 otherwise).
__global__ void tet_permute_kernel(int64_t E, int nq, int kind, int nmom, const int32_t *__restrict__ perm,
                                   const double *__restrict__ qp, const double *__restrict__ G,
                                   const double *__restrict__ sk, const double *__restrict__ sm, double *Gp,
                                   double *skp, double *smp, double *Sm) {
    for (int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; n < E; n += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = perm[n];
        for (int k = 0; k < 6; ++k) Gp[(int64_t)k * E + n] = G[(int64_t)k * E + e];
        double mo[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
        for (int q = 0; q < nq; ++q) {
            if (kind & 2) {
                const double s = sk[(int64_t)q * E + e];
                skp[(int64_t)q * E + n] = s;
                const double a = qp[3 * q], b = qp[3 * q + 1], c = qp[3 * q + 2];
                mo[0] += s;
                mo[1] += s * a;
                mo[2] += s * b;
                mo[3] += s * c;
                mo[4] += s * a * a;
                mo[5] += s * a * b;
                mo[6] += s * a * c;
                mo[7] += s * b * b;
                mo[8] += s * b * c;
                mo[9] += s * c * c;
            }
            if (kind & 1) smp[(int64_t)q * E + n] = sm[(int64_t)q * E + e];
        }
        if (nmom == 6)  // P1: S00 G
            for (int k = 0; k < 6; ++k) Sm[(int64_t)k * E + n] = mo[0] * G[(int64_t)k * E + e];
        else
            for (int k = 0; k < nmom; ++k) Sm[(int64_t)k * E + n] = mo[k];
    }
}

// Gauss points in physical space: xyz[e][q][3] = x_0 + J xi_q
__global__ void tet_qp_coords_kernel(TetArgs A, const double *__restrict__ coords, const double *__restrict__ qp,
                                     double *__restrict__ xyz) {
    const int nq = A.R.nq;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < A.E * nq; t += (int64_t)gridDim.x * blockDim.x) {
        const int q = (int)(t % nq);
        const int64_t e = t / nq;
        const double *x0 = coords + 3 * (int64_t)A.dofs[e];
        const double *xi = qp + 3 * q;
        for (int r = 0; r < 3; ++r) {
            double s = x0[r];
            for (int c = 0; c < 3; ++c) {
                const double *xc = coords + 3 * (int64_t)A.dofs[(int64_t)(c + 1) * A.E + e];
                s += (xc[r] - x0[r]) * xi[c];
            }
            xyz[3 * t + r] = s;
        }
    }
}

}  // namespace fg
