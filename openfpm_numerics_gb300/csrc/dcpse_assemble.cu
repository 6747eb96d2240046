// dcpse_assemble.cu -- DC-PSE kernel assembly on the device (FP64).
//
// Replaces Dcpse::initializeStaticSize (src/DCPSE/Dcpse.hpp:690-796) and the
// reference GPU path Dcpse_gpu::assembleLocalMatrices (src/DCPSE/Dcpse.cuh:
// 620-717: per-thread global scratch B, cuBLAS batched LU without pivoting,
// a separate calcKernels_gpu pass and host round trips).
//
// eps_kernel (a thread per particle) forms
//       eps  = (sum_q sum_d |x_pq,d|) / k / HOverEpsilon   (Vandermonde.hpp:63-81)
// for every particle.  Particles are then assembled in batches, each by three
// kernels that hand their results over through a plan-owned scratch buffer:
//  1. gram_kernel (one warp per particle)
//       Gram A_ij = sum_q B_qi B_qj,  B_qj = E_q V_qj,
//            V_qj = m_j(x_pq/eps), E_q = exp(-|x_pq|^2 / (2 eps^2))
//            (Vandermonde.hpp:36-49, DcpseDiagonalScalingMatrix.hpp:21-41,
//             Dcpse.hpp:755-757).  Computed once over the union of the bases
//            of all terms (Dx,Dy,Dz share one basis, Dxx,Dyy,Dzz another);
//            each lane owns Gram entries and accumulates them over q in
//            neighbour order.  Written to scratch with a status word per
//            particle (4 bits per basis group).
//  2. qr_kernel (a group of LPP lanes per particle, 32/LPP particles per
//       warp): solve A a = b for every right-hand side of each basis with
//       column-pivoting Householder QR (Businger-Golub; the role of Eigen's
//       colPivHouseholderQr at Dcpse.hpp:766), columns split over the lanes
//       of the group.  The QR is a long chain of scalar steps (pivot search,
//       square root, divisions); with few lanes per particle one warp
//       instruction advances many particles, which is what the FP64 pipe of
//       this part needs.  Coefficients go back to scratch.
//  3. weights_kernel (a warp takes a run of particles, its lanes their
//       concatenated neighbour rows)
//       K_q = exp(-|x_pq/eps|^2) sum_i a_i V_qi        (Dcpse.hpp:768-809)
// The FP64 pipe bounds all three; products and quotients that the integer
// pipes can round (dcpse_softfp.cuh) run there beside it, with the same bits.
//
// Every floating-point operation follows the order of the CPU oracle, and
// this translation unit is compiled with -fmad=false (fused multiply-adds are
// explicit fma calls), so the FP64 kernels equal the oracle's bit for bit
// whatever the batch size, lane grouping or CTA size.  Neighbour rows are
// processed in chunks of 32 (one row per lane), so any neighbour count is
// handled with fixed shared memory.
#include <algorithm>
#include <cstdio>

#include <cuda_bf16.h>

#include <type_traits>

#include "dcpse_internal.h"
#include "dcpse_softfp.cuh"

namespace dcpse {
namespace {

constexpr int kWarps = 4;  // warps per CTA of the Gram and weight kernels
constexpr int kCh = 32;    // neighbour rows per chunk
constexpr int kQrWarps = 2;  // warps per CTA of the QR kernel

// Scratch layout and shared-memory sizes of one assembly.
struct Split {
    int gstride;             // doubles of Gram entries per particle
    int cstride;             // doubles of coefficients per particle
    int nrhs[kMaxGroups];    // right-hand sides per group (per term or per output)
    int c_off[kMaxGroups];   // coefficient block of each group, [gn][nrhs]
    int nmax;                // largest basis
    int nrmax;               // most right-hand sides of a group
    int qtab;                // Gram entries (i <= j) of all groups
    int qwords;              // doubles of the largest [A|b] plus its solution block
    int pstride;             // doubles of QR work space per particle (set per lane grouping)
    int ldb;                 // row stride of the B chunk of the Gram kernel
    int nslots;              // monomial program slots per lane
    int nout;                // outputs of the plan
    int npairs;              // Gram entries per particle
    double* gram;            // [nb][gstride]
    double* coef;            // [nb][cstride]
    double* usc;             // [nb][dim][maxk] scaled offsets u = x_pq / eps of every row
    int64_t ustride;         // dim * maxk (+ maxk with vjp: E of every row)
    bool vjp;                // position VJP: column E c of B, two right-hand sides (b~, s) per group
    int maxk;
    double* scale;           // [nb][4] eps, 1 / eps, 2 eps^2, 1 / (2 eps^2)
    int32_t* gst;            // [nb] group status words
    // tensor-core Gram (DCPSE_ASSEMBLE_TC): B of every particle of the batch
    // and the exponents of its columns' largest entries
    double* qws;             // global QR work space (one slot per lane group) or nullptr
    int* qperm;              // its column permutations
    bool tc;
    int kpad;                // row stride of bmat (maxk rounded up to 16)
    double* bmat;            // [nb][nu][kpad]
    int32_t* bexp;           // [nb][32]
};

// offset1 bit for bit, without a comparison on the FP64 pipe (half >= 0)
template <int DIM>
__device__ __forceinline__ void load_offset(const Fma& F, const AsmArgs& a, const double* xp, int64_t q, double* o) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        o[d] = F.add(xp[d], -a.spos[q * DIM + d]);
        if (a.geom.per[d]) {
            const double L = a.geom.L[d], half = a.geom.half[d];
            const uint32_t oh = dhi(o[d]) & 0x7fffffffu, hh = dhi(half);
            if (oh > hh || (oh == hh && dlo(o[d]) > dlo(half)))
                o[d] = pipe_fma(o[d], F.one, (dhi(o[d]) >> 31) ? L : -L);
        }
    }
}

// bit of a status word: the coefficients of group g are in coef_range_or_zero
__device__ __forceinline__ int coef_bit(int g) { return 1 << (16 + g); }
__device__ __forceinline__ int group_status(int32_t word, int g) { return (word >> (4 * g)) & 15; }

// isfinite on the exponent bits (integer pipe, not the FP64 one)
__device__ __forceinline__ bool finite_bits(double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; }

// Tables every lane reads each row, staged in shared memory once per CTA.
struct ProgShared {
    unsigned char prog[kMaxSlots][2];
    unsigned char uslot[kMaxUnion];
};

__device__ __forceinline__ void stage_program(const AsmTables& T, ProgShared& P) {
    for (int e = threadIdx.x; e < T.nprog; e += blockDim.x) {
        P.prog[e][0] = T.prog[e][0];
        P.prog[e][1] = T.prog[e][1];
    }
    for (int e = threadIdx.x; e < T.nu; e += blockDim.x) P.uslot[e] = T.uslot[e];
    __syncthreads();
}

// Monomials of the union basis at u, into this lane's column of V
// ([slot][32]): m_j(u) = ((u0^e0) * u1^e1) * u2^e2 (Monomial.hpp:146-156)
// with the powers by ipow's squaring steps; the program performs exactly
// these multiplications, skipping factors equal to 1.0.
template <int DIM>
__device__ __forceinline__ void monomials(const double* u, double* V, const ProgShared& P, int nprog, int lane) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) V[d * 32 + lane] = u[d];
    V[DIM * 32 + lane] = 1.0;
    for (int o = 0; o < nprog; ++o)
        V[(DIM + 1 + o) * 32 + lane] = V[P.prog[o][0] * 32 + lane] * V[P.prog[o][1] * 32 + lane];
}

// The same on the integer pipes, for u in unit_range_or_zero (every power and
// product of the program is then in the range, or a zero).
template <int DIM>
__device__ __forceinline__ void monomials_int(const double* u, double* V, const ProgShared& P, int nprog, int lane) {
#pragma unroll
    for (int d = 0; d < DIM; ++d) V[d * 32 + lane] = u[d];
    V[DIM * 32 + lane] = 1.0;
    for (int o = 0; o < nprog; ++o)
        V[(DIM + 1 + o) * 32 + lane] = rn_mul_int(V[P.prog[o][0] * 32 + lane], V[P.prog[o][1] * 32 + lane]);
}

// ----------------------------------------------------------------- 0. eps --
// One thread per particle: eps = (sum_q sum_d |x_pq,d|) / k / HOverEpsilon
// summed sequentially over q (Vandermonde::computeEps), and the status of
// each basis group (too few neighbours for that basis, or a bad eps).
template <int DIM>
__global__ void __launch_bounds__(256) eps_kernel(AsmArgs a, Split S, int64_t b0, int64_t b1) {
    const AsmTables& T = *a.tab;
    const Fma F;
    const int ngroups = T.ngroups;
    for (int64_t it = b0 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; it < b1;
         it += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p = a.order ? (int64_t)a.order[it] : it;
        const int64_t beg = a.rowptr[p];
        const int k = (int)(a.rowptr[p + 1] - beg);
        double xp[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) xp[d] = a.pos[p * DIM + d];
        double s = 0.0;
        for (int q = 0; q < k; ++q) {
            double o[DIM];
            load_offset<DIM>(F, a, xp, a.cols[beg + q], o);
            double acc = fabs(o[0]);  // (0.0 + |o| is |o|)
#pragma unroll
            for (int d = 1; d < DIM; ++d) acc = F.add(acc, fabs(o[d]));
            s = F.add(s, acc);
        }
        s = s / (double)k;
        double eps = s / a.h_over_eps;
        if (a.eps_fixed) eps = a.eps_fixed[p];
        int32_t word = 0;
        const bool eps_ok = (eps > 0.0) && isfinite(eps);
        for (int g = 0; g < ngroups; ++g) {
            const int st = (k < T.gn[g]) ? ST_TOO_FEW : (eps_ok ? ST_OK : ST_BAD_EPS);
            word |= st << (4 * g);
        }
        a.eps[p] = eps;
        for (int g = 0; g < ngroups; ++g) a.eip_group[(int64_t)g * a.n + p] = 1.0 / ipow(eps, (unsigned)T.gord[g]);
        S.gst[it - b0] = word;
        double* sc = S.scale + (it - b0) * 4;
        const double d2 = 2.0 * eps * eps;
        sc[0] = eps;
        sc[1] = 1.0 / eps;
        sc[2] = d2;
        sc[3] = 1.0 / d2;
    }
}

// One neighbour row: u = x_pq / eps, the monomials at u in this lane's column
// of V, and E = exp(-|x_pq|^2 / (2 eps^2)) (returned); ints: E and the monomials
// are in the integer products' range.  The quotients, squares and monomials run
// on the integer pipes, which leaves the offsets, two sums and the exponential
// (23 FP64 instructions in 3D, 90 before) to the FP64 pipe, the bound of these
// kernels: 80^3 Gradient + Laplacian assembly 53.2 -> 46.3 ms.
template <int DIM>
__device__ __forceinline__ double gram_row(const Fma& F, const ExpShared& X, const AsmArgs& a, const double* sc,
                                           const double* xp, int64_t q, double (&u)[DIM], double* V,
                                           const ProgShared& P, int nprog, int lane, bool& ints) {
    double o[DIM];
    load_offset<DIM>(F, a, xp, q, o);
    const double eps = sc[0], reps = sc[1];
    bool unit = true;
#pragma unroll
    for (int d = 0; d < DIM; ++d) {
        u[d] = F.quot(o[d], eps, reps);
        unit = unit && unit_range_or_zero(u[d]);
    }
    double n2 = F.prod(o[0], o[0]);
#pragma unroll
    for (int d = 1; d < DIM; ++d) n2 = F.add(F.prod(o[d], o[d]), n2);
    const double E = cw_exp(F, X, F.quot(-n2, sc[2], sc[3]));
    if (unit)
        monomials_int<DIM>(u, V, P, nprog, lane);
    else
        monomials<DIM>(u, V, P, nprog, lane);
    ints = unit && int_range(E);
    return E;
}

// ---------------------------------------------------------------- 1. Gram --
// VJP: B has one more column, E_q (f_q - f_p), and the entries (i, nu) after
// the Gram entries are s = sum_q omega_q (f_q - f_p) v_q; E_q of every row is
// kept beside u for the chain rule.
template <int DIM, int NPP, bool VJP>
__global__ void __launch_bounds__(256) gram_kernel(AsmArgs a, Split S, int64_t b0, int64_t b1) {
    extern __shared__ double smem[];
    __shared__ ProgShared P;
    const AsmTables& T = *a.tab;
    __shared__ ExpShared X;
    stage_exp(X);
    stage_program(T, P);
    const Fma F;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    double* Bs = smem + (size_t)wib * (kCh * S.ldb + S.nslots * 32);
    double* V = Bs + kCh * S.ldb;
    const int nu = T.nu;
    const int npairs = T.npairs + (VJP ? nu : 0);
    const int ngroups = T.ngroups;
    const int nprog = T.nprog;

    // Gram entries owned by this lane
    int pi[NPP], pj[NPP];
#pragma unroll
    for (int t = 0; t < NPP; ++t) {
        int e = t * 32 + lane;
        pi[t] = (e < T.npairs) ? T.pi[e] : ((VJP && e < npairs) ? e - T.npairs : 0);
        pj[t] = (e < T.npairs) ? T.pj[e] : ((VJP && e < npairs) ? nu : 0);
    }

    const int wpc = blockDim.x >> 5;
    const int64_t nw = (int64_t)gridDim.x * wpc;
    for (int64_t it = b0 + (int64_t)blockIdx.x * wpc + wib; it < b1; it += nw) {
        const int64_t slot = it - b0;
        const int64_t p = a.order ? (int64_t)a.order[it] : it;
        const int64_t beg = a.rowptr[p];
        const int k = (int)(a.rowptr[p + 1] - beg);
        const int32_t word = S.gst[slot];
        bool any_ok = false;
        for (int g = 0; g < ngroups; ++g) any_ok |= group_status(word, g) == ST_OK;
        if (!any_ok) continue;  // warp-uniform
        double xp[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) xp[d] = a.pos[p * DIM + d];

        // A_ij = sum_q B_qi B_qj, B_qj = E_q m_j(x_pq / eps)
        double acc[NPP];
#pragma unroll
        for (int t = 0; t < NPP; ++t) acc[t] = 0.0;
        for (int c0 = 0; c0 < k; c0 += kCh) {
            int q = c0 + lane;
            const int cnt = min(kCh, k - c0);
            if (q < k) {
                double u[DIM];
                bool ints;
                const double E = gram_row<DIM>(F, X, a, S.scale + slot * 4, xp, a.cols[beg + q], u, V, P, nprog, lane, ints);
                double* Ur = S.usc + slot * S.ustride;
#pragma unroll
                for (int d = 0; d < DIM; ++d) Ur[d * S.maxk + q] = u[d];
                if (ints) {
                    for (int j = 0; j < nu; ++j) Bs[lane * S.ldb + j] = rn_mul_int(E, V[P.uslot[j] * 32 + lane]);
                } else {
                    for (int j = 0; j < nu; ++j) Bs[lane * S.ldb + j] = pipe_fma(E, V[P.uslot[j] * 32 + lane], F.nzero);
                }
                if constexpr (VJP) {
                    Ur[DIM * S.maxk + q] = E;
                    Bs[lane * S.ldb + nu] = F.prod(E, F.add(a.f[a.cols[beg + q]], -a.f[p]));
                }
            }
            __syncwarp();
            for (int r = 0; r < cnt; ++r) {
                const double* row = Bs + r * S.ldb;
#pragma unroll
                for (int t = 0; t < NPP; ++t)
                    if (t * 32 + lane < npairs) acc[t] = fma(row[pi[t]], row[pj[t]], acc[t]);
            }
            __syncwarp();
        }
        double* G = S.gram + slot * S.gstride;
#pragma unroll
        for (int t = 0; t < NPP; ++t)
            if (t * 32 + lane < npairs) G[t * 32 + lane] = acc[t];
    }
}

#include "dcpse_gram_tc.cuh"
#include "dcpse_vjp.cuh"

// Gram kernel for bases whose entries do not fit in the lanes' registers
// (more than 40 x 32 pairs, e.g. 7260 for the 120-function basis of
// |alpha| = 6 in 3D): the same rows of B, and every entry's sum continued
// from the batch scratch chunk after chunk, in the same sequential order, so
// the entries equal the register version's (and the reference's) bit for bit.
template <int DIM>
__global__ void __launch_bounds__(256) gram_wide_kernel(AsmArgs a, Split S, int64_t b0, int64_t b1) {
    extern __shared__ double smem[];
    __shared__ ProgShared P;
    const AsmTables& T = *a.tab;
    __shared__ ExpShared X;
    stage_exp(X);
    stage_program(T, P);
    const Fma F;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    double* Bs = smem + (size_t)wib * (kCh * S.ldb + S.nslots * 32);
    double* V = Bs + kCh * S.ldb;
    const int nu = T.nu;
    const int npairs = T.npairs;
    const int ngroups = T.ngroups;
    const int nprog = T.nprog;
    const int wpc = blockDim.x >> 5;
    const int64_t nw = (int64_t)gridDim.x * wpc;
    for (int64_t it = b0 + (int64_t)blockIdx.x * wpc + wib; it < b1; it += nw) {
        const int64_t slot = it - b0;
        const int64_t p = a.order ? (int64_t)a.order[it] : it;
        const int64_t beg = a.rowptr[p];
        const int k = (int)(a.rowptr[p + 1] - beg);
        const int32_t word = S.gst[slot];
        bool any_ok = false;
        for (int g = 0; g < ngroups; ++g) any_ok |= group_status(word, g) == ST_OK;
        if (!any_ok) continue;  // warp-uniform
        double xp[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) xp[d] = a.pos[p * DIM + d];
        double* G = S.gram + slot * S.gstride;
        for (int c0 = 0; c0 < k; c0 += kCh) {
            const int q = c0 + lane;
            const int cnt = min(kCh, k - c0);
            if (q < k) {
                double u[DIM];
                bool ints;
                const double E = gram_row<DIM>(F, X, a, S.scale + slot * 4, xp, a.cols[beg + q], u, V, P, nprog, lane, ints);
                double* Ur = S.usc + slot * S.ustride;
#pragma unroll
                for (int d = 0; d < DIM; ++d) Ur[d * S.maxk + q] = u[d];
                if (ints) {
                    for (int j = 0; j < nu; ++j) Bs[lane * S.ldb + j] = rn_mul_int(E, V[P.uslot[j] * 32 + lane]);
                } else {
                    for (int j = 0; j < nu; ++j) Bs[lane * S.ldb + j] = pipe_fma(E, V[P.uslot[j] * 32 + lane], F.nzero);
                }
            }
            __syncwarp();
            for (int e = lane; e < npairs; e += 32) {
                const int pi = T.pi[e], pj = T.pj[e];
                double acc = c0 == 0 ? 0.0 : G[e];
                for (int r = 0; r < cnt; ++r) acc = fma(Bs[r * S.ldb + pi], Bs[r * S.ldb + pj], acc);
                G[e] = acc;
            }
            __syncwarp();
        }
    }
}

// B for the tensor-core products: the SIMT Gram kernel's rows of B (u, E,
// the monomial program, in the same operations), stored to bmat[slot][j][q]
// in FP64, and for every column the exponent E_j with |B_qj| < 2^E_j (from
// the largest exponent field of the column), to bexp[slot][j].  One warp per
// particle, many per SM: the FP64 work of this part needs the latency hiding.
template <int DIM>
__global__ void __launch_bounds__(256) gram_b_kernel(AsmArgs a, Split S, int64_t b0, int64_t b1) {
    extern __shared__ double smem[];
    __shared__ ProgShared P;
    const AsmTables& T = *a.tab;
    __shared__ ExpShared X;
    stage_exp(X);
    stage_program(T, P);
    const Fma F;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    double* V = smem + (size_t)wib * (S.nslots * 32);
    const int nu = T.nu;
    const int ngroups = T.ngroups;
    const int nprog = T.nprog;
    const int wpc = blockDim.x >> 5;
    const int64_t nw = (int64_t)gridDim.x * wpc;
    for (int64_t it = b0 + (int64_t)blockIdx.x * wpc + wib; it < b1; it += nw) {
        const int64_t slot = it - b0;
        const int32_t word = S.gst[slot];
        bool any_ok = false;
        for (int g = 0; g < ngroups; ++g) any_ok |= group_status(word, g) == ST_OK;
        if (!any_ok) continue;  // warp-uniform
        const int64_t p = a.order ? (int64_t)a.order[it] : it;
        const int64_t beg = a.rowptr[p];
        const int k = (int)(a.rowptr[p + 1] - beg);
        double xp[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) xp[d] = a.pos[p * DIM + d];
        double* Bm = S.bmat + slot * (int64_t)nu * S.kpad;
        unsigned emax[kTcMaxNu];
#pragma unroll
        for (int j = 0; j < kTcMaxNu; ++j) emax[j] = 0;
        for (int c0 = 0; c0 < k; c0 += kCh) {
            const int q = c0 + lane;
            if (q < k) {
                double u[DIM];
                bool ints;
                const double E = gram_row<DIM>(F, X, a, S.scale + slot * 4, xp, a.cols[beg + q], u, V, P, nprog, lane, ints);
                double* Ur = S.usc + slot * S.ustride;
#pragma unroll
                for (int d = 0; d < DIM; ++d) Ur[d * S.maxk + q] = u[d];
#pragma unroll
                for (int j = 0; j < kTcMaxNu; ++j)
                    if (j < nu) {
                        const double v = V[P.uslot[j] * 32 + lane];
                        const double b = ints ? rn_mul_int(E, v) : E * v;
                        Bm[(int64_t)j * S.kpad + q] = b;
                        emax[j] = max(emax[j], ((unsigned)__double2hiint(b) >> 20) & 0x7ffu);
                    }
            }
            __syncwarp();
        }
        // |x| < 2^(e - 1022) for a normal x with exponent field e
        int mine = 0;
#pragma unroll
        for (int j = 0; j < kTcMaxNu; ++j) {
            const unsigned m = __reduce_max_sync(0xffffffffu, emax[j]);
            if (lane == j) mine = max((int)m, 1) - 1022;
        }
        S.bexp[slot * 32 + lane] = mine;
    }
}


// ------------------------------------------------------------------ 2. QR --
// All lanes of a warp run the same loop trip counts (the basis sizes are the
// plan's); particles differ only in their data, so every shuffle and warp
// barrier is reached by the whole warp.  A group whose factorisation breaks
// down (or that was not assembled) keeps running on its own work space and
// only its stores are suppressed.
template <int LPP, bool WS>
__global__ void __launch_bounds__(kQrWarps * 32) qr_kernel(AsmArgs a, Split S, int64_t b0, int64_t nb) {
    constexpr int PPW = 32 / LPP;
    extern __shared__ double smem[];
    const AsmTables& T = *a.tab;
    const bool fast = (a.flags & DCPSE_ASSEMBLE_FAST_FLAG) != 0;
    const int lane = threadIdx.x & 31;
    const int l = lane & (LPP - 1);
    const int sub = lane / LPP;
    const int wib = threadIdx.x >> 5;
    const int wpc = blockDim.x >> 5;
    const int pidx = wib * PPW + sub;  // particle slot of this lane group in the CTA
    // work space: shared memory, or a global slot per lane group when the
    // basis is too large for it (WS); a template argument, so that the shared
    // one is addressed as such
    const int64_t gslot = ((int64_t)blockIdx.x * wpc + wib) * PPW + sub;
    double* R = WS ? S.qws + gslot * S.pstride : smem + (size_t)pidx * S.pstride;
    int* perm = WS ? S.qperm + gslot * S.nmax
                   : reinterpret_cast<int*>(smem + (size_t)wpc * PPW * S.pstride) + pidx * S.nmax;
    // the Gram entry of every (i <= j) of every group, as entry << 16 | i << 8 | j
    uint32_t* tab = reinterpret_cast<uint32_t*>(smem + (size_t)wpc * PPW * S.pstride) + wpc * PPW * S.nmax;
    if (!WS && S.qtab) {
        int base = 0;
        for (int g = 0; g < T.ngroups; ++g) {
            const int n = T.gn[g];
            for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
                const int i = e / n, j = e - i * n;
                if (i > j) continue;
                const int ui = T.gidx[g][i], uj = T.gidx[g][j];
                tab[base + j * (j + 1) / 2 + i] =
                    (uint32_t)T.upair[min(ui, uj)][max(ui, uj)] << 16 | (uint32_t)i << 8 | (uint32_t)j;
            }
            base += n * (n + 1) / 2;
        }
        __syncthreads();
    }
    const int ngroups = T.ngroups;
    const Fma F;

    for (int64_t w0 = ((int64_t)blockIdx.x * wpc + wib) * PPW; w0 < nb; w0 += (int64_t)gridDim.x * wpc * PPW) {
        const int64_t slot = w0 + sub;
        const bool valid = slot < nb;
        int32_t word = valid ? S.gst[slot] : 0x11111111;
        const double* __restrict__ G = S.gram + (valid ? slot : 0) * S.gstride;
        int tab0 = 0;
        for (int g = 0; g < ngroups; ++g) {
            const int n = T.gn[g];
            const int nrhs = S.nrhs[g];
            const int ncol = n + nrhs;
            const int ldr = ncol;         // [A | b...], n rows
            double* Z = R + n * ncol;     // solutions, n x nrhs
            const bool active = valid && group_status(word, g) == ST_OK;
            // R = [A | b...]
            if (WS || !S.qtab) {
                for (int e = l; e < n * n; e += LPP) {
                    const int i = e / n, j = e - i * n;
                    const int ui = T.gidx[g][i], uj = T.gidx[g][j];
                    R[i * ldr + j] = active ? G[T.upair[min(ui, uj)][max(ui, uj)]] : 0.0;
                }
            } else {
                const int ne = n * (n + 1) / 2;
#pragma unroll 4
                for (int e = l; e < ne; e += LPP) {
                    const uint32_t t = tab[tab0 + e];
                    const int i = (int)(t >> 8) & 255, j = (int)t & 255;
                    const double v = active ? G[t >> 16] : 0.0;
                    R[i * ldr + j] = v;
                    R[j * ldr + i] = v;
                }
                tab0 += ne;
            }
            for (int e = l; e < n * nrhs; e += LPP) {
                const int i = e / nrhs, r = e - i * nrhs;
                double v = 0.0;
                if (active) {
                    if (S.vjp) {
                        // b~ = sum_o gbar_o b_o, then s
                        if (r == 0) {
                            for (int o = 0; o < T.nout_rhs[g]; ++o)
                                v += a.gbar[(int64_t)T.out_of_rhs[g][o] * a.n + b0 + slot] * T.b_out[g][o][i];
                        } else {
                            v = G[S.npairs + T.gidx[g][i]];
                        }
                    } else {
                        v = fast ? T.b_out[g][r][i] : T.b_term[g][r][i];
                    }
                }
                R[i * ldr + n + r] = v;
            }
            for (int i = l; i < n; i += LPP) perm[i] = i;
            __syncwarp();
            bool dead = !active;
            // The next pivot of this lane's columns: first largest squared norm
            // of the trailing block.  A norm is >= 0 or NaN, so the bits order
            // the values and a NaN counts below everything (key -1).
            long long best = -1;
            int bidx = 0x7fffffff;
            auto offer = [&](double sn, int j) {
                long long key = (long long)(((unsigned long long)dhi(sn) << 32) | dlo(sn));
                if (key > 0x7ff0000000000000ll || key < 0) key = -1;
                if (key > best) {
                    best = key;
                    bidx = j;
                }
            };
            for (int j = l; j < n; j += LPP) {
                double sn = 0.0;
                for (int i = 0; i < n; ++i) sn = fma(R[i * ldr + j], R[i * ldr + j], sn);
                offer(sn, j);
            }
            for (int kk = 0; kk < n; ++kk) {
#pragma unroll
                for (int o = LPP / 2; o > 0; o >>= 1) {
                    const long long ob = __shfl_xor_sync(0xffffffffu, best, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, bidx, o);
                    if (ob > best || (ob == best && oi < bidx)) {
                        best = ob;
                        bidx = oi;
                    }
                }
                const int piv = (bidx == 0x7fffffff) ? kk : bidx;
                // sigma: the pivot column's squared norm (NaN when all were)
                const double sigma = __hiloint2double((int)(best >> 32), (int)best);
                dead |= best <= 0;
                if (piv != kk) {
                    for (int i = l; i < n; i += LPP) {
                        const double t0 = R[i * ldr + kk];
                        R[i * ldr + kk] = R[i * ldr + piv];
                        R[i * ldr + piv] = t0;
                    }
                    if (l == 0) {
                        const int t0 = perm[kk];
                        perm[kk] = perm[piv];
                        perm[piv] = t0;
                    }
                }
                __syncwarp();
                const double alpha = R[kk * ldr + kk];
                const double nr = sqrt(sigma);
                const double beta = (!(dhi(alpha) >> 31) || is_zero(alpha)) ? -nr : nr;  // alpha >= 0
                const double den = F.add(alpha, -beta);
                // 1 / den on even lanes beside 1 / beta on odd ones
                double rden, rbeta;
                if constexpr (LPP == 1) {
                    rden = __drcp_rn(den);
                    rbeta = __drcp_rn(beta);
                } else {
                    const double rc = __drcp_rn((l & 1) ? beta : den);
                    rden = __shfl_sync(0xffffffffu, rc, lane & ~1);
                    rbeta = __shfl_sync(0xffffffffu, rc, lane | 1);
                }
                const double tau = F.quot(-den, beta, rbeta);  // (beta - alpha) / beta
                __syncwarp();
                for (int i = kk + 1 + l; i < n; i += LPP) R[i * ldr + kk] = F.quot(R[i * ldr + kk], den, rden);
                __syncwarp();
                if (l == 0) R[kk * ldr + kk] = beta;
                best = -1;
                bidx = 0x7fffffff;
                const double* v = R + (kk + 1) * ldr + kk;
                const int m = n - kk - 1;
                // the reflection of columns kk + 1 .., two of this lane's at a
                // time, and the squared norms the next pivot is chosen by
                int j = kk + 1 + l;
                for (; j + LPP < ncol; j += 2 * LPP) {
                    double* c0 = R + kk * ldr + j;
                    double* c1 = c0 + LPP;
                    double s0 = c0[0], s1 = c1[0];
                    c0 += ldr;
                    c1 += ldr;
#pragma unroll 4
                    for (int i = 0; i < m; ++i) {
                        const double vi = v[i * ldr];
                        s0 = fma(vi, c0[i * ldr], s0);
                        s1 = fma(vi, c1[i * ldr], s1);
                    }
                    s0 = F.mul(s0, tau);
                    s1 = F.mul(s1, tau);
                    c0[-ldr] = F.add(c0[-ldr], -s0);
                    c1[-ldr] = F.add(c1[-ldr], -s1);
                    double n0 = 0.0, n1 = 0.0;
#pragma unroll 4
                    for (int i = 0; i < m; ++i) {
                        const double vi = v[i * ldr];
                        const double x0 = fma(-s0, vi, c0[i * ldr]), x1 = fma(-s1, vi, c1[i * ldr]);
                        c0[i * ldr] = x0;
                        c1[i * ldr] = x1;
                        n0 = fma(x0, x0, n0);
                        n1 = fma(x1, x1, n1);
                    }
                    if (j < n) offer(n0, j);
                    if (j + LPP < n) offer(n1, j + LPP);
                }
                if (j < ncol) {
                    double* c0 = R + kk * ldr + j;
                    double s0 = c0[0];
                    c0 += ldr;
#pragma unroll 4
                    for (int i = 0; i < m; ++i) s0 = fma(v[i * ldr], c0[i * ldr], s0);
                    s0 = F.mul(s0, tau);
                    c0[-ldr] = F.add(c0[-ldr], -s0);
                    double n0 = 0.0;
#pragma unroll 4
                    for (int i = 0; i < m; ++i) {
                        const double x0 = fma(-s0, v[i * ldr], c0[i * ldr]);
                        c0[i * ldr] = x0;
                        n0 = fma(x0, x0, n0);
                    }
                    if (j < n) offer(n0, j);
                }
                __syncwarp();
            }
            // back substitution, right-hand sides split over the lanes; the
            // diagonal's reciprocals, a lane each, over row n - 1 of the
            // reflections (not needed any more)
            for (int i = l; i < n - 1; i += LPP) R[(n - 1) * ldr + i] = __drcp_rn(R[i * ldr + i]);
            const double rlast = __drcp_rn(R[(n - 1) * ldr + n - 1]);
            __syncwarp();
            for (int r = l; r < nrhs; r += LPP) {
                for (int i = n - 1; i >= 0; --i) {
                    double sv = R[i * ldr + n + r];
                    for (int j = i + 1; j < n; ++j) sv = fma(-R[i * ldr + j], Z[j * nrhs + r], sv);
                    Z[i * nrhs + r] = F.quot(sv, R[i * ldr + i], i == n - 1 ? rlast : R[(n - 1) * ldr + i]);
                }
            }
            __syncwarp();
            bool in_range = true;
            if (!dead) {
                double* C = S.coef + slot * S.cstride + S.c_off[g];
                for (int e = l; e < n * nrhs; e += LPP) {
                    const int i = e / nrhs, r = e - i * nrhs;
                    const double z = Z[i * nrhs + r];
                    C[perm[i] * nrhs + r] = z;
                    in_range = in_range && coef_range_or_zero(z);
                }
            } else if (active) {
                word = (word & ~(15 << (4 * g))) | (ST_SINGULAR << (4 * g));
            }
            const unsigned lanes = LPP == 32 ? 0xffffffffu : ((1u << LPP) - 1u) << (sub * LPP);
            if ((__ballot_sync(0xffffffffu, in_range) & lanes) == lanes) word |= coef_bit(g);
            __syncwarp();
        }
        if (valid && l == 0) S.gst[slot] = word;
    }
}

// ------------------------------------------------------------- 3. weights --
// NR right-hand sides of one group and one neighbour row in the reference's
// order, res_r = sum_i (A_ir V_i) ef (coefficients A of row stride ld).  INT: the
// products on the integer pipes, but every other product with ef, which keeps
// both pipes about equally busy (uneven 2D cloud, five terms: 1.47 ms with all
// of them on the integer pipes, at 66 % of those and 56 % of the FP64 pipe).
template <int NR, bool INT>
__device__ __forceinline__ void reference_sums(const Fma& F, const double* __restrict__ A, int ld, int n,
                                               const unsigned char* gslot, const double* V, int lane, double ef,
                                               double (&res)[NR]) {
#pragma unroll 2
    for (int i = 0; i < n; ++i) {
        const double v = V[gslot[i] * 32 + lane];
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const double t = INT ? rn_mul_int(A[i * ld + r], v) : F.mul(A[i * ld + r], v);
            res[r] = F.add(INT && (i & 1) == 0 ? rn_mul_int(t, ef) : F.mul(t, ef), res[r]);
        }
    }
}

// res_r = sum_i A_ir V_i by fused multiply-adds (fast assembly)
template <int NR>
__device__ __forceinline__ void fast_sums(const double* __restrict__ A, int ld, int n, const unsigned char* gslot,
                                          const double* V, int lane, double (&res)[NR]) {
    for (int i = 0; i < n; ++i) {
        const double v = V[gslot[i] * 32 + lane];
#pragma unroll
        for (int r = 0; r < NR; ++r) res[r] = fma(A[i * ld + r], v, res[r]);
    }
}

// The entries of up to 32 consecutive particles, one per lane: a warp takes
// `per_warp` particles, concatenates their rows and walks them 32 entries at a
// time (a binary search over the rows' ends gives a lane its particle), so that
// only the last step of all has idle lanes.  The particles' coefficients are
// read through L1; per-output sums live in this lane's column of shared memory.
//
// FP64-pipe bound: a warp per particle with its rows in chunks of 32 ran 14 %
// (3D) to 40 % (uneven 2D clouds) of its lanes idle, and in the reference's
// order every coefficient took two products and a sum on the pipe.  Now the
// monomials, the reference order's products and the scalings are on the integer
// pipes, the sums are three-register dfmas and the FP32 narrowing is on integers:
// 2e5 uneven particles, five terms in the reference's order 3.18 -> 1.34 ms; 80^3
// Gradient + Laplacian, fast assembly, a batch of 1.2e5 particles 2.44 -> 1.59 ms.
template <int DIM>
__global__ void __launch_bounds__(256) weights_kernel(AsmArgs a, Split S, int64_t b0, int64_t b1, int per_warp) {
    extern __shared__ double smem[];
    __shared__ ProgShared P;
    __shared__ ExpShared X;
    __shared__ unsigned char gslot[kMaxGroups][kMaxBasis];  // slot of basis function i of group g
    const AsmTables& T = *a.tab;
    const int ngroups = T.ngroups;
    for (int g = 0; g < ngroups; ++g)
        for (int i = threadIdx.x; i < T.gn[g]; i += blockDim.x) gslot[g][i] = T.uslot[T.gidx[g][i]];
    stage_exp(X);
    stage_program(T, P);  // (ends with a barrier)
    const Fma F;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    double* V = smem + (size_t)wib * (S.nslots + S.nout + S.nrmax) * 32;
    double* Wacc = V + S.nslots * 32;
    double* R = Wacc + S.nout * 32;
    const int nprog = T.nprog;
    const bool fast = (a.flags & DCPSE_ASSEMBLE_FAST_FLAG) != 0;
    const bool st_terms = a.k_term != nullptr;
    const int noutputs = T.noutputs;

    const int wpc = blockDim.x >> 5;
    const int64_t nw = (int64_t)gridDim.x * wpc;
    for (int64_t t0 = b0 + ((int64_t)blockIdx.x * wpc + wib) * per_warp; t0 < b1; t0 += nw * per_warp) {
        // lane l holds particle t0 + l of the warp's group
        const int np = (int)min((int64_t)per_warp, b1 - t0);
        int64_t lp = 0, lbeg = 0;
        int32_t lword = 0;
        int lk = 0;
        if (lane < np) {
            lp = a.order ? (int64_t)a.order[t0 + lane] : t0 + lane;
            lbeg = a.rowptr[lp];
            lk = (int)(a.rowptr[lp + 1] - lbeg);
            lword = S.gst[t0 + lane - b0];
        }
        int lend = lk;  // inclusive scan of the row lengths
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(full, lend, o);
            if (lane >= o) lend += v;
        }
        const int total = __shfl_sync(full, lend, 31);
        unsigned bad = 0;  // particles of the group with a non-finite kernel
        for (int e0 = 0; e0 < total; e0 += 32) {
            const int e = e0 + lane;
            int s = 0, hi = np - 1;  // first particle whose rows end past e
#pragma unroll
            for (int it = 0; it < 5; ++it) {
                const int mid = (s + hi) >> 1;
                const int v = __shfl_sync(full, lend, mid);
                if (s < hi) {
                    if (v > e)
                        hi = mid;
                    else
                        s = mid + 1;
                }
            }
            const int q = e - (__shfl_sync(full, lend, s) - __shfl_sync(full, lk, s));
            const int64_t at = __shfl_sync(full, lbeg, s) + q;
            const int64_t p = __shfl_sync(full, lp, s);
            const int32_t word = __shfl_sync(full, lword, s);
            bool nonfinite = false;
            if (e < total) {
                const int64_t slot = t0 - b0 + s;
                // u = x_pq / eps as the Gram kernel computed it (rows of particles
                // with no assembled group were skipped there and are not used here)
                double u[DIM];
                const double* Ur = S.usc + slot * S.ustride + q;
                bool unit = true;
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    u[d] = Ur[d * S.maxk];
                    unit = unit && unit_range_or_zero(u[d]);
                }
                double u2;
                if (unit) {
                    monomials_int<DIM>(u, V, P, nprog, lane);
                    u2 = rn_mul_int(u[0], u[0]);
#pragma unroll
                    for (int d = 1; d < DIM; ++d) u2 = F.add(rn_mul_int(u[d], u[d]), u2);
                } else {
                    monomials<DIM>(u, V, P, nprog, lane);
                    u2 = norm2<DIM>(u);
                }
                const double ef = cw_exp(F, X, -u2);
                const bool ints = unit && int_range(ef);
                for (int t = 0; t < noutputs; ++t) Wacc[t * 32 + lane] = 0.0;
                for (int g = 0; g < ngroups; ++g) {
                    const int n = T.gn[g];
                    const int nrhs = S.nrhs[g];
                    const bool ok = group_status(word, g) == ST_OK;
                    const double* __restrict__ Ag = S.coef + slot * S.cstride + S.c_off[g];
                    const double eip = a.eip_group[(int64_t)g * a.n + p];
                    // the sums of NR right-hand sides from r0 on, to this lane's
                    // column of R
                    auto block = [&](int r0, auto count) {
                        constexpr int NR = decltype(count)::value;
                        double res[NR];
#pragma unroll
                        for (int r = 0; r < NR; ++r) res[r] = 0.0;
                        if (fast)
                            fast_sums<NR>(Ag + r0, nrhs, n, gslot[g], V, lane, res);
                        else
                            reference_sums<NR, true>(F, Ag + r0, nrhs, n, gslot[g], V, lane, ef, res);
#pragma unroll
                        for (int r = 0; r < NR; ++r) R[(r0 + r) * 32 + lane] = res[r];
                    };
                    if (!ok) {
                        for (int r = 0; r < nrhs; ++r) R[r * 32 + lane] = 0.0;
                    } else if (!fast && !(ints && (word & coef_bit(g)))) {
                        for (int r = 0; r < nrhs; ++r) {
                            double res[1] = {0.0};
                            reference_sums<1, false>(F, Ag + r, nrhs, n, gslot[g], V, lane, ef, res);
                            R[r * 32 + lane] = res[0];
                        }
                    } else {
                        int r0 = 0;
                        for (; r0 + 3 <= nrhs; r0 += 3) block(r0, std::integral_constant<int, 3>{});
                        if (nrhs - r0 == 2)
                            block(r0, std::integral_constant<int, 2>{});
                        else if (nrhs - r0 == 1)
                            block(r0, std::integral_constant<int, 1>{});
                    }
#pragma unroll 1
                    for (int r = 0; r < nrhs; ++r) {
                        const double res = R[r * 32 + lane];
                        const double Kq = fast && ok ? F.prod(res, ef) : res;
                        int o2;
                        if (fast) {
                            o2 = T.out_of_rhs[g][r];
                        } else {
                            const int term = T.term_of_rhs[g][r];
                            if (st_terms) a.k_term[(int64_t)term * a.nnz + at] = Kq;
                            o2 = T.term_output[term];
                        }
                        nonfinite |= !finite_bits(Kq);
                        const double w = Wacc[o2 * 32 + lane], v = F.prod(Kq, eip);
                        // (0.0 + v is v but for v = -0.0)
                        double sum;
                        if (is_plus_zero(w))
                            sum = is_zero(v) ? 0.0 : v;
                        else
                            sum = pipe_fma(v, F.one, w);
                        Wacc[o2 * 32 + lane] = sum;
                    }
                }
#pragma unroll 1
                for (int t = 0; t < noutputs; ++t) {
                    const double w = Wacc[t * 32 + lane];
                    const int64_t i = (int64_t)t * a.nnz + at;
                    if (a.w64) a.w64[i] = w;
                    if (a.w32) {
                        const float w32 = narrow(w);
                        a.w32[i] = w32;
                        if (a.r16 || a.r32) {
                            const float r = narrow(F.add(w, -widen(w32)));
                            if (a.r16) reinterpret_cast<__nv_bfloat16*>(a.r16)[i] = __float2bfloat16_rn(r);
                            if (a.r32) a.r32[i] = r;
                        }
                    }
                }
            }
            bad |= __reduce_or_sync(full, nonfinite ? 1u << s : 0u);
        }
        for (unsigned m = bad; m; m &= m - 1) {
            // zero every stored row of this particle (the oracle zeroes the
            // affected term's kernels; fused outputs are zeroed entirely)
            const int s = __ffs(m) - 1;
            const int64_t beg = __shfl_sync(full, lbeg, s);
            const int k = __shfl_sync(full, lk, s);
            for (int q = lane; q < k; q += 32) {
                if (st_terms)
                    for (int t = 0; t < T.nterms; ++t) a.k_term[(int64_t)t * a.nnz + beg + q] = 0.0;
                for (int t = 0; t < noutputs; ++t) {
                    if (a.w64) a.w64[(int64_t)t * a.nnz + beg + q] = 0.0;
                    if (a.w32) a.w32[(int64_t)t * a.nnz + beg + q] = 0.0f;
                    if (a.r16)
                        reinterpret_cast<__nv_bfloat16*>(a.r16)[(int64_t)t * a.nnz + beg + q] = __float2bfloat16_rn(0.0f);
                    if (a.r32) a.r32[(int64_t)t * a.nnz + beg + q] = 0.0f;
                }
            }
        }
        if (lane < np) {
            int st = ST_OK;
            for (int g = 0; g < ngroups; ++g)
                if (st == ST_OK && group_status(lword, g) != ST_OK) st = group_status(lword, g);
            if (st == ST_OK && ((bad >> lane) & 1u)) st = ST_NONFINITE;
            a.status[lp] = st;
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------- launches --
int warps_of(const AsmArgs& a) { return (a.warps == 2 || a.warps == 8) ? a.warps : kWarps; }

int smem_attr(cudaDeviceAttr attr, int fallback) {
    int dev = 0, v = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&v, attr, dev) != cudaSuccess) return fallback;
    return v;
}

template <typename K>
cudaError_t persistent(K kern, int threads, size_t bytes, int64_t work_per_cta, int64_t units, int& grid_out) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, bytes);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    int64_t need = (units + work_per_cta - 1) / work_per_cta;
    int64_t grid = (int64_t)num_sms() * per_sm;
    if (grid > need) grid = need;
    if (grid < 1) grid = 1;
    grid_out = (int)grid;
    return cudaSuccess;
}

template <int DIM>
cudaError_t launch_eps(const AsmArgs& a, const Split& S, int64_t b0, int64_t b1, cudaStream_t s) {
    auto kern = eps_kernel<DIM>;
    int grid = 0;
    cudaError_t e = persistent(kern, 256, 0, 256, b1 - b0, grid);
    if (e != cudaSuccess) return e;
    kern<<<grid, 256, 0, s>>>(a, S, b0, b1);
    return cudaGetLastError();
}

template <int DIM, int NPP, bool VJP>
cudaError_t launch_gram(const AsmArgs& a, const Split& S, int64_t b0, int64_t b1, cudaStream_t s) {
    int warps = warps_of(a);
    const size_t per_warp = (size_t)(kCh * S.ldb + S.nslots * 32) * sizeof(double);
    if constexpr (NPP == 0) {
        // large bases: as many warps as their B chunks leave room for
        const int fit = smem_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, 227 * 1024) / (int)per_warp;
        warps = std::max(1, std::min(warps, fit));
        const size_t bytes = per_warp * warps;
        auto kern = gram_wide_kernel<DIM>;
        int grid = 0;
        cudaError_t e = persistent(kern, warps * 32, bytes, warps, b1 - b0, grid);
        if (e != cudaSuccess) return e;
        kern<<<grid, warps * 32, bytes, s>>>(a, S, b0, b1);
        return cudaGetLastError();
    }
    const size_t bytes = per_warp * warps;
    auto kern = gram_kernel<DIM, NPP == 0 ? 1 : NPP, VJP>;
    int grid = 0;
    cudaError_t e = persistent(kern, warps * 32, bytes, warps, b1 - b0, grid);
    if (e != cudaSuccess) return e;
    kern<<<grid, warps * 32, bytes, s>>>(a, S, b0, b1);
    return cudaGetLastError();
}

// Work space of one particle: [A|b] then the solutions of the largest group,
// padded to LPP mod 16 doubles so that the lane groups of a half warp (16
// lanes, 64-bit accesses) fall on distinct shared-memory banks.
int qr_pstride(const Split& S, int lpp) { return S.qwords + ((lpp - S.qwords) & 15); }

size_t qr_bytes(const Split& S, int lpp, bool table = true) {
    return (size_t)kQrWarps * (32 / lpp) * (qr_pstride(S, lpp) * sizeof(double) + S.nmax * sizeof(int)) +
           (table ? (size_t)S.qtab * sizeof(uint32_t) : 0);
}

// CTAs per SM of the QR with its work space in global memory (one warp and
// one particle each)
constexpr int kQrGlobalPerSm = 4;

template <int LPP>
cudaError_t launch_qr(const AsmArgs& a, Split S, int64_t b0, int64_t nb, cudaStream_t s) {
    constexpr int PPW = 32 / LPP;
    S.pstride = qr_pstride(S, LPP);
    // without the table of Gram entries where it is what does not fit
    if (qr_bytes(S, LPP) > (size_t)smem_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, 227 * 1024)) S.qtab = 0;
    if constexpr (LPP == 32)
        if (S.qws) {
            const int64_t grid = std::min<int64_t>((int64_t)num_sms() * kQrGlobalPerSm, nb);
            qr_kernel<LPP, true><<<(unsigned)std::max<int64_t>(grid, 1), 32, 0, s>>>(a, S, b0, nb);
            return cudaGetLastError();
        }
    const size_t bytes = qr_bytes(S, LPP);
    auto kern = qr_kernel<LPP, false>;
    int grid = 0;
    cudaError_t e = persistent(kern, kQrWarps * 32, bytes, (int64_t)kQrWarps * PPW, nb, grid);
    if (e != cudaSuccess) return e;
    kern<<<grid, kQrWarps * 32, bytes, s>>>(a, S, b0, nb);
    return cudaGetLastError();
}

template <int DIM>
cudaError_t launch_weights(const AsmArgs& a, const Split& S, int64_t b0, int64_t b1, cudaStream_t s) {
    int warps = warps_of(a);
    const size_t per_warp = (size_t)((S.nslots + S.nout + S.nrmax) * 32) * sizeof(double);
    // large bases: as many warps as their monomials leave room for
    warps = std::max(1, std::min(warps, smem_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, 227 * 1024) / (int)per_warp));
    const size_t bytes = per_warp * warps;
    auto kern = weights_kernel<DIM>;
    // particles a warp takes at a time: 16 leave a few idle lanes in a hundred,
    // fewer when that would leave warps of the GPU without any
    const int64_t nb = b1 - b0;
    const int64_t chip = (int64_t)num_sms() * 32;
    const int take = (int)std::max<int64_t>(1, std::min<int64_t>(16, nb / chip));
    int grid = 0;
    cudaError_t e = persistent(kern, warps * 32, bytes, (int64_t)warps * take, nb, grid);
    if (e != cudaSuccess) return e;
    kern<<<grid, warps * 32, bytes, s>>>(a, S, b0, b1, take);
    return cudaGetLastError();
}

// Lanes per particle of the QR: the fewest from two on that still leave >= 6
// warps per SM resident within the shared-memory budget, then up to eight while
// the particles give the GPU less than a warp per scheduler.  Measured (whole
// fast assembly, ms, for 1 / 2 / 4 / 8 / 16 lanes): 60^3 Gradient + Laplacian 25.5
// / 19.9 / 17.4 / 18.9 / 22.7; 2D Laplacian, 65,536 particles 1.01 / 0.95 / 1.04 /
// 1.14 / 1.39, 4,096 particles 0.274 / 0.249 / 0.237 / 0.232 / 0.243; uneven 2D
// cloud, 2e5 particles, five operators 4.07 / 3.58 / 3.78 / 4.43 / 5.57.
int qr_lanes_auto(const Split& S, int64_t nb) {
    const int per_sm = smem_attr(cudaDevAttrMaxSharedMemoryPerMultiprocessor, 228 * 1024);
    const int per_block = smem_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, 227 * 1024);
    for (int lpp : {2, 4, 8, 16}) {
        const size_t b = qr_bytes(S, lpp);
        if (b > (size_t)per_block) continue;
        const int blocks = (int)(per_sm / (b + 1024));
        if (blocks * kQrWarps < 6) continue;
        while (lpp < 8 && nb * lpp / 32 < (int64_t)num_sms() * 4) lpp *= 2;
        return lpp;
    }
    return 32;
}

cudaError_t launch_qr_any(const AsmArgs& a, const Split& S, int lpp, int64_t b0, int64_t nb, cudaStream_t s) {
    switch (lpp) {
        case 1: return launch_qr<1>(a, S, b0, nb, s);
        case 2: return launch_qr<2>(a, S, b0, nb, s);
        case 4: return launch_qr<4>(a, S, b0, nb, s);
        case 8: return launch_qr<8>(a, S, b0, nb, s);
        case 16: return launch_qr<16>(a, S, b0, nb, s);
        default: return launch_qr<32>(a, S, b0, nb, s);
    }
}

template <int DIM>
cudaError_t launch_gram_tc(const AsmArgs& a, const Split& S, int64_t b0, int64_t b1, cudaStream_t s) {
    {
        const int warps = warps_of(a);
        const size_t bytes = (size_t)(S.nslots * 32) * sizeof(double) * warps;
        auto kb = gram_b_kernel<DIM>;
        int grid = 0;
        cudaError_t e = persistent(kb, warps * 32, bytes, warps, b1 - b0, grid);
        if (e != cudaSuccess) return e;
        kb<<<grid, warps * 32, bytes, s>>>(a, S, b0, b1);
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    const TcLayout L = tc_layout(S.maxk, S.npairs);
    auto kern = gram_tc_kernel;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.bytes);
    if (e != cudaSuccess) return e;
    // one CTA per SM holds all its tensor memory, two particles per CTA at a time
    const int64_t grid = std::min<int64_t>((b1 - b0 + 1) / 2, (int64_t)num_sms());
    kern<<<(unsigned)grid, kTcThreads, L.bytes, s>>>(a, S, b0, b1, L);
    return cudaGetLastError();
}

template <int DIM, int NPP>
cudaError_t run(const AsmArgs& a, const AsmTables& h, const Split& S, int lpp, cudaStream_t s) {
    for (int64_t b0 = 0; b0 < a.n; b0 += a.scratch_particles) {
        const int64_t b1 = std::min(a.n, b0 + a.scratch_particles);
        cudaError_t e = launch_eps<DIM>(a, S, b0, b1, s);
        if (e == cudaSuccess)
            e = S.tc ? launch_gram_tc<DIM>(a, S, b0, b1, s) : launch_gram<DIM, NPP, false>(a, S, b0, b1, s);
        if (e == cudaSuccess) e = launch_qr_any(a, S, lpp, b0, b1 - b0, s);
        if (e == cudaSuccess) e = launch_weights<DIM>(a, S, b0, b1, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

template <int DIM>
cudaError_t dispatch(const AsmArgs& a, const AsmTables& h, const Split& S, int lpp, cudaStream_t s) {
    // Gram entries per lane: the smallest instantiated count that holds them
    // all (a slot no lane uses would still occupy the FP64 pipe every row)
    const int npp = (h.npairs + 31) / 32;
    if (npp <= 2) return run<DIM, 2>(a, h, S, lpp, s);
    if (npp <= 4) return run<DIM, 4>(a, h, S, lpp, s);
    if (npp <= 7) return run<DIM, 7>(a, h, S, lpp, s);
    if (npp <= 8) return run<DIM, 8>(a, h, S, lpp, s);
    if (npp <= 16) return run<DIM, 16>(a, h, S, lpp, s);
    if (npp <= 40) return run<DIM, 40>(a, h, S, lpp, s);
    return run<DIM, 0>(a, h, S, lpp, s);  // the wide Gram kernel
}

template <int DIM>
cudaError_t launch_chain(const AsmArgs& a, const Split& S, int ngroups, int64_t b0, int64_t b1, cudaStream_t s) {
    const int warps = warps_of(a);
    const size_t bytes = (size_t)(S.cstride + (S.nslots + 2 * ngroups) * 32) * sizeof(double) * warps;
    auto kern = vjp_chain_kernel<DIM>;
    int grid = 0;
    cudaError_t e = persistent(kern, warps * 32, bytes, warps, b1 - b0, grid);
    if (e != cudaSuccess) return e;
    kern<<<grid, warps * 32, bytes, s>>>(a, S, b0, b1);
    return cudaGetLastError();
}

template <int DIM>
cudaError_t vjp_run(const AsmArgs& a, const AsmTables& h, const Split& S, int lpp, cudaStream_t s) {
    const int npp = (h.npairs + h.nu + 31) / 32;
    for (int64_t b0 = 0; b0 < a.n; b0 += a.scratch_particles) {
        const int64_t b1 = std::min(a.n, b0 + a.scratch_particles);
        cudaError_t e = launch_eps<DIM>(a, S, b0, b1, s);
        if (e == cudaSuccess)
            e = npp <= 2   ? launch_gram<DIM, 2, true>(a, S, b0, b1, s)
                : npp <= 7 ? launch_gram<DIM, 7, true>(a, S, b0, b1, s)
                : npp <= 8 ? launch_gram<DIM, 8, true>(a, S, b0, b1, s)
                           : launch_gram<DIM, 40, true>(a, S, b0, b1, s);
        if (e == cudaSuccess) e = launch_qr_any(a, S, lpp, b0, b1 - b0, s);
        if (e == cudaSuccess) e = launch_chain<DIM>(a, S, h.ngroups, b0, b1, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

Split make_split(const AsmTables& h, int flags, bool vjp = false) {
    Split S{};
    const bool fast = (flags & DCPSE_ASSEMBLE_FAST_FLAG) != 0;
    S.vjp = vjp;
    S.gstride = (h.npairs + (vjp ? h.nu : 0) + 1) & ~1;
    S.nmax = 1;
    S.qwords = 1;
    int off = 0;
    for (int g = 0; g < h.ngroups; ++g) {
        const int n = h.gn[g];
        S.nrhs[g] = vjp ? 2 : (fast ? h.nout_rhs[g] : h.nterm_rhs[g]);
        S.c_off[g] = off;
        off += n * S.nrhs[g];
        S.nmax = std::max(S.nmax, n);
        S.qtab += n * (n + 1) / 2;
        S.nrmax = std::max(S.nrmax, S.nrhs[g]);
        S.qwords = std::max(S.qwords, n * (n + S.nrhs[g]) + n * S.nrhs[g]);
    }
    S.cstride = (off + 1) & ~1;
    S.ldb = (h.nu + (vjp ? 1 : 0)) | 1;
    S.nslots = h.nslots;
    S.nout = h.noutputs;
    S.npairs = h.npairs;
    return S;
}

int tc_kpad(int maxk) { return ((std::max(maxk, 1) + 15) / 16) * 16; }

}  // namespace

bool assembly_uses_tc(const AsmTables& h, int flags, int maxk) {
    if (!(flags & DCPSE_ASSEMBLE_TC) || !(flags & DCPSE_ASSEMBLE_FAST_FLAG) || h.nu > kTcMaxNu || maxk > kTcMaxK)
        return false;
    // the planes, the monomial scratch and the pair sums fit in one CTA
    const TcLayout L = tc_layout(maxk, h.npairs);
    return L.bytes + 4096 <= (size_t)smem_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, 227 * 1024);
}

int64_t assembly_scratch_bytes(const AsmTables& h, int flags, int maxk) {
    const Split S = make_split(h, flags);
    int64_t b = (int64_t)(S.gstride + S.cstride + 4 + (int64_t)h.dim * std::max(maxk, 1)) * (int64_t)sizeof(double) +
                (int64_t)sizeof(int32_t);
    if (assembly_uses_tc(h, flags, maxk))
        b += (int64_t)h.nu * tc_kpad(maxk) * (int64_t)sizeof(double) + 32 * (int64_t)sizeof(int32_t);
    return b;
}

int64_t vjp_scratch_bytes(const AsmTables& h, int maxk) {
    const Split S = make_split(h, DCPSE_ASSEMBLE_FAST_FLAG, true);
    return (int64_t)(S.gstride + S.cstride + 4 + (int64_t)(h.dim + 1) * std::max(maxk, 1)) * (int64_t)sizeof(double) +
           (int64_t)sizeof(int32_t);
}

int64_t assembly_qr_ws_bytes(const AsmTables& h, int flags) {
    Split S = make_split(h, flags);
    if (qr_bytes(S, 32, false) <= (size_t)smem_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, 227 * 1024)) return 0;
    const int64_t slots = (int64_t)num_sms() * kQrGlobalPerSm;
    return slots * ((int64_t)qr_pstride(S, 32) * (int64_t)sizeof(double) + (int64_t)S.nmax * (int64_t)sizeof(int));
}

int64_t binning_tmp_elems(int64_t n, int maxk, int width) {
    const int64_t nb = maxk / (width > 0 ? width : 1) + 1;
    return nb + 1 + scan_tmp_elems(nb);
}

namespace {
__global__ void khist_kernel(const int64_t* __restrict__ rowptr, int64_t n, int width, int32_t* __restrict__ hist) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&hist[(int)(rowptr[p + 1] - rowptr[p]) / width], 1);
}

__global__ void kscatter_kernel(const int64_t* __restrict__ rowptr, int64_t n, int width, int64_t* fill,
                                int32_t* __restrict__ order) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        const int b = (int)(rowptr[p + 1] - rowptr[p]) / width;
        order[atomicAdd((unsigned long long*)&fill[b], 1ull)] = (int32_t)p;
    }
}
}  // namespace

cudaError_t bin_by_count(const int64_t* rowptr, int64_t n, int maxk, int width, int32_t* order, int32_t* hist,
                         int64_t* tmp64, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    if (width < 1) width = 1;
    const int64_t nb = maxk / width + 1;
    int64_t* starts = tmp64;            // nb + 1
    int64_t* scan_tmp = tmp64 + nb + 1;
    cudaError_t e = cudaMemsetAsync(hist, 0, sizeof(int32_t) * nb, s);
    if (e != cudaSuccess) return e;
    const int grid = (int)std::min<int64_t>((n + 255) / 256, (int64_t)num_sms() * 8);
    khist_kernel<<<grid, 256, 0, s>>>(rowptr, n, width, hist);
    e = exclusive_scan_i32(hist, nb, starts, scan_tmp, s);
    if (e != cudaSuccess) return e;
    kscatter_kernel<<<grid, 256, 0, s>>>(rowptr, n, width, starts, order);
    return cudaGetLastError();
}

cudaError_t assemble(const AsmArgs& a, const AsmTables& h, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    if (!a.scratch || a.scratch_particles < 1) return cudaErrorInvalidValue;
    Split S = make_split(h, a.flags);
    const int64_t nb = a.scratch_particles;
    S.gram = a.scratch;
    S.coef = S.gram + nb * S.gstride;
    S.maxk = std::max(a.maxk, 1);
    S.ustride = (int64_t)h.dim * S.maxk;
    S.scale = S.coef + nb * S.cstride;
    S.usc = S.scale + nb * 4;
    S.tc = assembly_uses_tc(h, a.flags, a.maxk);
    if (S.tc) {
        S.kpad = tc_kpad(a.maxk);
        S.bmat = S.usc + nb * S.ustride;
        S.bexp = reinterpret_cast<int32_t*>(S.bmat + nb * (int64_t)h.nu * S.kpad);
        S.gst = S.bexp + nb * 32;
    } else {
        S.gst = reinterpret_cast<int32_t*>(S.usc + nb * S.ustride);
    }
    int lpp = a.qr_lanes;
    if (lpp != 1 && lpp != 2 && lpp != 4 && lpp != 8 && lpp != 16 && lpp != 32) lpp = qr_lanes_auto(S, std::min(a.n, nb));
    if (a.qws) {
        // large bases: one warp per particle, the work space in global memory
        lpp = 32;
        S.qws = a.qws;
        S.qperm = reinterpret_cast<int*>(a.qws + (int64_t)num_sms() * kQrGlobalPerSm * qr_pstride(S, 32));
    } else if (qr_bytes(S, lpp, false) > (size_t)smem_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, 227 * 1024)) {
        // a lane grouping whose work space does not fit is refused before any launch
        return cudaErrorInvalidConfiguration;
    }
    if (h.dim == 3) return dispatch<3>(a, h, S, lpp, s);
    if (h.dim == 2) return dispatch<2>(a, h, S, lpp, s);
    return dispatch<1>(a, h, S, lpp, s);
}

cudaError_t vjp_entries(const AsmArgs& a, const AsmTables& h, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    if (!a.scratch || a.scratch_particles < 1) return cudaErrorInvalidValue;
    Split S = make_split(h, DCPSE_ASSEMBLE_FAST_FLAG, true);
    const int64_t nb = a.scratch_particles;
    S.gram = a.scratch;
    S.coef = S.gram + nb * S.gstride;
    S.maxk = std::max(a.maxk, 1);
    S.ustride = (int64_t)(h.dim + 1) * S.maxk;
    S.scale = S.coef + nb * S.cstride;
    S.usc = S.scale + nb * 4;
    S.gst = reinterpret_cast<int32_t*>(S.usc + nb * S.ustride);
    int lpp = a.qr_lanes;
    if (lpp != 1 && lpp != 2 && lpp != 4 && lpp != 8 && lpp != 16 && lpp != 32) lpp = qr_lanes_auto(S, std::min(a.n, nb));
    if (qr_bytes(S, lpp, false) > (size_t)smem_attr(cudaDevAttrMaxSharedMemoryPerBlockOptin, 227 * 1024))
        lpp = 32;  // a lane grouping chosen for the assembly's right-hand sides
    if (h.dim == 3) return vjp_run<3>(a, h, S, lpp, s);
    if (h.dim == 2) return vjp_run<2>(a, h, S, lpp, s);
    return vjp_run<1>(a, h, S, lpp, s);
}

}  // namespace dcpse
