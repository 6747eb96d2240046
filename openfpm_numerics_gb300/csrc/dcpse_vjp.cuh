// dcpse_vjp.cuh -- position VJP of the assembly: the per-entry chain rule
// (included by dcpse_assemble.cu, whose eps, Gram and QR kernels run first).
//
// For particle p and basis group g the Gram kernel leaves A and s = sum_q
// omega_q c_q v_q (its extra column E c), the QR kernel a~ = A^-1 b~ and
// lambda = A^-1 s.  With r_q = c_q - v_q.lambda, va_q = v_q.a~ and
// e = eps^-|alpha| (dcpse_adjoint.cu):
//   gu_q = sum_g e omega (r grad(v.a~) - va grad(v.lambda)) - 2 e omega va r u_q
// and grad x_pq = gu_q / eps + dd sign(x_pq), dd from the eps terms.
//
// FP64-pipe bound (a warp instruction holds it 16 cycles).  One kernel did all
// of it, a warp per particle: its QR ran a warp wide on at most 21 columns, and
// the chain rule formed every derivative monomial from powers, per basis
// function and group (3D Gradient + Laplacian: about 580 FP64 instructions per
// 32 entries).  Here the monomials come from the monomial program (16
// products, on the integer pipes), the coefficient of each union monomial is
// summed over the groups first and meets its derivatives, which are other slots
// of the same program, once: about 165 per 32 entries.

struct ChainShared {
    ProgShared P;
    unsigned char gslot[kMaxGroups][kMaxBasisSmall];  // slot of basis function i of group g
    unsigned char guse[kMaxUnion][kMaxGroups];        // 1 + basis index of union monomial j in group g, 0: absent
    unsigned char dslot[kMaxUnion][kMaxDim];
    unsigned char uexp[kMaxUnion][kMaxDim];
};

// small integers as doubles (an int -> double conversion runs on the FP64 pipe)
__constant__ double kSmallInt[kMaxExp + 1] = {0.0, 1.0, 2.0, 3.0, 4.0, 5.0, 6.0, 7.0, 8.0};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One warp per particle, one neighbour row per lane.  Per warp in shared
// memory: (a~, lambda) pairs of every group, the monomial slots of 32 rows and
// two coefficients per group and row.
template <int DIM>
__global__ void __launch_bounds__(256) vjp_chain_kernel(AsmArgs a, Split S, int64_t b0, int64_t b1) {
    extern __shared__ double smem[];
    __shared__ ChainShared X;
    const AsmTables& T = *a.tab;
    const int ngroups = T.ngroups, nu = T.nu;
    for (int e = threadIdx.x; e < nu * kMaxGroups; e += blockDim.x) X.guse[e / kMaxGroups][e % kMaxGroups] = 0;
    for (int e = threadIdx.x; e < nu * kMaxDim; e += blockDim.x) {
        X.dslot[e / kMaxDim][e % kMaxDim] = T.dslot[e / kMaxDim][e % kMaxDim];
        X.uexp[e / kMaxDim][e % kMaxDim] = T.uexp[e / kMaxDim][e % kMaxDim];
    }
    stage_program(T, X.P);  // (ends with a barrier)
    for (int g = 0; g < ngroups; ++g)
        for (int i = threadIdx.x; i < T.gn[g]; i += blockDim.x) {
            X.gslot[g][i] = T.uslot[T.gidx[g][i]];
            X.guse[T.gidx[g][i]][g] = (unsigned char)(i + 1);
        }
    __syncthreads();
    const Fma F;
    const int lane = threadIdx.x & 31;
    const int wib = threadIdx.x >> 5;
    double* Cs = smem + (size_t)wib * (S.cstride + (S.nslots + 2 * ngroups) * 32);
    double* V = Cs + S.cstride;
    double* CC = V + S.nslots * 32;
    const int nprog = T.nprog;
    const int wpc = blockDim.x >> 5;
    const int64_t nw = (int64_t)gridDim.x * wpc;
    for (int64_t it = b0 + (int64_t)blockIdx.x * wpc + wib; it < b1; it += nw) {
        const int64_t slot = it - b0;
        const int64_t p = it;
        const int64_t beg = a.rowptr[p];
        const int k = (int)(a.rowptr[p + 1] - beg);
        double* __restrict__ Gp = a.gentry + beg * DIM;
        bool ok = true;  // every group assembled and regular
        for (int g = 0; g < ngroups; ++g) ok = ok && group_status(S.gst[slot], g) == ST_OK;
        if (!ok) {  // warp-uniform
            for (int e = lane; e < k * DIM; e += 32) Gp[e] = 0.0;
            if (lane < DIM) a.gown[p * DIM + lane] = 0.0;
            continue;
        }
        for (int e = lane; e < S.cstride; e += 32) Cs[e] = S.coef[slot * S.cstride + e];
        __syncwarp();
        const double ieps = S.scale[slot * 4 + 1];
        // d Phi / d eps from e = eps^-|alpha|: -|alpha| e s^T a~ / eps
        double Dsc = 0.0;
        const double* sv = S.gram + slot * S.gstride + S.npairs;
        for (int g = 0; g < ngroups; ++g) {
            const double c = -kSmallInt[T.gord[g]] * a.eip_group[(int64_t)g * a.n + p];
            for (int i = lane; i < T.gn[g]; i += 32)
                Dsc = fma(c * sv[T.gidx[g][i]], Cs[S.c_off[g] + 2 * i], Dsc);
        }
        const double fp = a.f[p];
        const double* Ur = S.usc + slot * S.ustride;
        double gsum = 0.0;
        for (int c0 = 0; c0 < k; c0 += kCh) {
            const int q = c0 + lane;
            if (q >= k) break;  // rows of this lane are done; no warp sync below
            double u[DIM], gu[DIM];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                u[d] = Ur[d * S.maxk + q];
                gu[d] = 0.0;
            }
            const double E = Ur[DIM * S.maxk + q];
            const double om = F.prod(E, E);
            const double cq = F.add(a.f[a.cols[beg + q]], -fp);
            bool unit = true;
#pragma unroll
            for (int d = 0; d < DIM; ++d) unit = unit && unit_range_or_zero(u[d]);
            if (unit)
                monomials_int<DIM>(u, V, X.P, nprog, lane);
            else
                monomials<DIM>(u, V, X.P, nprog, lane);
            double ga = 0.0;
            for (int g = 0; g < ngroups; ++g) {
                const double* C = Cs + S.c_off[g];
                const int n = T.gn[g];
                double va = 0.0, vl = 0.0;
                for (int i = 0; i < n; ++i) {
                    const double v = V[X.gslot[g][i] * 32 + lane];
                    va = fma(v, C[2 * i], va);
                    vl = fma(v, C[2 * i + 1], vl);
                }
                const double eo = F.prod(a.eip_group[(int64_t)g * a.n + p], om);
                const double c1 = F.prod(eo, F.add(cq, -vl));
                ga = fma(va, c1, ga);
                CC[(2 * g) * 32 + lane] = c1;
                CC[(2 * g + 1) * 32 + lane] = -F.prod(eo, va);
            }
            for (int j = 0; j < nu; ++j) {
                double beta = 0.0;
                for (int g = 0; g < ngroups; ++g) {
                    const int i = X.guse[j][g];
                    if (i == 0) continue;
                    const double* C = Cs + S.c_off[g] + 2 * (i - 1);
                    beta = fma(CC[(2 * g) * 32 + lane], C[0], beta);
                    beta = fma(CC[(2 * g + 1) * 32 + lane], C[1], beta);
                }
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const int e = X.uexp[j][d];
                    if (e == 0) continue;
                    const double b = e == 1 ? beta : F.prod(beta, kSmallInt[e]);
                    gu[d] = fma(b, V[X.dslot[j][d] * 32 + lane], gu[d]);
                }
            }
            ga = F.add(-ga, -ga);
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                gu[d] = fma(ga, u[d], gu[d]);
                gsum = fma(gu[d], u[d], gsum);
                Gp[q * DIM + d] = F.prod(gu[d], ieps);
            }
        }
        // the eps terms, along sign(x_pq) (u has x_pq's sign); without them
        // for a fixed eps
        const double dd = a.eps_fixed ? 0.0 : warp_sum(Dsc - gsum) * ieps / ((double)k * a.h_over_eps);
        const double dz = 0.0 * dd;  // (NaN where dd is not finite)
        double own[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) own[d] = 0.0;
        for (int q = lane; q < k; q += 32) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
                const double o = Ur[d * S.maxk + q];
                const double sg = is_zero(o) ? dz : ((dhi(o) >> 31) ? -dd : dd);
                const double v = F.add(Gp[q * DIM + d], sg);
                Gp[q * DIM + d] = v;
                own[d] = F.add(v, own[d]);
            }
        }
#pragma unroll
        for (int d = 0; d < DIM; ++d) {
            own[d] = warp_sum(own[d]);
            if (lane == d) a.gown[p * DIM + d] = own[d];
        }
        __syncwarp();
    }
}
