// dcpse_nbr_group.cuh -- neighbour search by groups of cells (included by
// dcpse_neighbors.cu).
//
// One set on the packed grid (cells of side >= rc / 2).  A warp takes the
// particles of G^DIM cells and the (G + 4)^DIM cells around them: every
// candidate is located and loaded once for all of the group's particles, U x 32
// at a time in registers, and each particle is tested against them from a
// shared-memory broadcast.  The accepted columns go to a staging row per
// particle (cap entries), so that one search serves the counts and the columns;
// the rows are sorted out of it.  A row longer than cap only counts: the caller
// then runs the fill pass.
//
// Bound by instructions issued.  A warp per particle located and loaded its 343
// candidates (3D, 2.74 per cell) for itself, twice (count and fill): about 1030
// instructions each.  Groups of 2^3 cells test 592 candidates per particle, at
// 0.6 instructions each, and spread the loading over 22 particles.
//
// The decisions are those of the packed kernels: FP32 coordinates relative to
// the group's lower corner (within 4 + G cell sides, so the margin's error
// bound of 200 u S^2 holds: each coordinate is off by at most 2 u times that),
// the FP64 predicate within the margin and for NaN.
#pragma once

// Most steps of one warp, particles x chunks of 32 U candidates; the particles of
// a group beyond it go to the warp-per-particle search (stage_left).  Cells take
// half the largest radius as their side, so a group of a part whose own radii are
// r times smaller holds r^2 (2D) or r^3 times the particles and as many times the
// candidates, all for one warp: 2e5 points in 2D, 30 % of them in a patch of
// radii 8 times smaller, took 72 ms without a bound, 3.4 ms with one (5.3 ms by
// two passes of a warp per particle).  Ordinary groups take about 110 steps, those
// of a part with half the radii 1,500.  Between 512 and 8192, 1024 was fastest or
// within 2 % of it on nearly all of 33 sets (1 to 8 times smaller radii, clusters,
// grids of few cells): that part at 2e5 points 0.94 ms with 2048, 0.64 with 1024.
constexpr int64_t kGroupSteps = 1024;

struct GroupGrid {
    int ng[3];       // groups per axis
    int64_t total;
};

template <int DIM, int G, int U>
__global__ void __launch_bounds__(256) nbr_group_kernel(NbrArgs a, GroupGrid gg, int32_t* __restrict__ counts,
                                                        int* maxk, int32_t* __restrict__ stage, int cap,
                                                        int32_t* __restrict__ left) {
    constexpr int W = G + 2 * kPackR;                 // cells of the region per axis
    constexpr int NR = DIM == 3 ? W * W : W;          // its rows along axis 0
    constexpr int NS = 2 * NR;                        // segments: a row, and its part wrapped around axis 0
    constexpr int PR = DIM == 3 ? G * G : G;          // rows of the group's own cells
    __shared__ int s_end[8][NS], s_beg[8][NS], s_dx[8][NS];
    __shared__ float4 s_p[8][32];   // x, y, z, lower threshold
    __shared__ float2 s_q[8][32];   // upper threshold, particle
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned lt_mask = (1u << lane) - 1u;
    int *end = s_end[wib], *beg = s_beg[wib], *sdx = s_dx[wib];
    const int nc0 = a.cells.nc[0], nc1 = a.cells.nc[1], nc2 = a.cells.nc[2];
    int kmax = 0;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t g = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; g < gg.total; g += nw) {
        const int bx = (int)(g % gg.ng[0]) * G;
        const int by = (int)(g / gg.ng[0] % gg.ng[1]) * G;
        const int bz = DIM == 3 ? (int)(g / gg.ng[0] / gg.ng[1]) * G : 0;
        // the group's particles: row r holds cells bx .. of row (by + r % G, bz + r / G)
        int pstart = 0, plen = 0;
        if (lane < PR) {
            const int y = by + lane % G, z = DIM == 3 ? bz + lane / G : 0;
            if (y < nc1 && z < nc2) {
                const int64_t row = (int64_t)nc0 * (y + (int64_t)nc1 * z);
                pstart = (int)a.cstart[row + bx];
                plen = (int)a.cstart[row + min(bx + G, nc0)] - pstart;
            }
        }
        int pend = plen;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(full, pend, o);
            if (lane >= o) pend += v;
        }
        const int np = __shfl_sync(full, pend, 31);
        if (np == 0) continue;
        // the region's segments of the cell-ordered set
        int total = 0;
        for (int s0 = 0; s0 < NS; s0 += 32) {
            const int s = s0 + lane, r = s >> 1;
            int b = 0, len = 0, dx = 0;
            if (s < NS) {
                int y = by + r % W - kPackR, z = DIM == 3 ? bz + r / W - kPackR : 0;
                if (a.geom.per[1]) y = y < 0 ? y + nc1 : (y >= nc1 ? y - nc1 : y);
                if (DIM == 3 && a.geom.per[2]) z = z < 0 ? z + nc2 : (z >= nc2 ? z - nc2 : z);
                int x0 = bx - kPackR, x1 = bx + G - 1 + kPackR;  // inclusive
                if ((s & 1) == 0) {
                    x0 = max(x0, 0);
                    x1 = min(x1, nc0 - 1);
                } else if (!a.geom.per[0]) {
                    x1 = x0 - 1;
                } else if (x0 < 0) {  // the cells below 0 are those below nc0
                    x0 += nc0;
                    x1 = nc0 - 1;
                    dx = -nc0;
                } else {              // (empty unless the row passes nc0)
                    x0 = 0;
                    x1 -= nc0;
                    dx = nc0;
                }
                if (y >= 0 && y < nc1 && z >= 0 && z < nc2 && x0 <= x1) {
                    const int64_t row = (int64_t)nc0 * (y + (int64_t)nc1 * z);
                    b = (int)a.cstart[row + x0];
                    len = (int)a.cstart[row + x1 + 1] - b;
                }
            }
            int e = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(full, e, o);
                if (lane >= o) e += v;
            }
            if (s < NS) {
                end[s] = total + e;
                beg[s] = b - (total + e - len);  // + position in the concatenation
                sdx[s] = dx - bx;
            }
            total += __shfl_sync(full, e, 31);
        }
        __syncwarp();
        if ((int64_t)np * ((total + 32 * U - 1) / (32 * U)) > kGroupSteps) {
            // a crowd: its particles to the warp-per-particle search
            int at = lane == 0 ? atomicAdd(&maxk[1], np) : 0;
            at = __shfl_sync(full, at, 0);
            for (int r = 0; r < PR; ++r) {
                const int t0 = __shfl_sync(full, pstart, r), len = __shfl_sync(full, plen, r);
                for (int i = lane; i < len; i += 32) left[at + i] = a.cidx[t0 + i];
                at += len;
            }
            __syncwarp();  // the next group rewrites the segments
            continue;
        }
        for (int p0 = 0; p0 < np; p0 += 32) {
            const int nb = min(32, np - p0);
            // lane i's particle
            int pid = 0;
            {
                const int i = p0 + lane;
                int r = 0;
#pragma unroll
                for (int t = 0; t < PR - 1; ++t) r += i >= __shfl_sync(full, pend, t);
                const int t = i - (__shfl_sync(full, pend, r) - __shfl_sync(full, plen, r)) + __shfl_sync(full, pstart, r);
                float4 P = make_float4(0.f, 0.f, 0.f, 0.f);
                float tout = 0.f;
                if (lane < nb) {
                    pid = a.cidx[t];
                    const float4 rel = a.srel[t];
                    P.x = rel.x + (float)(__float_as_int(rel.w) - bx) * a.csf[0];
                    P.y = rel.y + (float)(r % G) * a.csf[1];
                    if (DIM == 3) P.z = rel.z + (float)(r / G) * a.csf[2];
                    const double rc = a.rcut_pp ? a.rcut_pp[pid] : a.rcut;
                    const double rc2 = rc * rc;
                    P.w = (float)(rc2 - a.band);
                    tout = (float)(rc2 + a.band);
                }
                s_p[wib][lane] = P;
                s_q[wib][lane] = make_float2(tout, __int_as_float(pid));
            }
            __syncwarp();
            int k = 0;  // lane i: accepted so far by particle i
            for (int c0 = 0; c0 < total; c0 += 32 * U) {
                float x[U], y[U], z[U];
                int32_t q[U];
                int t[U];
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int c = c0 + 32 * u + lane;
                    // outside every cutoff
                    x[u] = 3.0e38f;
                    y[u] = z[u] = 0.f;
                    q[u] = -1;
                    t[u] = 0;
                    if (c < total) {
                        int lo = 0, hi = NS - 1;  // first segment whose end exceeds c
                        while (lo < hi) {
                            const int mid = (lo + hi) >> 1;
                            if (end[mid] > c)
                                hi = mid;
                            else
                                lo = mid + 1;
                        }
                        t[u] = beg[lo] + c;
                        const float4 rel = a.srel[t[u]];
                        q[u] = a.cidx[t[u]];
                        const int r = lo >> 1;
                        x[u] = rel.x + (float)(__float_as_int(rel.w) + sdx[lo]) * a.csf[0];
                        y[u] = rel.y + (float)(r % W - kPackR) * a.csf[1];
                        if (DIM == 3) z[u] = rel.z + (float)(r / W - kPackR) * a.csf[2];
                    }
                }
                for (int i = 0; i < nb; ++i) {
                    const float4 P = s_p[wib][i];
                    const float2 Q = s_q[wib][i];
                    const int pi = __float_as_int(Q.y);
                    int ki = __shfl_sync(full, k, i);
                    bool acc[U], exact[U], any = false;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const float o0 = P.x - x[u], o1 = P.y - y[u];
                        float d2 = fmaf(o1, o1, o0 * o0);
                        if (DIM == 3) {
                            const float o2 = P.z - z[u];
                            d2 = fmaf(o2, o2, d2);
                        }
                        acc[u] = d2 < P.w;
                        exact[u] = !acc[u] && !(d2 > Q.x);  // the band, NaN
                        any = any || exact[u];
                    }
                    // a warp-uniform branch: the FP64 test issues only when
                    // some lane needs it
                    if (__any_sync(full, any)) {
                        const double rc = a.rcut_pp ? a.rcut_pp[pi] : a.rcut;
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            if (exact[u] && q[u] >= 0) {
                                // (a particle outside a periodic box keeps the +-2
                                // cells of the cell it was clamped into)
                                double o[DIM];
                                bool near = true;
#pragma unroll
                                for (int d = 0; d < DIM; ++d) {
                                    const double xp = a.pd[(int64_t)pi * DIM + d], xq = a.spos[(int64_t)t[u] * DIM + d];
                                    o[d] = offset1(a.geom, d, xp, xq);
                                    const int nc = a.cells.nc[d];
                                    int dc = abs(cell_coord(xp, a.cells.lo[d], a.cells.ics[d], nc) -
                                                 cell_coord(xq, a.cells.lo[d], a.cells.ics[d], nc));
                                    if (a.geom.per[d]) dc = min(dc, nc - dc);
                                    near = near && dc <= kPackR;
                                }
                                acc[u] = near && norm2<DIM>(o) < rc * rc;
                            }
                    }
                    int32_t* row = stage + (int64_t)pi * cap;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        const bool ok = acc[u] && !(a.self_skip && q[u] == pi);
                        const unsigned bal = __ballot_sync(full, ok);
                        const int at = ki + __popc(bal & lt_mask);
                        if (ok && at < cap) row[at] = q[u];
                        ki += __popc(bal);
                    }
                    if (lane == i) k = ki;
                }
            }
            if (lane < nb) {
                counts[pid] = k;
                kmax = max(kmax, k);
            }
            __syncwarp();  // the next batch rewrites the particles
        }
        __syncwarp();      // the next group rewrites the segments
    }
    kmax = __reduce_max_sync(full, kmax);
    if (lane == 0 && kmax > 0) atomicMax(maxk, kmax);
}

// Cells per group and axis: 2 in 3D (22 particles at the lists' usual 2.74 per
// cell), 4 in 2D (38), one or two where that would leave the GPU's schedulers
// without a warp each; none that would put a periodic axis' cells twice into a
// region.  0: the group search does not serve.
inline int group_side(const NbrArgs& a) {
    if (!a.packed || !a.fast || a.dim < 2) return 0;
    const int64_t warps = (int64_t)num_sms() * 8;
    for (int G : {4, 2, 1}) {
        if (G == 4 && a.dim == 3) continue;
        bool fits = true;
        int64_t groups = 1;
        for (int d = 0; d < a.dim; ++d) {
            fits = fits && (!a.geom.per[d] || a.cells.nc[d] >= G + 2 * kPackR);
            groups *= (a.cells.nc[d] + G - 1) / G;
        }
        if (fits && (groups >= warps || G == 1)) return G;
    }
    return 0;
}

template <int DIM, int G, int U>
cudaError_t launch_group(const NbrArgs& a, int32_t* counts, int* maxk, int32_t* stage, int cap, int32_t* left,
                         cudaStream_t s) {
    GroupGrid gg{};
    gg.total = 1;
    for (int d = 0; d < 3; ++d) {
        gg.ng[d] = d < DIM ? (a.cells.nc[d] + G - 1) / G : 1;
        gg.total *= gg.ng[d];
    }
    const int64_t blocks = (gg.total + 7) / 8;
    nbr_group_kernel<DIM, G, U><<<(unsigned)std::min<int64_t>(blocks, 0x7fffffff), 256, 0, s>>>(a, gg, counts, maxk,
                                                                                              stage, cap, left);
    return cudaGetLastError();
}
