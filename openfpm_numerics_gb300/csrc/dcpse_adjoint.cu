// dcpse_adjoint.cu -- vector-Jacobian products of the batched DC-PSE apply.
//
// The reference has no adjoint; these are the derivatives of its operator
// (src/DCPSE/Dcpse.hpp:690-809 assembly, :467-499 apply) with the
// neighbour lists held fixed.  With outputs y_o,p = sum_q W_o,pq (f_q - f_p):
//
//  * field VJP:   (dL/df)_q = sum_o [ sum_{p: q in N(p)} W_o,pq g_o,p
//                                     - g_o,q sum_r W_o,qr ]
//    through a transposed neighbour list (rows sorted by source particle, so
//    the sums run in a fixed order), built once per list;
//
//  * position VJP: for particle p and basis g, with c_q = f_q - f_p,
//    omega_q = exp(-|u_q|^2), u_q = x_pq / eps, v_q = m(u_q),
//    A = sum_q omega_q v_q v_q^T,  b~ = sum_o g_o,p b_o,g,
//    Phi = eps^-|alpha| s^T a~,  s = sum_q c_q omega_q v_q,  a~ = A^-1 b~:
//      lambda = A^-1 s,
//      dPhi/domega_q = e (v_q.a~)(c_q - v_q.lambda),
//      dPhi/dv_q     = e omega_q [ (c_q - v_q.lambda) a~ - (v_q.a~) lambda ],
//    chained through omega_q, v_q(u_q), u_q = x_pq/eps and
//    eps = sum_q |x_pq|_1 / (k HOverEpsilon), eps^-|alpha| into per-entry
//    contributions G_pq:  grad x_p += G_pq,  grad x_q -= G_pq.
//
// FP64 throughout.  The eps, Gram and QR kernels are the assembly's
// (dcpse_assemble.cu, dcpse_vjp.cuh); this unit holds the transposed lists, the
// field VJP and the gather of the position VJP's per-entry contributions.
#include "dcpse_internal.h"

namespace dcpse {
namespace {

// ---------------------------------------------------- transposed CSR build --
__global__ void tcount_kernel(const int32_t* __restrict__ cols, int64_t nnz, int32_t* __restrict__ cnt) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < nnz; j += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&cnt[cols[j]], 1);
}

__global__ void tfill_kernel(const int64_t* __restrict__ rowptr, const int32_t* __restrict__ cols, int64_t n,
                             int64_t* fill, int32_t* __restrict__ tsrc, int64_t* __restrict__ tidx) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        for (int64_t j = rowptr[p]; j < rowptr[p + 1]; ++j) {
            unsigned long long slot = atomicAdd((unsigned long long*)&fill[cols[j]], 1ull);
            tsrc[slot] = (int32_t)p;
            tidx[slot] = j;
        }
    }
}

// warp per transposed row: order entries by source particle (distinct)
__global__ void tsort_kernel(const int64_t* __restrict__ trow, int64_t n, const int32_t* __restrict__ src_in,
                             const int64_t* __restrict__ idx_in, int32_t* __restrict__ src_out,
                             int64_t* __restrict__ idx_out) {
    const int lane = threadIdx.x & 31;
    const int64_t w0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t q = w0; q < n; q += nw) {
        const int64_t b = trow[q];
        const int k = (int)(trow[q + 1] - b);
        for (int i0 = 0; i0 < k; i0 += 32) {
            const int i = i0 + lane;
            const int32_t v = (i < k) ? src_in[b + i] : 0;
            int rank = 0;
            for (int j = 0; j < k; ++j) rank += (src_in[b + j] < v);
            if (i < k) {
                src_out[b + rank] = v;
                idx_out[b + rank] = idx_in[b + i];
            }
        }
    }
}

__global__ void rowsum_kernel(const int64_t* __restrict__ rowptr, int64_t n, int nout, const double* __restrict__ w64,
                              const float* __restrict__ w32, int64_t ws, double* __restrict__ rs) {
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
        for (int o = 0; o < nout; ++o) {
            double s = 0.0;
            for (int64_t j = rowptr[p]; j < rowptr[p + 1]; ++j)
                s = s + (w64 ? w64[(int64_t)o * ws + j] : (double)w32[(int64_t)o * ws + j]);
            rs[(int64_t)o * n + p] = s;
        }
    }
}

// (L^T g)_q in FP64, thread per transposed row, fixed order
__global__ void vjp_field_kernel(const int64_t* __restrict__ trow, const int32_t* __restrict__ tsrc,
                                 const int64_t* __restrict__ tidx, int64_t n, int nout, const double* __restrict__ w64,
                                 const float* __restrict__ w32, int64_t ws, const double* __restrict__ rs,
                                 const double* __restrict__ g, double* __restrict__ out) {
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        double acc = 0.0;
        for (int64_t t = trow[q]; t < trow[q + 1]; ++t) {
            const int64_t j = tidx[t];
            const int64_t p = tsrc[t];
            for (int o = 0; o < nout; ++o) {
                const double w = w64 ? w64[(int64_t)o * ws + j] : (double)w32[(int64_t)o * ws + j];
                acc = fma(w, g[(int64_t)o * n + p], acc);
            }
        }
        for (int o = 0; o < nout; ++o) acc = fma(-g[(int64_t)o * n + q], rs[(int64_t)o * n + q], acc);
        out[q] = acc;
    }
}

// (L^T g)_q on the sliced ELL layout of the transposed list (slices of 32
// rows stored entry-major, rows sorted by length within windows of 256; the
// weights of every output gathered into it): a row per thread, coalesced
// column and weight streams, the cotangents gathered per output.  Each row
// sums its entries in the CSR kernel's order (by source particle, outputs
// innermost) and subtracts the row-sum terms last, so the results are the
// CSR kernel's bit for bit; padding entries have weight 0 on the row itself.
// FP32 weights come widened to double at the layout's build (exact, as the
// CSR kernel's per-use conversion is, which runs at the FP64 rate here).
template <int NO>
__global__ void __launch_bounds__(256) vjp_field_sell_kernel(VjpSellArgs a) {
    const double* __restrict__ wt = a.w;
    const int lane = threadIdx.x & 31;
    constexpr int U = NO <= 2 ? 4 : 2;  // entries in flight per thread
    for (int64_t win = blockIdx.x; win < a.nwin; win += gridDim.x) {
        const int64_t s = win * 8 + (threadIdx.x >> 5);
        const int32_t row = a.srow[s * 32 + lane];
        if (row < 0) continue;
        const int64_t b = a.off[s];
        const int L = (int)((a.off[s + 1] - b) / 32);
        const int32_t* __restrict__ c = a.cols + b + lane;
        const double* __restrict__ w = wt + b + lane;
        double acc = 0.0;
        for (int j0 = 0; j0 < L; j0 += U) {
            int32_t q[U];
            double wv[U][NO], gv[U][NO];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int j = j0 + u;
                q[u] = j < L ? c[(int64_t)j * 32] : row;
#pragma unroll
                for (int o = 0; o < NO; ++o) wv[u][o] = j < L ? w[(int64_t)o * a.total + (int64_t)j * 32] : 0.0;
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int o = 0; o < NO; ++o) gv[u][o] = a.g[(int64_t)o * a.n + q[u]];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (j0 + u < L) {
#pragma unroll
                    for (int o = 0; o < NO; ++o) acc = fma(wv[u][o], gv[u][o], acc);
                }
            }
        }
#pragma unroll
        for (int o = 0; o < NO; ++o) acc = fma(-a.g[(int64_t)o * a.n + row], a.rs[(int64_t)o * a.n + row], acc);
        a.out[row] = acc;
    }
}

// transposed weights of every output, as doubles: wt[o * nnz + t] =
// w[o * ws + tidx[t]] (FP32 weights widened, exactly)
template <typename T>
__global__ void transpose_outputs_kernel(const int64_t* __restrict__ tidx, int64_t nnz, int nout,
                                         const T* __restrict__ w, int64_t ws, double* __restrict__ wt) {
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nnz; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t j = tidx[t];
        for (int o = 0; o < nout; ++o) wt[(int64_t)o * nnz + t] = (double)w[(int64_t)o * ws + j];
    }
}

// grad x_i -= sum over the entries pointing at i of their gradients: eight lanes
// per transposed row (the row's own sums are in grad already, vjp_entries)
template <int DIM>
__global__ void __launch_bounds__(256) vjp_gather_kernel(const int64_t* __restrict__ trow,
                                                         const int64_t* __restrict__ tidx, int64_t n,
                                                         const double* __restrict__ G, double* __restrict__ grad) {
    const int sub = threadIdx.x & 7;
    const int64_t nr = ((int64_t)gridDim.x * blockDim.x) >> 3;
    const int64_t i0 = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3;
    for (int64_t w = i0 - ((threadIdx.x >> 3) & 3); w < n; w += nr) {  // (warp-uniform)
        const int64_t i = w + ((threadIdx.x >> 3) & 3);
        double s[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) s[d] = 0.0;
        const int64_t e = i < n ? trow[i + 1] : 0;
        for (int64_t t = (i < n ? trow[i] : 0) + sub; t < e; t += 8) {
            const int64_t j = tidx[t];
#pragma unroll
            for (int d = 0; d < DIM; ++d) s[d] += G[j * DIM + d];
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
            for (int d = 0; d < DIM; ++d) s[d] += __shfl_xor_sync(0xffffffffu, s[d], o);
        if (i < n && sub < DIM) {
            double v = s[0];
#pragma unroll
            for (int d = 1; d < DIM; ++d)
                if (sub == d) v = s[d];
            grad[i * DIM + sub] -= v;
        }
    }
}

int grid_for(int64_t items) {
    int64_t g = (items + 255) / 256, cap = (int64_t)num_sms() * 8;
    return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace

cudaError_t build_transpose(const int64_t* rowptr, const int32_t* cols, int64_t n, int64_t nnz, int32_t* cnt,
                            int64_t* trow, int64_t* fill, int32_t* tsrc_tmp, int64_t* tidx_tmp, int32_t* tsrc,
                            int64_t* tidx, int64_t* scan_tmp, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (n > 0 ? n : 1), s);
    if (e != cudaSuccess || n == 0) return e;
    if (nnz > 0) tcount_kernel<<<grid_for(nnz), 256, 0, s>>>(cols, nnz, cnt);
    e = exclusive_scan_i32(cnt, n, trow, scan_tmp, s);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyAsync(fill, trow, sizeof(int64_t) * n, cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return e;
    tfill_kernel<<<grid_for(n), 256, 0, s>>>(rowptr, cols, n, fill, tsrc_tmp, tidx_tmp);
    tsort_kernel<<<grid_for(n * 32), 256, 0, s>>>(trow, n, tsrc_tmp, tidx_tmp, tsrc, tidx);
    return cudaGetLastError();
}

cudaError_t row_sums(const int64_t* rowptr, int64_t n, int nout, const double* w64, const float* w32, int64_t ws,
                     double* rs, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    rowsum_kernel<<<grid_for(n), 256, 0, s>>>(rowptr, n, nout, w64, w32, ws, rs);
    return cudaGetLastError();
}

cudaError_t vjp_field(const int64_t* trow, const int32_t* tsrc, const int64_t* tidx, int64_t n, int nout,
                      const double* w64, const float* w32, int64_t ws, const double* rs, const double* g, double* out,
                      cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    vjp_field_kernel<<<grid_for(n), 256, 0, s>>>(trow, tsrc, tidx, n, nout, w64, w32, ws, rs, g, out);
    return cudaGetLastError();
}

cudaError_t vjp_field_sell(const VjpSellArgs& a, int nout, cudaStream_t s) {
    if (a.nwin == 0) return cudaSuccess;
    if (a.nwin > 0x7fffffff) return cudaErrorInvalidValue;
    const unsigned grid = (unsigned)a.nwin;
    switch (nout) {
#define DCPSE_VJPS_CASE(NO)                                       \
    case NO:                                                      \
        vjp_field_sell_kernel<NO><<<grid, 256, 0, s>>>(a);        \
        break;
        DCPSE_VJPS_CASE(1)
        DCPSE_VJPS_CASE(2)
        DCPSE_VJPS_CASE(3)
        DCPSE_VJPS_CASE(4)
        DCPSE_VJPS_CASE(5)
        DCPSE_VJPS_CASE(6)
        DCPSE_VJPS_CASE(7)
        DCPSE_VJPS_CASE(8)
#undef DCPSE_VJPS_CASE
        default:
            return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t transpose_outputs(const int64_t* tidx, int64_t nnz, int nout, const double* w64, const float* w32,
                              int64_t ws, double* wt, cudaStream_t s) {
    if (nnz == 0) return cudaSuccess;
    if (w64)
        transpose_outputs_kernel<double><<<grid_for(nnz), 256, 0, s>>>(tidx, nnz, nout, w64, ws, wt);
    else
        transpose_outputs_kernel<float><<<grid_for(nnz), 256, 0, s>>>(tidx, nnz, nout, w32, ws, wt);
    return cudaGetLastError();
}

cudaError_t vjp_gather(const int64_t* trow, const int64_t* tidx, int64_t n, int dim, const double* gentry,
                       double* grad, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const int grid = grid_for(n * 8);
    if (dim == 3)
        vjp_gather_kernel<3><<<grid, 256, 0, s>>>(trow, tidx, n, gentry, grad);
    else if (dim == 2)
        vjp_gather_kernel<2><<<grid, 256, 0, s>>>(trow, tidx, n, gentry, grad);
    else
        vjp_gather_kernel<1><<<grid, 256, 0, s>>>(trow, tidx, n, gentry, grad);
    return cudaGetLastError();
}

}  // namespace dcpse
