// The generated-polynomial calling convention over a term table: energies and
// gradients of a polynomial at caller-supplied variables.
//
// This is the convention of the reference's generated programs
// (poly_2b_v6x::eval(nd, a, x, t, g), potential/2b/poly-2b-v6x.h:95, with
// x[v * nd + i]; the per-configuration MB-nrg eval(a, x, g) programs are the
// nd = 1 case), served for every evaluator from its term table in the w
// variables (term_table.cuh) and the coefficients currently set on the
// device: x is transformed to w, the gradient back.  A warp per
// configuration: lane l takes terms l, l+32, ...; the configuration's variables and gradient accumulators sit in shared
// memory (gradient by shared-memory atomics), the energy is reduced across
// the warp.
#include <cuda_runtime.h>

#include "launch_cache.cuh"
#include "table_kernels.h"
#include "term_table.cuh"

#define MBX_POLY_WARPS 4
#define MBX_POLY_MAXV 128

namespace {

// out[v] = sum over row v of +-in[column], less base[v] where given; lanes
// over the rows
__device__ __forceinline__ void signed_rows(const int* __restrict__ row, const int* __restrict__ col,
                                            const double* __restrict__ base, int nvars, const double* in, double* out,
                                            size_t stride) {
    for (int v = threadIdx.x & 31; v < nvars; v += 32) {
        double s = base ? -base[v] : 0.0;
        for (int q = row[v]; q < row[v + 1]; ++q) {
            const int c = col[q];
            s += c > 0 ? in[c - 1] : -in[-c - 1];
        }
        out[v * stride] = s;
    }
}

}  // namespace

template <int NP>
__global__ void __launch_bounds__(MBX_POLY_WARPS * 32)
    poly_table_kernel(long nd, int nvars, const double* __restrict__ x_soa, double* __restrict__ g_soa,
                      double* __restrict__ e, const PolyTable P) {
    __shared__ double xs[MBX_POLY_WARPS][MBX_POLY_MAXV];
    __shared__ double gs[MBX_POLY_WARPS][MBX_POLY_MAXV];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long stride = (long)gridDim.x * MBX_POLY_WARPS;
    for (long i = blockIdx.x * (long)MBX_POLY_WARPS + w; i < nd; i += stride) {
        // x in gs for the transform, w in xs
        for (int v = lane; v < nvars; v += 32) gs[w][v] = x_soa[(long)v * nd + i];
        __syncwarp();
        signed_rows(P.wrow, P.w, P.w0, nvars, gs[w], xs[w], 1);
        __syncwarp();
        for (int v = lane; v < nvars; v += 32) gs[w][v] = 0.0;
        __syncwarp();
        const auto xv = [&](int v) { return xs[w][v]; };
        double en = 0.0;
        for (long q = lane; q < P.nterms; q += 32) {
            const int4 tm = __ldg(P.terms + q);
            const double c = __ldg(P.coef + tm.x) * __ldg(P.tcoef + q);
            if (g_soa)
                en += term_value_grad<NP>(tm, c, xv, [&](int v, double dv) { atomicAdd(&gs[w][v], dv); });
            else
                en += term_value<NP>(tm, c, xv);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) en += __shfl_xor_sync(0xffffffffu, en, o);
        __syncwarp();
        if (lane == 0) e[i] = en;
        if (g_soa) signed_rows(P.wtrow, P.wt, nullptr, nvars, gs[w], g_soa + i, (size_t)nd);
        __syncwarp();
    }
}

int mbx_launch_poly_table(long nd, int nvars, const double* x, double* g, double* e, const PolyTable& P, int sms,
                          cudaStream_t s) {
    if (nvars < 1 || nvars > MBX_POLY_MAXV || P.pairs < 1 || P.pairs > MBX_TERM_PAIRS) return (int)cudaErrorInvalidValue;
    const long want = (nd + MBX_POLY_WARPS - 1) / MBX_POLY_WARPS;
    const int grid = (int)(want < (long)sms * 8 ? (want > 0 ? want : 1) : (long)sms * 8);
    if (P.pairs <= 4)
        poly_table_kernel<4><<<grid, MBX_POLY_WARPS * 32, 0, s>>>(nd, nvars, x, g, e, P);
    else
        poly_table_kernel<MBX_TERM_PAIRS><<<grid, MBX_POLY_WARPS * 32, 0, s>>>(nd, nvars, x, g, e, P);
    return (int)cudaGetLastError();
}

// Coefficient adjoint: out[k] += sum over n-mers of scale * dP/da_k (adjoint
// of E = sum_n scale_n P(c, w_n), c = F a, for refitting).
//
// Every term is the product of two half-monomials z (WTable.halves).  A block
// takes a share of the n-mers, MBX_ADJ_N at a time: their z, and scale * z,
// go to shared memory once; then every thread multiplies the pairs of its own
// MBX_ADJ_Q terms, and keeps one sum per term in registers over all of the
// block's n-mers, so that nothing is reduced across threads.  The blocks' sums
// are added up in a fixed order (adjoint_terms_kernel), then the terms of
// every coefficient (adjoint_coef_kernel) and F^T of those
// (adjoint_out_kernel): the result is the same from call to call.  Bound by
// the shared-memory reads of two doubles per term and n-mer, the second
// scattered, the first mostly the same for a warp's lanes: 20000 MB-pol 3b
// trimers (7425 terms) 163 us, where walking the 33525 terms in x, a lane per
// n-mer, took 14 ms.  Warps past the last term skip the products: a call for
// 30000 dimers of 2226 terms (MB-pol 2b) takes 107 us, 122 with them; of 429
// (Li-H2O) 57 and 83.
#define MBX_ADJ_THREADS 512
#define MBX_ADJ_N 8
#define MBX_ADJ_Q 8

extern __shared__ __align__(16) double mbx_adj_smem[];

__global__ void __launch_bounds__(MBX_ADJ_THREADS)
    coef_adjoint_kernel(const double* __restrict__ wv, int count, const AdjointTable P, double* __restrict__ part) {
    constexpr int N = MBX_ADJ_N, LD = N + 1;   // odd row length: the rows of a warp's lanes spread over the banks
    double* ws = mbx_adj_smem;                 // [nvars + 1][N], the last row the scales
    double* z = ws + (P.nvars + 1) * N;        // [nhalf][LD]
    double* zs = z + P.nhalf * LD;             // scale * z
    const int t0 = blockIdx.y * (MBX_ADJ_THREADS * MBX_ADJ_Q) + threadIdx.x;
    unsigned pair[MBX_ADJ_Q];
    double acc[MBX_ADJ_Q];
#pragma unroll
    for (int q = 0; q < MBX_ADJ_Q; ++q) {
        const int t = t0 + q * MBX_ADJ_THREADS;
        pair[q] = t < P.nterms ? P.pair[t] : 0u;
        acc[q] = 0.0;
    }
    for (int base = blockIdx.x * N; base < count; base += gridDim.x * N) {
        for (int i = threadIdx.x; i < (P.nvars + 1) * N; i += MBX_ADJ_THREADS) {
            const int n = base + i % N;
            ws[i] = n < count ? wv[(size_t)(i / N) * count + n] : 0.0;   // (scale 0 past the end)
        }
        __syncthreads();
        for (int i = threadIdx.x; i < P.nhalf * N; i += MBX_ADJ_THREADS) {
            const int n = i % N, h = i / N;
            const int2 f = P.half[h];
            double m = 1.0;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const int e = (f.y >> (8 * j)) & 255;
                if (e == 0) break;
                const double x = ws[((f.x >> (8 * j)) & 255) * N + n];
                m *= x;
                for (int p = 1; p < e; ++p) m *= x;
            }
            z[h * LD + n] = m;
            zs[h * LD + n] = m * ws[P.nvars * N + n];
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < MBX_ADJ_Q; ++q) {
            if (t0 + q * MBX_ADJ_THREADS >= P.nterms) break;
            const double* a = zs + (pair[q] & 0xffff) * LD;
            const double* b = z + (pair[q] >> 16) * LD;
#pragma unroll
            for (int n = 0; n < N; ++n) acc[q] = fma(a[n], b[n], acc[q]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < MBX_ADJ_Q; ++q) {
        const int t = t0 + q * MBX_ADJ_THREADS;
        if (t < P.nterms) part[(size_t)blockIdx.x * P.nterms + P.term[t]] = acc[q];
    }
}

// sum[t] = sum over blocks of part[block][t]: 32 terms a block, 8 strands of
// blocks each, joined in order.
__global__ void __launch_bounds__(256) adjoint_terms_kernel(const double* __restrict__ part, int nblock, int nterms,
                                                            double* __restrict__ sum) {
    __shared__ double s[8][32];
    const int t = blockIdx.x * 32 + threadIdx.x;
    double v = 0.0;
    if (t < nterms)
        for (int b = threadIdx.y; b < nblock; b += 8) v += part[(size_t)b * nterms + t];
    s[threadIdx.y][threadIdx.x] = v;
    __syncthreads();
    if (threadIdx.y == 0 && t < nterms) {
        for (int j = 1; j < 8; ++j) v += s[j][threadIdx.x];
        sum[t] = v;
    }
}

// dc[j] = signed sum over the terms of coefficient j.
__global__ void __launch_bounds__(128) adjoint_coef_kernel(const AdjointTable P, const double* __restrict__ sum,
                                                           double* __restrict__ dc) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= P.ncw) return;
    double v = 0.0;
    for (int t = P.first[j]; t < P.first[j + 1]; ++t) v = fma(P.tcoef[t], sum[t], v);
    dc[j] = v;
}

// out += F^T dc; a warp per fitted coefficient.
__global__ void __launch_bounds__(128) adjoint_out_kernel(const AdjointTable P, const double* __restrict__ dc,
                                                          double* __restrict__ out) {
    const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (k >= P.ncoef) return;
    double v = 0.0;
    for (int q = P.ftrow[k] + lane; q < P.ftrow[k + 1]; q += 32) v = fma(P.ftf[q], dc[P.ftk[q]], v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) out[k] += v;
}

namespace {
// term ranges (grid y) and most blocks over the n-mers (grid x): two blocks an SM
int adjoint_ranges(const AdjointTable& P) {
    return (P.nterms + MBX_ADJ_THREADS * MBX_ADJ_Q - 1) / (MBX_ADJ_THREADS * MBX_ADJ_Q);
}
}  // namespace

int mbx_coef_adjoint_blocks(const AdjointTable& P, int sms) {
    const int ny = adjoint_ranges(P);
    return (2 * sms + ny - 1) / ny;
}

int mbx_launch_coef_adjoint(const double* wv, int count, const AdjointTable& P, double* work, double* out, int sms,
                            cudaStream_t s) {
    const size_t smem = ((size_t)(P.nvars + 1) * MBX_ADJ_N + 2 * (size_t)P.nhalf * (MBX_ADJ_N + 1)) * sizeof(double);
    const int want = (count + MBX_ADJ_N - 1) / MBX_ADJ_N, most = mbx_coef_adjoint_blocks(P, sms);
    const int nx = want < most ? (want > 0 ? want : 1) : most;
    double* sum = work + (size_t)most * P.nterms;
    const int r = launch_any_smem<coef_adjoint_kernel>(dim3(nx, adjoint_ranges(P)), MBX_ADJ_THREADS, smem, s, wv, count, P,
                                                       work);
    if (r) return r;
    adjoint_terms_kernel<<<(P.nterms + 31) / 32, dim3(32, 8), 0, s>>>(work, nx, P.nterms, sum);
    double* dc = sum + P.nterms;
    adjoint_coef_kernel<<<(P.ncw + 127) / 128, 128, 0, s>>>(P, sum, dc);
    adjoint_out_kernel<<<(P.ncoef + 3) / 4, 128, 0, s>>>(P, dc, out);
    return (int)cudaGetLastError();
}
