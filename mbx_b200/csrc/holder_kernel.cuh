// Evaluation kernels for the 2-body/3-body evaluators (one template for all
// types; the per-type pieces come from the generated traits T in gen/*.cuh).
//
// One n-mer per thread for the straight-line polynomials: the n-mer's atoms
// are gathered, moved to the image next to the n-mer's first monomer
// (GetCloseDimerImage / GetCloseTrimerImage), the polynomial variables are
// built in FP64, the polynomial and its gradient run out of registers (the
// generated Horner trie), then the switch, the chain rule to atoms (including
// the lone-pair redistribution), the virial and the gradient scatter follow.
// This is the work of x2b_v9x::eval / x3b_v2x::eval / the MB-nrg evaluators
// (potential/2b/x2b-v9x.cpp:1514-1819, potential/3b/x3b-v2x.cpp:1403-1808,
// x2b_A1B2Z2_C1D4_deg3_exp0_v1x.cpp:954, x2b_A1B4_A1B4_deg4_exp0_v1x.cpp:1600,
// mbnrg_3b_A1B4_C1D2_C1D2_deg3_v1.cpp:1481) fused with the gather, image and
// scatter steps of System::Get2B/Get3B (bblock/system.cpp:2425-2725,
// 2769-3073).
//
// The polynomial is that in the symmetry-adapted variables w
// (mbx_b200/codegen/wbasis.py): T::to_w takes the variables x to w, T::from_w
// the gradient back.  It has 3 to 8 times fewer terms (MB-pol 3b gradients of
// 132k trimers: 1.36 ms in x, 0.35 ms in w; the types that had no
// straight-line code ran from their term tables, 1 M NaCl 29 ms a step, now
// 1.05).
#pragma once
#include "holder_common.cuh"
#include "table_kernels.h"
#include "term_table.cuh"

// Precision / output modes.
enum { HM_ENERGY = 0, HM_GRAD_FP64 = 1 };

// Scratch of the mixed-precision evaluation (three kernels: variables, the
// polynomial on the tensor cores, chain rule), for up to cap n-mers: the shifted FP32
// variables and the trie's gradient, variable-major ([v * cap + t]), the
// polynomial's value and whether the n-mer is within the evaluator's cutoff.
struct PairScratch {
    float* dx;
    double* q;    // radial factor of each variable (var_exp_q), for the chain rule of pair_finish_kernel
    float* g;
    double* ep;
    unsigned char* live;
    long cap;
    int* err;   // status word: kernels that wait on barriers report a timeout here (bit 8)
};

struct HolderArgs {
    long n;                    // number of n-mers (capacity when n_dev is set)
    const int* n_dev;          // optional device-side count (read by the kernel, clamped to n)
    const int* status;         // optional: a nonzero word means the n-mer build failed; do nothing
    int* counter;              // work counter (zeroed before the launch): blocks claim units (LockPlan)
    int split;                 // system input, 1: the last round's chunks may be cut by trie pieces (sums in another order)
    const int4* nmers;         // system input: (m0, m1, m2, anchor slot), holder order
    const double* xyz;         // system input: site array (3 per site); AoS input: [n][NREAL*3]
    const int* first_index;    // system input: first site of every monomer
    BoxParams bp;
    double* grad;              // system: site-array gradient (+=); AoS: [n][NREAL*3] (+=)
    double* out;               // [0] energy, [1..6] virial xx xy xz yy yz zz (+=)
    double* e_per;             // optional: switched energy of every n-mer
    const double* coef;        // custom linear coefficients (global) or null
    int aos;                   // 1: AoS per-n-mer input (already imaged, no gather)
    // batched configurations (system input): per-configuration boxes and
    // energy + virial sums (8 doubles each), the configuration of every monomer
    const BoxParams* conf_bp;  // null: one configuration in bp
    const int* mon_conf;
    double* conf_out;
    // term table of the polynomial (term_table.cuh), for the table-driven kernels
    const int4* terms;         // (k, six (variable, exponent) byte pairs)
    const double* tcoef;       // term multiplicities
    long nterms;
    // code prefetch launch of a lockstep kernel (prime_passes > 0; see
    // prime_pieces): of the rest only out (null) is read
    int prime_passes, prime_npieces;
    PairScratch ps;            // mixed precision: scratch of the three kernels
};

__device__ __forceinline__ double ld_volatile(const double* p) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

// Real atoms of the evaluator's largest monomer (loop bound over one monomer's atoms).
template <class T>
__host__ __device__ constexpr int max_nat() {
    return T::NAT0 > T::NAT1 ? (T::NAT0 > T::NAT2 ? T::NAT0 : T::NAT2) : (T::NAT1 > T::NAT2 ? T::NAT1 : T::NAT2);
}

// GetCloseDimerImage / GetCloseTrimerImage: every monomer but the anchor slot
// moved to the image next to the anchor's first atom.
template <class T>
__device__ __forceinline__ void image_nmer(const BoxParams& bp, int anchor, double (&r)[T::NREAL][3]) {
    const int nat[3] = {T::NAT0, T::NAT1, T::NAT2};
    const int first[3] = {T::FIRST0, T::FIRST1, T::FIRST2};
    {
        double p0[3];
#pragma unroll
        for (int s = 0; s < T::NBODY; ++s)
            if (s == anchor) { p0[0] = r[first[s]][0]; p0[1] = r[first[s]][1]; p0[2] = r[first[s]][2]; }
#pragma unroll
        for (int s = 0; s < T::NBODY; ++s) {
            if (s == anchor) continue;
            double q0[3] = {r[first[s]][0], r[first[s]][1], r[first[s]][2]};
            double d[3];
            image_shift(bp, p0, q0, d);
#pragma unroll
            for (int a = 0; a < max_nat<T>(); ++a) {
                if (a < nat[s]) {
                    double q[3] = {r[first[s] + a][0], r[first[s] + a][1], r[first[s] + a][2]};
                    apply_shift(bp, d, q);
                    r[first[s] + a][0] = q[0];
                    r[first[s] + a][1] = q[1];
                    r[first[s] + a][2] = q[2];
                }
            }
        }
    }
}

template <class T, bool VOL>
__device__ __forceinline__ void load_nmer(const HolderArgs& A, long t, double (&r)[T::NREAL][3]) {
    constexpr int MAXNAT = max_nat<T>();
    if (A.aos) {
        const double* p = A.xyz + (size_t)t * (T::NREAL * 3);
#pragma unroll
        for (int i = 0; i < T::NREAL; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) r[i][c] = VOL ? ld_volatile(p + 3 * i + c) : __ldg(p + 3 * i + c);
        return;
    }
    const int4 nm = __ldg(A.nmers + t);
    const int mon[3] = {nm.x, nm.y, nm.z};
    const int nat[3] = {T::NAT0, T::NAT1, T::NAT2};
    const int first[3] = {T::FIRST0, T::FIRST1, T::FIRST2};
#pragma unroll
    for (int s = 0; s < T::NBODY; ++s) {
        const double* p = A.xyz + 3 * (size_t)__ldg(A.first_index + mon[s]);
#pragma unroll
        for (int a = 0; a < 3 * MAXNAT; ++a) {
            if (a < 3 * nat[s]) r[first[s] + a / 3][a % 3] = VOL ? ld_volatile(p + a) : __ldg(p + a);
        }
    }
    if (A.conf_bp) {
        const BoxParams& bp = A.conf_bp[__ldg(A.mon_conf + nm.x)];
        if (bp.use_pbc) image_nmer<T>(bp, nm.w, r);
    } else if (A.bp.use_pbc) {
        image_nmer<T>(A.bp, nm.w, r);
    }
}

// First-atom distances (pairs 01, 02, 12) and the skip rule of the type.
template <class T>
__device__ __forceinline__ bool pair_dists(const double (&r)[T::NREAL][3], double (&d)[3][3], double (&rr)[3]) {
    const int first[3] = {T::FIRST0, T::FIRST1, T::FIRST2};
    const int pa[3] = {0, 0, 1}, pb[3] = {1, 2, 2};
    constexpr int NP = T::NBODY == 2 ? 1 : 3;
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const int i = first[pa[p]], j = first[pb[p]];
        d[p][0] = r[i][0] - r[j][0];
        d[p][1] = r[i][1] - r[j][1];
        d[p][2] = r[i][2] - r[j][2];
        rr[p] = sqrt(d[p][0] * d[p][0] + d[p][1] * d[p][1] + d[p][2] * d[p][2]);
    }
    const double rf = T::RF;
    if (T::SKIP == 0) return rr[0] > rf;
    if (T::SKIP == 1)
        return (rr[0] > rf && rr[1] > rf) || (rr[0] > rf && rr[2] > rf) || (rr[1] > rf && rr[2] > rf);
    return rr[0] > rf && rr[1] > rf && rr[2] > rf;
}

// Switch value and the gradient of the switch with respect to first atoms,
// scaled by the unswitched energy ep, added into tg.
template <class T>
__device__ __forceinline__ double apply_switch(const double (&d)[3][3], const double (&rr)[3], double ep,
                                               double (&tg)[T::NREAL][3], bool grads) {
    const int first[3] = {T::FIRST0, T::FIRST1, T::FIRST2};
    if (!T::SWITCH_TRIPLE) {
        double gs;
        const double sw = f_switch(rr[0], T::RI, T::RF, gs);
        if (grads) {
            const double f = gs * ep / rr[0];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                tg[first[0]][c] += f * d[0][c];
                tg[first[1]][c] -= f * d[0][c];
            }
        }
        return sw;
    }
    // SWITCH_TRIPLE 1: s0 s1 + s0 s2 + s1 s2; 2: the same minus 2 s0 s1 s2;
    // 3: 1 - cos^2((S - 1) pi / 2) on S = s0 + s1 + s2, 0 below S = 1 and 1
    // above S = 2 (mbnrg_3b_A1B2C4_D1E2_D1E2_deg3_v1.cpp:2464-2471, gradient
    // -(pi / 2) sin(pi S) strictly inside (1, 2), :2563-2570)
    double g0, g1, g2;
    const double s0 = f_switch(rr[0], T::RI, T::RF, g0);
    const double s1 = f_switch(rr[1], T::RI, T::RF, g1);
    const double s2 = f_switch(rr[2], T::RI, T::RF, g2);
    if (T::SWITCH_TRIPLE == 3) {
        const double S = s0 + s1 + s2;
        if (grads && S > 1.0 && S < 2.0) {
            const double dS = -(M_PI / 2.0) * sin(M_PI * S) * ep;
            const double f0 = g0 * dS / rr[0], f1 = g1 * dS / rr[1], f2 = g2 * dS / rr[2];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                tg[first[0]][c] += f0 * d[0][c] + f1 * d[1][c];
                tg[first[1]][c] += f2 * d[2][c] - f0 * d[0][c];
                tg[first[2]][c] -= f1 * d[1][c] + f2 * d[2][c];
            }
        }
        if (S < 1.0) return 0.0;
        if (S > 2.0) return 1.0;
        const double cs = cos((S - 1.0) * M_PI / 2.0);
        return 1.0 - cs * cs;
    }
    const double c = T::SWITCH_TRIPLE == 2 ? 2.0 : 0.0;
    if (grads) {
        const double f0 = g0 * (s1 + s2 - c * s1 * s2) * ep / rr[0];
        const double f1 = g1 * (s0 + s2 - c * s0 * s2) * ep / rr[1];
        const double f2 = g2 * (s0 + s1 - c * s0 * s1) * ep / rr[2];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            tg[first[0]][c] += f0 * d[0][c] + f1 * d[1][c];
            tg[first[1]][c] += f2 * d[2][c] - f0 * d[0][c];
            tg[first[2]][c] -= f1 * d[1][c] + f2 * d[2][c];
        }
    }
    return s0 * s1 + s0 * s2 + s1 * s2 - c * s0 * s1 * s2;
}

// Adds v[0..7) into dst[0..7) (one configuration's energy and virial), one
// atomic per value for all lanes of the warp that are here with the same dst.
__device__ __forceinline__ void conf_accumulate(double* dst, const double (&v)[7]) {
    const int lane = threadIdx.x & 31;
    const unsigned act = __activemask();
    const unsigned peers = __match_any_sync(act, (unsigned long long)dst);
    const int leader = __ffs(peers) - 1;
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        double sum = 0.0;
        for (unsigned m = peers; m; m &= m - 1) sum += __shfl_sync(peers, v[i], __ffs(m) - 1);
        if (lane == leader && sum != 0.0) atomicAdd(dst + i, sum);
    }
}

// The chain rule, from what the kernel at hand holds: PairFactors or WColumns.
// dP/dv (FP32) and the radial factors (FP64) of n-mer t in the mixed path's
// scratch, read where the chain rule uses them
struct PairGrad {
    const float* __restrict__ g;
    long cap, t;
    __device__ __forceinline__ double operator[](int v) const { return (double)__ldg(g + v * cap + t); }
};
struct PairQ {
    const double* __restrict__ q;
    long cap, t;
    __device__ __forceinline__ double operator[](int v) const { return __ldcs(q + v * cap + t); }
};
struct PairFactors {
    PairGrad g;
    PairQ q;
};
template <class T>
__device__ __forceinline__ void chain_rule(const double (&s)[T::NSITES][3], const PairFactors& f,
                                           double (&sg)[T::NSITES][3]) {
    T::chain_q(s, f.g, f.q, sg);
}

// The w and dP/dw of the lockstep kernels, in shared-memory columns of stride S.
template <int S>
struct WColumns {
    const double* x;
    const double* g;
};
template <class T, int S>
__device__ __forceinline__ void chain_rule(const double (&s)[T::NSITES][3], const WColumns<S>& f,
                                           double (&sg)[T::NSITES][3]) {
    T::template chain_w<S>(s, f.x, f.g, sg);
}

// Everything after the polynomial: chain rule, switch, virial, scatter.  g:
// dP/dv as chain_rule takes it.  For system input ep and g may be a part of
// the n-mer's polynomial whose rest other threads add (LockPlan): all it
// writes are sums.
template <class T, class G>
__device__ __forceinline__ void finish_nmer(const HolderArgs& A, long t, double ep, const G& g, bool grads,
                                            double (&acc)[7]) {
    double r[T::NREAL][3];
    load_nmer<T, true>(A, t, r);
    double d[3][3], rr[3];
    pair_dists<T>(r, d, rr);
    double tg[T::NREAL][3];
    if (grads) {
        double s[T::NSITES][3], sg[T::NSITES][3];
        T::sites(r, s);
        chain_rule<T>(s, g, sg);
#pragma unroll
        for (int i = 0; i < T::NREAL; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) tg[i][c] = sg[i][c];
    }
    const double sw = apply_switch<T>(d, rr, ep, tg, false);
    double v[7] = {0, 0, 0, 0, 0, 0, 0};
    auto virial = [&]() {
#pragma unroll
        for (int i = 0; i < T::NREAL; ++i) {
            v[1] -= r[i][0] * tg[i][0];
            v[2] -= r[i][0] * tg[i][1];
            v[3] -= r[i][0] * tg[i][2];
            v[4] -= r[i][1] * tg[i][1];
            v[5] -= r[i][1] * tg[i][2];
            v[6] -= r[i][2] * tg[i][2];
        }
    };
    if (grads) {
        // VIRIAL_RAW: the evaluator's virial is that of the polynomial
        // gradient alone, before the switch (x2b_A1B2C4_D1E2_deg3_v1x.cpp:1353-1391)
        if (T::VIRIAL_RAW) virial();
#pragma unroll
        for (int i = 0; i < T::NREAL; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) tg[i][c] *= sw;
        apply_switch<T>(d, rr, ep, tg, true);
        if (!T::VIRIAL_RAW) virial();
    }
    const double es = sw * ep;
    if (A.e_per) A.e_per[t] = es;
    v[0] = es;
    if (A.conf_out) {
        conf_accumulate(A.conf_out + 8 * __ldg(A.mon_conf + __ldg(A.nmers + t).x), v);
    } else {
#pragma unroll
        for (int i = 0; i < 7; ++i) acc[i] += v[i];
    }
    if (!grads) return;
    if (A.aos) {
        double* p = A.grad + (size_t)t * (T::NREAL * 3);
#pragma unroll
        for (int i = 0; i < T::NREAL; ++i)
#pragma unroll
            for (int c = 0; c < 3; ++c) p[3 * i + c] += tg[i][c];
        return;
    }
    const int4 nm = __ldg(A.nmers + t);
    const int mon[3] = {nm.x, nm.y, nm.z};
    const int nat[3] = {T::NAT0, T::NAT1, T::NAT2};
    const int first[3] = {T::FIRST0, T::FIRST1, T::FIRST2};
#pragma unroll
    for (int s = 0; s < T::NBODY; ++s) {
        double* p = A.grad + 3 * (size_t)__ldg(A.first_index + mon[s]);
#pragma unroll
        for (int a = 0; a < max_nat<T>(); ++a)
            if (a < nat[s])
#pragma unroll
                for (int c = 0; c < 3; ++c) atomicAdd(p + 3 * a + c, tg[first[s] + a][c]);
    }
}

// Number of n-mers to evaluate (0 when the n-mer build reported a failure).
__device__ __forceinline__ long nmer_count(const HolderArgs& A) {
    if (A.status && *A.status) return 0;
    if (!A.n_dev) return A.n;
    const long c = *A.n_dev;
    return c < A.n ? c : A.n;
}

// Dynamic shared memory of the lockstep kernels (their x/g columns).
extern __shared__ __align__(16) unsigned char mbx_dyn_smem[];

// Code prefetch mode of the lockstep kernels.  Once other work has evicted a
// trie's code from L2 (the rest of an MD step between two force calls), the
// first pass of each SM through it waits on DRAM for every instruction fetch.
// An SM only gains from code that SMs of its own half of the chip have
// fetched.  A prefetch launch of the same kernel (ptxas compiles a
// __noinline__ piece separately for every kernel that calls it, so only the
// kernel's own launch fetches the code the evaluation runs) has one warp per
// block run piece (block + j * grid) mod npieces in pass j: every piece
// fetched by several SMs spread over the chip, all pieces at once.  It is
// launched beside the n-mer search, ahead of the evaluation.  The lanes' x and
// g columns share one [v][L] array (x at columns 0-31, g at 32-63) of zeros;
// the results are discarded.
template <int L, class V, class Piece>
__device__ __forceinline__ void prime_pieces(const HolderArgs& A, int nvars, Piece&& piece) {
    static_assert(L >= 64, "x and g columns of the prefetch overlap");
    V* xs = reinterpret_cast<V*>(mbx_dyn_smem) + threadIdx.x;
    V* gs = xs + 32;
#pragma unroll 1
    for (int v = 0; v < nvars; ++v) {
        xs[v * L] = V(0);
        gs[v * L] = V(0);
    }
    __syncwarp();
    double sum = 0.0;
#pragma unroll 1
    for (int j = 0; j < A.prime_passes; ++j) {
        const int k = (int)(((long)blockIdx.x + (long)j * gridDim.x) % A.prime_npieces);
        sum += piece(k, xs, gs);
        __syncwarp();
    }
    if (A.out) A.out[threadIdx.x] = sum;   // null in a prefetch launch; keeps the calls
}

// The work of a lockstep grid of nslot blocks over nchunk chunks of n-mers
// and npiece pieces of the trie: whole chunks in full rounds, then the chunks
// of the last, partial round cut by pieces, so that the blocks that would
// otherwise be idle take a share of the polynomial each (value and gradient
// are sums over the pieces; every share ends with its own chain rule, switch
// and scatter).
struct LockPlan {
    long whole, units;
    int parts;
    __device__ __forceinline__ LockPlan(long nchunk, long nslot, int npiece, bool split) {
        whole = split ? nchunk / nslot * nslot : nchunk;
        const long rest = nchunk - whole;
        parts = rest > 0 ? (int)(nslot / rest < npiece ? nslot / rest : npiece) : 1;
        units = whole + rest * parts;
    }
    // chunk and pieces [k0, k1) of unit u
    __device__ __forceinline__ long unit(long u, int npiece, int& k0, int& k1) const {
        if (u < whole) {
            k0 = 0;
            k1 = npiece;
            return u;
        }
        const long v = u - whole;
        const int p = (int)(v % parts);
        k0 = p * npiece / parts;
        k1 = (p + 1) * npiece / parts;
        return whole + v / parts;
    }
};

// One n-mer per thread, all warps of a block in lockstep through the trie:
// the straight-line polynomial is thousands of instructions, more than the
// instruction cache holds, so the block's warps go through it piece by piece
// together (a barrier after each piece) and one fetch of a piece's code serves
// all of them.  Threads without an n-mer (past the end, or beyond the
// evaluator's cutoff) run the pieces on zero variables and discard the result;
// warps of such threads only keep the barriers.  Persistent grid; a block
// claims units (LockPlan) from A.counter (or strides statically without it).
template <class T, class CC, int MODE>
__global__ void __launch_bounds__(T::LOCK_THREADS, 1) holder_lock_kernel(const HolderArgs A) {
    constexpr bool grads = (MODE == HM_GRAD_FP64);
    constexpr int L = T::LOCK_THREADS;   // == blockDim.x
    constexpr int NP = grads ? T::NPIECES : T::NPIECES_E;
    double* xs = reinterpret_cast<double*>(mbx_dyn_smem) + threadIdx.x;
    double* gs = xs + T::NVARS * L;      // used in gradient mode only
    __shared__ long s_unit;
    const auto piece = [&](int k, const double* x, double* g) -> double {
        if constexpr (MODE == HM_ENERGY) return T::template pip_e_piece<L>(k, CC{}, x);
        else return T::template pip_piece<L>(k, CC{}, x, g);
    };
    if (A.prime_passes > 0) {
        prime_pieces<L, double>(A, T::NVARS, piece);
        return;
    }
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    const long n = nmer_count(A);
    const LockPlan plan((n + L - 1) / L, gridDim.x, NP, A.split != 0);
    long u = blockIdx.x;
    for (;;) {
        if (A.counter) {
            if (threadIdx.x == 0) s_unit = atomicAdd(A.counter, 1);
            __syncthreads();
            u = s_unit;
            __syncthreads();
        }
        if (u >= plan.units) break;
        int k0, k1;
        const long t = plan.unit(u, NP, k0, k1) * L + threadIdx.x;
        bool live = t < n;
        {
            double x[T::NVARS];
#pragma unroll
            for (int v = 0; v < T::NVARS; ++v) x[v] = 0.0;
            if (live) {
                double r[T::NREAL][3];
                load_nmer<T, false>(A, t, r);
                double d[3][3], rr[3];
                if (pair_dists<T>(r, d, rr)) {
                    if (A.e_per) A.e_per[t] = 0.0;
                    live = false;
                } else {
                    double s[T::NSITES][3];
                    T::sites(r, s);
                    T::vars(s, x);
                    T::to_w(x);
                }
            }
#pragma unroll
            for (int v = 0; v < T::NVARS; ++v) {
                xs[v * L] = x[v];
                if (grads) gs[v * L] = 0.0;
            }
        }
        const bool busy = __any_sync(0xffffffffu, live);
        double ep = 0.0;
#pragma unroll 1
        for (int k = k0; k < k1; ++k) {
            if (busy) ep += piece(k, xs, gs);
            __syncthreads();
        }
        if (live) finish_nmer<T>(A, t, ep, WColumns<L>{xs, gs}, grads, acc);
        u += gridDim.x;
    }
    block_reduce_add<7>(acc, A.out);
}

// Variables of n-mer t shifted to the type's FP32 basis, dx = x - x0 rounded
// to FP32 (x itself is built in FP64).  Returns false, with x = 0, for t >= n
// or an n-mer beyond the evaluator's cutoff.
template <class T>
__device__ __forceinline__ bool nmer_vars_f32(const HolderArgs& A, long t, long n, float (&xf)[T::NVARS],
                                              double* q = nullptr) {
    double x[T::NVARS];
#pragma unroll
    for (int v = 0; v < T::NVARS; ++v) x[v] = 0.0;
    bool live = t < n;
    if (live) {
        double r[T::NREAL][3];
        load_nmer<T, false>(A, t, r);
        double d[3][3], rr[3];
        if (pair_dists<T>(r, d, rr)) {
            if (A.e_per) A.e_per[t] = 0.0;
            live = false;
        } else {
            double s[T::NSITES][3];
            T::sites(r, s);
            if (q) {
                // with the radial factors, stored for pair_finish_kernel as
                // they are computed (streaming stores: read once, by that
                // kernel, they should not push other data out of L2)
                struct {
                    double* p;
                    long cap, t;
                    __device__ __forceinline__ void put(int v, double f) { __stcs(p + v * cap + t, f); }
                } qw{q, A.ps.cap, t};
                T::vars_q(s, x, qw);
            } else {
                T::vars(s, x);
            }
        }
    }
    T::shift(x, xf);
    return live;
}

// Mixed-precision evaluation in three kernels.  The FP64 work around the
// polynomial (gather, image, variables; later the switch, chain rule, virial
// and scatter) is latency-bound and needs many warps, the tensor-core kernel
// takes whole SMs:
//   pair_vars_kernel    one n-mer per thread at full occupancy: the FP64
//                       variables, shifted to the FP32 basis, into A.ps.dx
//   qf_eval_kernel      the polynomial (qf_kernel.cuh), dx in, gradient and
//                       value out
//   pair_finish_kernel  one n-mer per thread at full occupancy: switch,
//                       chain rule (FP64), virial, scatter, energy sums
// The variables, switch, chain rule and sums stay FP64.
template <class T>
__global__ void __launch_bounds__(256, 2) pair_vars_kernel(const HolderArgs A) {
    const long n = nmer_count(A);
    const long cap = A.ps.cap;
    for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
        float xf[T::NVARS];
        const bool live = nmer_vars_f32<T>(A, t, n, xf, A.ps.q);
#pragma unroll
        for (int v = 0; v < T::NVARS; ++v) {
            A.ps.dx[v * cap + t] = xf[v];
            A.ps.g[v * cap + t] = 0.0f;   // the tensor-core kernel adds into g and ep
        }
        A.ps.ep[t] = 0.0;
        A.ps.live[t] = live ? 1 : 0;
    }
}

template <class T>
__global__ void __launch_bounds__(128, 3) pair_finish_kernel(const HolderArgs A) {
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    const long n = nmer_count(A);
    const long cap = A.ps.cap;
    for (long t = blockIdx.x * (long)blockDim.x + threadIdx.x; t < n; t += (long)gridDim.x * blockDim.x) {
        if (!A.ps.live[t]) continue;
        // the chain rule from the radial factors pair_vars_kernel stored: no
        // square root, exponential or division per variable here
        finish_nmer<T>(A, t, A.ps.ep[t], PairFactors{{A.ps.g, cap, t}, {A.ps.q, cap, t}}, true, acc);
    }
    block_reduce_add<7>(acc, A.out);
}

// 1-body MB-nrg evaluation (x1b_*::eval, e.g. x1b_A1B4_v1x::eval,
// potential/1b/x1b_A1B4_deg5_exp0_v1x.cpp:361-419): no image, no switch, no
// cutoff.  A lane per monomer, the warp walking the term table in step, every lane
// applying each term to its own monomer, whose variables and gradient
// accumulators sit in shared-memory columns [v][lane]; variables, chain rule
// and the virial -sum r (x) g over the monomer's atoms as the reference's
// evaluator does.
// A.first_index: first site of each monomer to evaluate (A.n of them); one
// thread per monomer writes its gradient, so no atomics.  Dynamic shared
// memory: 4 warps x 2 x NVARS x 32 doubles.
template <class T>
__global__ void __launch_bounds__(128) onebody_table_kernel(const HolderArgs A) {
    static_assert(T::NBODY == 1, "1-body evaluators only");
    double* xc = reinterpret_cast<double*>(mbx_dyn_smem) + ((threadIdx.x >> 5) * 2 * T::NVARS) * 32 +
                 (threadIdx.x & 31);
    double* gc = xc + T::NVARS * 32;
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    const bool grads = A.grad != nullptr;
    for (long base = blockIdx.x * (long)blockDim.x; base < A.n; base += (long)gridDim.x * blockDim.x) {
        const long t = base + threadIdx.x;
        const bool live = t < A.n;
        double r[T::NREAL][3];
        double s[T::NSITES][3];
        {
            double x[T::NVARS];
#pragma unroll
            for (int v = 0; v < T::NVARS; ++v) x[v] = 0.0;
            if (live) {
                const double* p = A.xyz + 3 * (size_t)__ldg(A.first_index + t);
#pragma unroll
                for (int i = 0; i < T::NREAL; ++i)
#pragma unroll
                    for (int c = 0; c < 3; ++c) r[i][c] = p[3 * i + c];
                T::sites(r, s);
                T::vars(s, x);
                T::to_w(x);
            }
#pragma unroll
            for (int v = 0; v < T::NVARS; ++v) {
                xc[v * 32] = x[v];
                gc[v * 32] = 0.0;
            }
        }
        __syncwarp();
        double e = 0.0;
        if (__any_sync(0xffffffffu, live)) {
            const auto xv = [&](int v) { return xc[v * 32]; };
            for (long q = 0; q < A.nterms; ++q) {
                const int4 tm = __ldg(A.terms + q);
                const double c = __ldg(A.coef + tm.x) * __ldg(A.tcoef + q);
                if (grads)
                    e += term_value_grad<T::TPAIRS>(tm, c, xv, [&](int v, double dv) { gc[v * 32] += dv; });
                else
                    e += term_value<T::TPAIRS>(tm, c, xv);
            }
        }
        __syncwarp();
        if (live) {
            acc[0] += e;
            if (grads) {
                double g[T::NVARS];
#pragma unroll
                for (int v = 0; v < T::NVARS; ++v) g[v] = gc[v * 32];
                T::from_w(g);
                double sg[T::NSITES][3];
                T::chain(s, g, sg);
                const int ia[6] = {0, 0, 0, 1, 1, 2}, ib[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
                for (int k = 0; k < 6; ++k) {
                    double v = 0.0;
#pragma unroll
                    for (int i = 0; i < T::NREAL; ++i) v -= r[i][ia[k]] * sg[i][ib[k]];
                    acc[1 + k] += v;
                }
                double* q = A.grad + 3 * (size_t)__ldg(A.first_index + t);
#pragma unroll
                for (int i = 0; i < T::NREAL; ++i)
#pragma unroll
                    for (int c = 0; c < 3; ++c) q[3 * i + c] += sg[i][c];
            }
        }
        __syncwarp();
    }
    block_reduce_add<7>(acc, A.out);
}

// The variables of an n-mer of AoS input in w and its weight times the switch
// (0 beyond the evaluator's cutoff) for the coefficient adjoint.  An n-mer
// without weight has zeros, so that it adds nothing whatever its coordinates
// (padding with coincident atoms has infinite variables).
template <class T>
__device__ __forceinline__ double adjoint_vars(const HolderArgs& A, const double* __restrict__ w, long t,
                                               double (&x)[T::NVARS]) {
    double scale = 0.0;
    double r[T::NREAL][3];
    load_nmer<T, false>(A, t, r);
    double d[3][3], rr[3];
    if (!pair_dists<T>(r, d, rr)) {
        double tg[T::NREAL][3];
        scale = apply_switch<T>(d, rr, 0.0, tg, false) * (w ? w[t] : 1.0);
    }
    if (scale != 0.0) {
        double s[T::NSITES][3];
        T::sites(r, s);
        T::vars(s, x);
        T::to_w(x);
    } else {
#pragma unroll
        for (int v = 0; v < T::NVARS; ++v) x[v] = 0.0;
    }
    return scale;
}

// First step of the coefficient adjoint (coef_adjoint_kernel has the second):
// the w variables of n-mers first .. first + count and, as row NVARS, their
// weight times the switch, variable-major in wv with stride count.  One n-mer
// per thread.
template <class T>
__global__ void __launch_bounds__(128) holder_wvars_kernel(const HolderArgs A, const double* __restrict__ w,
                                                           long first, int count, double* __restrict__ wv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    double x[T::NVARS];
    const double scale = adjoint_vars<T>(A, w, first + i, x);
#pragma unroll
    for (int v = 0; v < T::NVARS; ++v) wv[(size_t)v * count + i] = x[v];
    wv[(size_t)T::NVARS * count + i] = scale;
}

// The whole coefficient adjoint of a polynomial of at most MBX_SMALL_TERMS
// terms: an n-mer per thread, every term's sum over a warp by shuffles, over a
// block's warps and n-mers in shared memory, over the blocks by the block that
// finishes last, always in the same order.  part: MBX_SMALL_TERMS doubles a
// block; ticket: 0 before and after.  Bound by the launch and, above some 10^5
// n-mers, by the shuffles.  A call for the 9 terms of Na-Na: 23, 31 and 36 us
// for 1, 30,000 and 150,000 dimers, 33, 74 and 306 through the tiles of
// coef_adjoint_kernel and its four other launches.  The line lies between the
// library's 23 terms (He-He: 34 us for 30,000, 75) and 62 (CS-H2: 49 us through
// the tiles; walking as many terms took 65).
template <class T>
__global__ void __launch_bounds__(128) holder_dcoef_small_kernel(const HolderArgs A, const double* __restrict__ w,
                                                                 const AdjointTable P, double* part, unsigned* ticket,
                                                                 double* out) {
    __shared__ double xs[4][T::NVARS][32], sum[4][MBX_SMALL_TERMS];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    sum[warp][lane] = 0.0;
    for (long base = blockIdx.x * (long)blockDim.x; base < A.n; base += (long)gridDim.x * blockDim.x) {
        const long t = base + threadIdx.x;
        double x[T::NVARS], scale = 0.0;
#pragma unroll
        for (int v = 0; v < T::NVARS; ++v) x[v] = 0.0;
        if (t < A.n) scale = adjoint_vars<T>(A, w, t, x);
#pragma unroll
        for (int v = 0; v < T::NVARS; ++v) xs[warp][v][lane] = x[v];
        __syncwarp();
        const auto xv = [&](int v) { return xs[warp][v][lane]; };
        for (int q = 0; q < P.nterms; ++q) {
            double v = term_value<T::TPAIRS>(__ldg(P.terms + q), scale, xv);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane == 0) sum[warp][q] += v;
        }
        __syncwarp();
    }
    __syncthreads();
    if (warp == 0) {
        part[blockIdx.x * MBX_SMALL_TERMS + lane] = sum[0][lane] + sum[1][lane] + sum[2][lane] + sum[3][lane];
        __threadfence();
        __syncwarp();
        if (lane == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double v = 0.0;
    for (int b = warp; b < gridDim.x; b += 4) v += __ldcg(part + b * MBX_SMALL_TERMS + lane);
    sum[warp][lane] = v;
    __syncthreads();
    if (warp == 0) sum[0][lane] += sum[1][lane] + sum[2][lane] + sum[3][lane];
    __syncthreads();
    // dE/dc of every w coefficient, then F^T of those
    double* dc = sum[1];
    for (int j = threadIdx.x; j < P.ncw; j += blockDim.x) {
        double d = 0.0;
        for (int q = P.first[j]; q < P.first[j + 1]; ++q) d = fma(P.tcoef[q], sum[0][q], d);
        dc[j] = d;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < P.ncoef; k += blockDim.x) {
        double d = 0.0;
        for (int q = P.ftrow[k]; q < P.ftrow[k + 1]; ++q) d = fma(P.ftf[q], dc[P.ftk[q]], d);
        out[k] += d;
    }
    if (threadIdx.x == 0) *ticket = 0;
}
