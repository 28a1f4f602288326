// nnls_warp.cuh -- warp-cooperative Lawson-Hanson NNLS in FP64 (one voxel per warp).
//
// Restates src/NNLS.jl (unsafe_nnls! at 605-825 and its Tikhonov form at
// 827-1061) and the NNLSProblem warm start of src/lsqnonneg.jl:30-164.
//
// GB300 mapping (all control flow is warp-uniform; every lane holds the same
// scalars):
//   * the working matrix lives in shared memory, column-major with an odd
//     leading dimension so both row-parallel and column-parallel accesses are
//     free of bank conflicts;
//   * the reference's physical column swaps are replaced by the idx
//     permutation itself: logical column j lives in physical column
//     idx[j]-1, which is exactly where the reference's swaps would have moved
//     its data, so adds and deletes move no matrix data;
//   * Householder application and dual updates run lanes-over-columns, each
//     lane accumulating its column sequentially in the reference's row order
//     (so those dot products are bitwise the reference's);
//   * Householder construction, the warm-start scalars and residual norms run
//     lanes-over-rows with butterfly reductions (reassociated sums, like the
//     reference's @simd loops).
// Every loop is bounded; the NNLS iteration cap is the reference's 3n.
//
// Only the sequential column loops are unrolled (8 rows: their loads overlap);
// the lane-strided ones run one to three times and stay rolled, or the solver
// would be 107 KB of code waiting for instruction fetch instead of 65: 32x32x4
// voxels x 32 echoes, chi2, 18.5 -> 17.4 ms (17.7 with 2 rows, 17.4 with 4),
// 120x120x1 x 48 echoes, L-curve, 128.2 -> 125.2 ms (128.6, 126.4).
#pragma once
#include <cuda_runtime.h>
#include <math_constants.h>

namespace dk {

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(FULL, v, o));
    return v;
}
__device__ __forceinline__ double bcast(double v, int src) { return __shfl_sync(FULL, v, src); }
__device__ __forceinline__ int bcasti(int v, int src) { return __shfl_sync(FULL, v, src); }

// Julia's Base.max / Base.min for Float64 (NaN-propagating, -0.0 < 0.0),
// decided on the integer pipes: tkey orders non-NaN doubles as their values
// with -0.0 below +0.0, which is the order signbit(x - y) gives (x - y is -0.0
// only for x = -0.0, y = +0.0; for equal values, infinities included, x is
// kept).
__device__ __forceinline__ long long tkey(double d) {
    const long long b = __double_as_longlong(d);
    return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}
__device__ __forceinline__ bool isnan_bits(double d);
__device__ __forceinline__ double jmax(double x, double y) {
    if (isnan_bits(x) || isnan_bits(y)) return CUDART_NAN;
    return tkey(x) < tkey(y) ? y : x;
}
__device__ __forceinline__ double jmin(double x, double y) {
    if (isnan_bits(x) || isnan_bits(y)) return CUDART_NAN;
    return tkey(x) < tkey(y) ? x : y;
}

// Order-preserving integer image of a double for comparisons on the integer
// pipes (the FP64 pipe is the kernel's bottleneck): for non-NaN a, b,
// okey(a) < okey(b) iff a < b, with -0.0 and +0.0 mapped to the same key.
__device__ __forceinline__ long long okey(double d) {
    long long b = __double_as_longlong(d);
    if ((b << 1) == 0) return 0;
    return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}
__device__ __forceinline__ bool isnan_bits(double d) {
    return (__double_as_longlong(d) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}
// d > 0 on the integer pipes (false for zeros and NaN).
__device__ __forceinline__ bool pos_bits(double d) {
    const long long b = __double_as_longlong(d);
    return b > 0 && b <= 0x7ff0000000000000LL;
}
// d <= 0 on the integer pipes (true for zeros, false for NaN).
__device__ __forceinline__ bool nonpos_bits(double d) {
    const long long b = __double_as_longlong(d);
    return !isnan_bits(d) && (b <= 0);
}
// d > t for a threshold t with its sign bit clear (+0.0 or positive) or NaN,
// on the integer pipes: such doubles order like their bit patterns; negative d
// and NaN d give false, and so does every d against a NaN threshold, as the
// FP64 comparison does.  (t = -0.0 is not covered: +0.0 would compare above
// it.  The solver's thresholds are tol * (sum of squares + mu^2), never -0.0.)
__device__ __forceinline__ bool gt_nonneg_bits(double d, double t) {
    const long long b = __double_as_longlong(d);
    return b > __double_as_longlong(t) && b <= 0x7ff0000000000000LL && !isnan_bits(t);
}
// Warp-wide maximum of the bit patterns of non-negative doubles (0: no entry)
// and the smallest index j that holds it; warp_bitsmin likewise the minimum.
// Three integer warp reductions instead of a butterfly's fifteen shuffles.
__device__ __forceinline__ unsigned long long warp_bitsmax(unsigned long long v, int &j) {
    const unsigned hi = (unsigned)(v >> 32), lo = (unsigned)v;
    const unsigned mh = __reduce_max_sync(FULL, hi), ml = __reduce_max_sync(FULL, hi == mh ? lo : 0u);
    j = (int)__reduce_min_sync(FULL, hi == mh && lo == ml ? (unsigned)j : 0xffffffffu);
    return (unsigned long long)mh << 32 | ml;
}
__device__ __forceinline__ unsigned long long warp_bitsmin(unsigned long long v, int &j) {
    const unsigned hi = (unsigned)(v >> 32), lo = (unsigned)v;
    const unsigned mh = __reduce_min_sync(FULL, hi), ml = __reduce_min_sync(FULL, hi == mh ? lo : 0xffffffffu);
    j = (int)__reduce_min_sync(FULL, hi == mh && lo == ml ? (unsigned)j : 0xffffffffu);
    return (unsigned long long)mh << 32 | ml;
}

// Steps of a Sturm sequence on the integer pipes (an FP64 comparison holds the
// FP64 pipe like any other FP64 instruction): whether p counts as negative (a
// zero takes the sign opposite to its predecessor's), and the rescaling of the
// last two terms by a power of two once the exponent leaves +-400.
__device__ __forceinline__ bool sturm_neg(double p, bool neg) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(p);
    if ((u << 1) == 0) return !neg;
    return u > 0x8000000000000000ull && u <= 0xfff0000000000000ull;  // p < 0, NaN excluded
}
__device__ __forceinline__ void sturm_rescale(double &p1, double &p2) {
    const int hi = __double2hiint(p1), f = hi & 0x7ff00000;
    if ((unsigned)(f - (623 << 20)) > (800u << 20) && (((unsigned)hi << 1) | (unsigned)__double2loint(p1)) != 0u) {
        const double sc = __hiloint2double((2046 << 20) - f, 0);
        p1 *= sc;
        p2 *= sc;
    }
}
// wsum of two values at once: the first butterfly step exchanges a and b
// between the warp halves, so both sums take five additions instead of ten;
// each sum is added in wsum's order, so the results are wsum's bit for bit.
__device__ __forceinline__ void wsum2(double a, double b, double &sa, double &sb) {
    const bool hi = (threadIdx.x & 16) != 0;
    double v = __dadd_rn(hi ? b : a, __shfl_xor_sync(FULL, hi ? a : b, 16));
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_xor_sync(FULL, v, o));
    sa = __shfl_sync(FULL, v, 0);
    sb = __shfl_sync(FULL, v, 16);
}

// The kernels' dynamic shared memory.
extern __shared__ __align__(16) double dk_smem[];

// A pointer into it, held as a byte offset.  The solvers are out of line, and
// through a plain pointer argument the compiler no longer knows the address
// space: every access becomes a generic load or store with a 64-bit address (a
// window check, a longer latency and two address instructions instead of one).
// Indexing dk_smem itself keeps them 32-bit shared-memory accesses:
// 240x240x1 x 48 echoes, L-curve: mixed 72.1 -> 66.3 ms; 120x120x1 FP64 method
// 136.7 -> 131.2 ms.  (Bytes of register spills, stores / loads, by that change:
// k_voxels_plain 328 / 928 -> 68 / 160, k_voxels_mixed 0 / 0 -> 112 / 228.)
template <class T>
struct Sh {
    int off;
    __device__ __forceinline__ T *ptr() const { return reinterpret_cast<T *>(reinterpret_cast<char *>(dk_smem) + off); }
    __device__ __forceinline__ T &operator[](int i) const { return ptr()[i]; }
    __device__ __forceinline__ T &operator*() const { return *ptr(); }
    __device__ __forceinline__ Sh operator+(int i) const { return Sh{off + i * (int)sizeof(T)}; }
    __device__ __forceinline__ Sh &operator+=(int i) { off += i * (int)sizeof(T); return *this; }
    template <class U>
    __device__ __forceinline__ Sh<U> as() const { return Sh<U>{off}; }
};
using ShD = Sh<double>;
using ShI = Sh<int>;

// The nres largest of N eigenvalues by bisection on [lo, hi] with count_below(x)
// = eigenvalues below x, one eigenvalue per lane, each to its own bracket b - a
// <= max(atol, 4 eps b); put(t, a, b) takes the t-th largest's.  Eigenvalues that
// still share a bracket share its midpoint too, so while few brackets are
// distinct the idle lanes evaluate the next levels' midpoints of each -- a
// subtree of 3 to 31 -- and a pass of the sequence settles 2 to 5 levels: about
// 33 passes instead of 50 for a GCV voxel, 240x240x1 x 56 echoes at 60 T2 times,
// mixed method, 130.6 -> 120.2 ms.
template <class Count, class Put>
static __device__ __forceinline__ void warp_bisect(Count &count_below, int N, int nres, double lo, double hi, double atol,
                                                   const ShD sa, const ShD sb, Put put) {
    const int lane = threadIdx.x & 31;
    #pragma unroll 1
    for (int base = 0; base < nres; base += 32) {
        const int t = base + lane;  // t-th largest eigenvalue
        const bool mine = t < nres;
        const int idx = N - 1 - t;  // its index in ascending order
        double a = lo, b = hi;
        bool done = !mine;
        #pragma unroll 1
        for (int it = 0; it < 80 && __any_sync(FULL, !done);) {
            // distinct brackets (neighbours' in lane order) and the levels a pass settles
            const long long ka = __double_as_longlong(a), kb = __double_as_longlong(b);
            const long long ua = __shfl_up_sync(FULL, ka, 1), ub = __shfl_up_sync(FULL, kb, 1);
            const bool first = mine && (lane == 0 || ka != ua || kb != ub);
            const unsigned msk = __ballot_sync(FULL, first);
            const int nd = __popc(msk), grp = __popc(msk & ((2u << lane) - 1u)) - 1;
            const int L = nd <= 1 ? 5 : (nd <= 2 ? 4 : (nd <= 4 ? 3 : (nd <= 10 ? 2 : 1))), nodes = (1 << L) - 1;
            __syncwarp();
            if (first) { sa[grp] = a; sb[grp] = b; }
            __syncwarp();
            // this lane's midpoint: node `nd` of a bracket's subtree, children 2 nd + 1 (left), 2 nd + 2
            const int wg = lane / nodes, node1 = lane - wg * nodes + 1, wr = wg < nd ? wg : 0;
            double wa = sa[wr], wb = sb[wr];
            #pragma unroll 1
            for (int l = 30 - __clz(node1); l >= 0; --l) {
                const double mid = 0.5 * (wa + wb);
                if (node1 >> l & 1) wa = mid; else wb = mid;
            }
            const int c = count_below(0.5 * (wa + wb));
            int node = 0;
            #pragma unroll 1
            for (int l = 0; l < L; ++l, ++it) {
                const int cm = __shfl_sync(FULL, c, (grp < 0 ? 0 : grp) * nodes + node);
                if (!done && it < 80) {
                    const double mid = 0.5 * (a + b);
                    if (cm > idx) b = mid; else a = mid;
                    node = 2 * node + (cm > idx ? 1 : 2);
                    done = (b - a) <= fmax(atol, 4.0 * 2.220446049250313e-16 * b);
                }
                if (node >= nodes) node = 0;  // (the last level's children are not used)
            }
        }
        if (mine) put(t, a, b);
    }
}

// An 8-byte copy from global to shared memory without a register in between;
// copy_async_wait completes the warp's copies.
__device__ __forceinline__ void copy_async(const ShD dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst.ptr())), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async_wait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}

// Per-warp views of the NNLS workspace (shared memory).
struct NnlsWS {
    ShD C;    // lda x n, physical columns
    ShD b;    // (m + n) | 1 whatever lda is (right-hand side, transformed in place)
    ShD zz;   // (m + n) | 1
    ShD x;    // n, indexed by original column (0-based)
    ShD w;    // n, indexed by logical position (0-based)
    ShI idx;  // n, 1-based original column at each logical position
    Sh<unsigned char> diag;  // n, indexed by original column
    ShD rdiag;               // n, RN(1/diagonal) of each physical column in set P
    ShI posof;               // n, 1-based logical position of each physical column (inverse of idx)
    ShI zl;                  // n, scratch list of physical columns
    int lda;
    // rows lim + 1 .. lim + lsp of the columns (the last padding rows, which only
    // solves with nearly every column in set P reach) in global scratch
    int lim, lsp;
    double *sp;
};
// Row i (1-based) of physical column p, and the same past lim.  kSpill: the call
// may reach such rows (out-of-line copies for those calls, so that the others
// test nothing per row).
__device__ __forceinline__ double *spilled(const NnlsWS &s, int p) { return s.sp + (long)p * s.lsp - s.lim - 1; }  // [i], i > lim
template <bool kSpill>
__device__ __forceinline__ double row_get(const NnlsWS &s, int p, int i) {
    return !kSpill || i <= s.lim ? s.C[i - 1 + p * s.lda] : spilled(s, p)[i];
}
template <bool kSpill>
__device__ __forceinline__ void row_set(const NnlsWS &s, int p, int i, double v) {
    if (!kSpill || i <= s.lim) s.C[i - 1 + p * s.lda] = v;
    else spilled(s, p)[i] = v;
}

// Physical columns whose logical position is >= jfirst, in increasing
// physical order, written to s.zl; returns their count.  Column-parallel
// loops walk this list so the lanes of a half-warp read distinct bank pairs
// (odd leading dimension), instead of the random physical columns that the
// logical order would give.
__device__ __forceinline__ int warp_active_cols(const NnlsWS &s, int n, int jfirst) {
    const int lane = threadIdx.x & 31;
    int base = 0;
    #pragma unroll 1
    for (int c = 0; c < n; c += 32) {
        int p = c + lane;
        bool z = p < n && s.posof[p] >= jfirst;
        unsigned msk = __ballot_sync(0xffffffffu, z);
        if (z) s.zl[base + __popc(msk & ((1u << lane) - 1))] = p;
        base += __popc(msk);
    }
    __syncwarp();
    return base;
}

// a / b from r = RN(1/b): q = RN(a r), remainder e = a - b q (exact by fma),
// q' = RN(q + e r).  Markstein's correction (P. Markstein, IBM J. Res. Dev.
// 34(1), 1990) returns the correctly rounded quotient for normal operands, so
// results are bitwise those of a / b at three FP64 operations instead of a
// full division.
__device__ __forceinline__ double mdiv(double a, double b, double r) {
    double q = __dmul_rn(a, r);
    double e = fma(-q, b, a);
    return fma(e, r, q);
}

// Base.hypot for Float64 (C. F. Borges, "An Improved Algorithm for
// hypot(a,b)", 2019, fma-corrected), used by NNLS.orthogonal_rotmat.
static __device__ double jl_hypot(double x, double y) {
    if (isinf(x) || isinf(y)) return CUDART_INF;
    double ax = fabs(x), ay = fabs(y);
    if (ay > ax) { double t = ax; ax = ay; ay = t; }
    if (ay <= ax * 1.0536712127723509e-08) return ax;
    double scale = 2.220446049250313e-16 * 1.4916681462400413e-154;
    if (ax > 9.480751908109176e+153) {
        ax = ax * scale; ay = ay * scale; scale = 1.0 / scale;
    } else if (ay < 1.4916681462400413e-154) {
        ax = ax / scale; ay = ay / scale;
    } else {
        scale = 1.0;
    }
    double h = sqrt(fma(ax, ax, __dmul_rn(ay, ay)));
    double hsq = __dmul_rn(h, h), axsq = __dmul_rn(ax, ax);
    h -= (fma(-ay, ay, hsq - axsq) + fma(h, h, -hsq) - fma(ax, ax, -axsq)) / (2 * h);
    return h * scale;
}

// construct_apply_householder!(A, b, ip, jp, m), src/NNLS.jl:259-336.
// Writes only the pivot column's physical storage (see header note).
template <bool kSpill>
__device__ __forceinline__ double warp_cah_t(const NnlsWS &s, int ip, int jp, int m) {
    const int lane = threadIdx.x & 31;
    if (ip > m) return 0.0;
    const int pc = s.idx[jp - 1] - 1;  // pivot column
    const ShD col = s.C + pc * s.lda;
    double alpha = col[ip - 1];
    double part = 0.0;
    #pragma unroll 1
    for (int i = ip + lane; i <= m; i += 32) { const double v = row_get<kSpill>(s, pc, i); part = fma(v, v, part); }
    double xnorm = sqrt(wsum(part));
    if ((__double_as_longlong(xnorm) << 1) == 0) return -1.0;  // xnorm == 0
    double beta = copysign(xnorm, alpha);
    alpha = alpha + beta;
    // 1 / alpha, alpha / beta and 1 / beta in one division, a lane each (a
    // division is ~10 FP64 warp instructions whatever its active lanes)
    const double qd = (lane == 1 ? alpha : 1.0) / (lane == 0 ? alpha : beta);
    const double ralpha = bcast(qd, 0), rbeta = bcast(qd, 2);
    double tau = bcast(qd, 1);
    // quotients A[i,jp]/alpha, staged in zz (free between solves of the main loop)
    part = 0.0;
    #pragma unroll 1
    for (int i = ip + 1 + lane; i <= m; i += 32) {
        double qi = mdiv(row_get<kSpill>(s, pc, i), alpha, ralpha);
        s.zz[i - 1] = qi;
        part = fma(s.b[i - 1], qi, part);
    }
    double sm = s.b[ip - 1] + wsum(part);
    sm *= -tau;
    double A1 = -beta;
    double b1 = s.b[ip - 1] + sm;
    // b1 / A1 > 0: same nonzero sign and no underflow of the quotient (told by
    // the bit patterns unless |b1| is 2^-899 of |A1| or a value is not normal)
    const int hb = __double2hiint(b1), ha = __double2hiint(A1), eb = hb >> 20 & 0x7ff, ea = ha >> 20 & 0x7ff;
    bool good;
    if (eb > 0 && ea > 0 && eb < 0x7ff && ea < 0x7ff && eb > ea - 899) good = (hb ^ ha) >= 0;
    else if (b1 != 0 && fabs(b1) > 0x1p-900 * fabs(A1)) good = (b1 > 0) == (A1 > 0);
    else good = b1 / A1 > 0;
    if (good) {
        if (ip < m) {
            __syncwarp();
            #pragma unroll 1
            for (int i = ip + 1 + lane; i <= m; i += 32) {
                double qi = s.zz[i - 1];
                row_set<kSpill>(s, pc, i, qi);
                s.b[i - 1] = fma(sm, qi, s.b[i - 1]);
            }
            const double rA1 = -rbeta;  // 1 / (-beta), exact negation
            if (lane == 0) {
                s.b[ip - 1] = b1;
                col[ip - 1] = A1;
                s.rdiag[s.idx[jp - 1] - 1] = rA1;
            }
            __syncwarp();
        } else {
            tau = 0.0;  // column swap only: done by the caller's idx swap
            const double rd = 1.0 / col[ip - 1];
            if (lane == 0) s.rdiag[s.idx[jp - 1] - 1] = rd;
            __syncwarp();
        }
        return tau;
    }
    return -1.0;
}

static __device__ __noinline__ double warp_cah_spill(const NnlsWS s, int ip, int jp, int m) { return warp_cah_t<true>(s, ip, jp, m); }
__device__ __forceinline__ double warp_cah(const NnlsWS &s, int ip, int jp, int m) {
    return m > s.lim ? warp_cah_spill(s, ip, jp, m) : warp_cah_t<false>(s, ip, jp, m);
}

// apply_householder_dual!(A, w, b, tau, j1, m1), src/NNLS.jl:379-436.
// Lanes over logical columns j1+1..n; a column's two sums run down its rows in
// one lane.  A round of at most 16 columns spreads the update between them over
// all lanes, (column, row) pairs at a time: with 8 columns 2.25 instead of 3
// FP64 warp instructions per row: 120x120x1 x 48 echoes, L-curve, 125.5 -> 120.1
// ms; 32x32x4 x 32 echoes, chi2, 17.3 -> 16.75 ms.
template <bool kSpill>
__device__ __forceinline__ void warp_ahd_t(const NnlsWS &s, int n, double tau, int j1, int m1) {
    const int lane = threadIdx.x & 31;
    if (j1 >= m1) return;
    const int pu = s.idx[j1 - 1] - 1, mi = kSpill ? min(m1, s.lim) : m1;  // rows up to mi in shared memory
    const ShD u = s.C + pu * s.lda;                          // u[j1-1] is the diagonal; treated as 1
    const double *us = spilled(s, pu);
    const int nz = warp_active_cols(s, n, j1 + 1);
    #pragma unroll 1
    for (int r0 = 0; r0 < nz; r0 += 32) {
        const int r = r0 + lane, cnt = nz - r0;
        const bool mine = r < nz;
        const int p = mine ? s.zl[r] : 0;
        const ShD a = s.C + p * s.lda;
        double *as = spilled(s, p);
        double sm = 0.0;
        if (mine) {
            sm = fma(a[j1 - 1], 1.0, 0.0);
            #pragma unroll 8
            for (int i = j1 + 1; i <= mi; ++i) sm = fma(a[i - 1], u[i - 1], sm);
            #pragma unroll 1
            for (int i = mi + 1; kSpill && i <= m1; ++i) sm = fma(as[i], us[i], sm);
            sm *= -tau;
            a[j1 - 1] = a[j1 - 1] + sm;
        }
        if (cnt > 16) {
            if (mine) {
                double wj = 0.0;
                #pragma unroll 8
                for (int i = j1 + 1; i <= mi; ++i) {
                    double v = fma(sm, u[i - 1], a[i - 1]);
                    wj = fma(v, s.b[i - 1], wj);
                    a[i - 1] = v;
                }
                #pragma unroll 1
                for (int i = mi + 1; kSpill && i <= m1; ++i) {
                    double v = fma(sm, us[i], as[i]);
                    wj = fma(v, s.b[i - 1], wj);
                    as[i] = v;
                }
                s.w[s.posof[p] - 1] = wj;
            }
        } else {
            const int lg = cnt > 8 ? 4 : (cnt > 4 ? 3 : (cnt > 2 ? 2 : (cnt > 1 ? 1 : 0)));  // 2^lg >= cnt lanes a row
            const int c = lane & ((1 << lg) - 1);
            __syncwarp();
            const double smc = __shfl_sync(FULL, sm, c);
            if (c < cnt) {
                const int q = s.zl[r0 + c];
                const ShD ac = s.C + q * s.lda;
                double *acs = spilled(s, q);
                int i = j1 + 1 + (lane >> lg);
                #pragma unroll 4
                for (; i <= mi; i += 32 >> lg) ac[i - 1] = fma(smc, u[i - 1], ac[i - 1]);
                #pragma unroll 1
                for (; kSpill && i <= m1; i += 32 >> lg) acs[i] = fma(smc, us[i], acs[i]);
            }
            __syncwarp();
            if (mine) {
                double wj = 0.0;
                #pragma unroll 8
                for (int i = j1 + 1; i <= mi; ++i) wj = fma(a[i - 1], s.b[i - 1], wj);
                #pragma unroll 1
                for (int i = mi + 1; kSpill && i <= m1; ++i) wj = fma(as[i], s.b[i - 1], wj);
                s.w[s.posof[p] - 1] = wj;
            }
        }
    }
    __syncwarp();
}

static __device__ __noinline__ void warp_ahd_spill(const NnlsWS s, int n, double tau, int j1, int m1) { warp_ahd_t<true>(s, n, tau, j1, m1); }
__device__ __forceinline__ void warp_ahd(const NnlsWS &s, int n, double tau, int j1, int m1) {
    if (m1 > s.lim) warp_ahd_spill(s, n, tau, j1, m1);
    else warp_ahd_t<false>(s, n, tau, j1, m1);
}

// compute_dual!(w, A, b, j1, m1), src/NNLS.jl:441-470.  Lanes over columns.
template <bool kSpill>
__device__ __forceinline__ void warp_compute_dual_t(const NnlsWS &s, int n, int j1, int m1) {
    const int lane = threadIdx.x & 31;
    const int nz = warp_active_cols(s, n, j1), mi = kSpill ? min(m1, s.lim) : m1;
    #pragma unroll 1
    for (int r0 = 0; r0 < nz; r0 += 32) {
        int r = r0 + lane;
        if (r < nz) {
            const int p = s.zl[r];
            const ShD a = s.C + p * s.lda;
            const double *as = spilled(s, p);
            double sm = 0.0;
            #pragma unroll 8
            for (int i = j1; i <= mi; ++i) sm = fma(a[i - 1], s.b[i - 1], sm);
            #pragma unroll 1
            for (int i = mi + 1; kSpill && i <= m1; ++i) sm = fma(as[i], s.b[i - 1], sm);
            s.w[s.posof[p] - 1] = sm;
        }
    }
    __syncwarp();
}

static __device__ __noinline__ void warp_compute_dual_spill(const NnlsWS s, int n, int j1, int m1) { warp_compute_dual_t<true>(s, n, j1, m1); }
__device__ __forceinline__ void warp_compute_dual(const NnlsWS &s, int n, int j1, int m1) {
    if (m1 > s.lim) warp_compute_dual_spill(s, n, j1, m1);
    else warp_compute_dual_t<false>(s, n, j1, m1);
}

// zz[1:n] = b[1:n]; solve_triangular_system!(zz, A, n), src/NNLS.jl:506-523.
// Lanes over rows; the column sweep is sequential as in the reference.  Up to
// 64 rows stay on their lanes (two each), so a step of the chain passes through
// one shuffle instead of shared memory and two warp barriers.
static __device__ void warp_solve_tri(const NnlsWS &s, int n) {
    const int lane = threadIdx.x & 31;
    if (n <= 64) {
        double z0 = lane < n ? s.b[lane] : 0.0, z1 = lane + 32 < n ? s.b[lane + 32] : 0.0;
        #pragma unroll 1
        for (int j = n; j > 32; --j) {
            const int pj = s.idx[j - 1] - 1;
            const ShD a = s.C + pj * s.lda;
            const double zj = mdiv(bcast(z1, j - 33), a[j - 1], s.rdiag[pj]), zi = -zj;
            z0 = fma(a[lane], zi, z0);
            if (lane < j - 33) z1 = fma(a[lane + 32], zi, z1);
            if (lane == j - 33) z1 = zj;
        }
        #pragma unroll 1
        for (int j = min(n, 32); j >= 1; --j) {
            const int pj = s.idx[j - 1] - 1;
            const ShD a = s.C + pj * s.lda;
            const double zj = mdiv(bcast(z0, j - 1), a[j - 1], s.rdiag[pj]), zi = -zj;
            if (lane < j - 1) z0 = fma(a[lane], zi, z0);
            if (lane == j - 1) z0 = zj;
        }
        if (lane < n) s.zz[lane] = z0;
        if (lane + 32 < n) s.zz[lane + 32] = z1;
        __syncwarp();
        return;
    }
    #pragma unroll 1
    for (int i = lane; i < n; i += 32) s.zz[i] = s.b[i];
    __syncwarp();
    #pragma unroll 1
    for (int j = n; j >= 1; --j) {
        const int pj = s.idx[j - 1] - 1;
        const ShD a = s.C + pj * s.lda;
        double zi = -mdiv(s.zz[j - 1], a[j - 1], s.rdiag[pj]);
        #pragma unroll 1
        for (int i = 1 + lane; i <= j - 1; i += 32) s.zz[i - 1] = fma(a[i - 1], zi, s.zz[i - 1]);
        __syncwarp();
        if (lane == 0) s.zz[j - 1] = -zi;
        __syncwarp();
    }
}

// Logical position j1..n of the largest positive dual (the first one, as the
// reference's `w[j] > wmax` scan from wmax = 0), 0 when there is none.  Positive
// doubles order like their bit patterns, so the search runs on the integer pipes.
__device__ __forceinline__ int warp_largest_dual(const NnlsWS &s, int n, int j1) {
    const int lane = threadIdx.x & 31;
    unsigned long long km = 0;
    int jm = 0;
    #pragma unroll 1
    for (int j = j1 + lane; j <= n; j += 32) {
        const double w = s.w[j - 1];
        const unsigned long long k = (unsigned long long)__double_as_longlong(w);
        if (pos_bits(w) && k > km) { km = k; jm = j; }
    }
    warp_bitsmax(km, jm);
    return jm;
}

struct NnlsResult {
    int nsetp;
    int mode;
    double rnorm;
    double xx;  // ||x||^2 (set by the mixed method's solver only)
};

// Main + secondary loops of unsafe_nnls! (tikh = false) and of its Tikhonov
// form (tikh = true, rows M = m0 + n with lazily activated padding rows).
static __device__ NnlsResult warp_nnls(const NnlsWS &s, int M, int n, int m0, bool tikh, double lam, int max_iter) {
    const int lane = threadIdx.x & 31;
    int m = tikh ? m0 : M;
    int nsetp = 0, iter = 0, mode = 0;
    bool terminated = false;
    #pragma unroll 1
    for (;;) {
        if (nsetp >= n || (!tikh && nsetp >= m)) break;
        int jmax = nsetp;
        double tau = 0.0;
        #pragma unroll 1
        for (;;) {
            jmax = warp_largest_dual(s, n, nsetp + 1);
            if (jmax == 0) { terminated = true; break; }  // no positive dual
            if (tikh && !s.diag[s.idx[jmax - 1] - 1]) {
                if (lane == 0) row_set<true>(s, s.idx[jmax - 1] - 1, m + 1, lam);
                __syncwarp();
            }
            tau = warp_cah(s, nsetp + 1, jmax, tikh ? min(m + 1, M) : m);
            if (!isnan_bits(tau) && __double_as_longlong(tau) >= 0) break;  // tau >= 0 (-1: refused)
            __syncwarp();
            if (lane == 0) {
                s.w[jmax - 1] = 0.0;
                if (tikh && m < M) row_set<true>(s, s.idx[jmax - 1] - 1, m + 1, 0.0);
            }
            __syncwarp();
        }
        if (terminated) break;
        if (tikh && !s.diag[s.idx[jmax - 1] - 1]) {
            m = min(m + 1, M);
            __syncwarp();
            if (lane == 0) s.diag[s.idx[jmax - 1] - 1] = 1;
        }
        nsetp += 1;
        __syncwarp();
        if (lane == 0) {
            int t = s.idx[nsetp - 1];
            s.idx[nsetp - 1] = s.idx[jmax - 1];
            s.idx[jmax - 1] = t;
            s.posof[s.idx[nsetp - 1] - 1] = nsetp;
            s.posof[t - 1] = jmax;
        }
        __syncwarp();
        if (nsetp < n) warp_ahd(s, n, tau, nsetp, m);
        {
            const int pc = s.idx[nsetp - 1] - 1;
            #pragma unroll 1
            for (int i = nsetp + 1 + lane; i <= m; i += 32) row_set<true>(s, pc, i, 0.0);
        }
        __syncwarp();
        if (lane == 0) s.w[nsetp - 1] = 0.0;
        __syncwarp();
        warp_solve_tri(s, nsetp);
        bool dual_flag = false;
        #pragma unroll 1
        for (;;) {
            iter += 1;
            if (iter > max_iter) { mode = 1; terminated = true; break; }
            // feasibility step, src/NNLS.jl:700-727 (first minimum wins)
            int imv = nsetp;
            double alpha = 2.0;
            bool moved = false;
            {
                long long a_key = okey(2.0);
                double a_loc = 2.0;
                int i_loc = 0;
                #pragma unroll 1
                for (int i = 1 + lane; i <= nsetp; i += 32) {
                    double zi = s.zz[i - 1];
                    if (!isnan_bits(zi) && okey(zi) <= 0) {
                        double xi = s.x[s.idx[i - 1] - 1];
                        double t = -xi / (zi - xi);
                        long long tk = okey(t);
                        if (!isnan_bits(t) && a_key > tk) { a_key = tk; a_loc = t; i_loc = i; }
                    }
                }
                moved = __any_sync(FULL, i_loc != 0);
#pragma unroll 1
                for (int o = moved ? 16 : 0; o > 0; o >>= 1) {
                    long long ok = __shfl_xor_sync(FULL, a_key, o);
                    double oa = __shfl_xor_sync(FULL, a_loc, o);
                    int oi = __shfl_xor_sync(FULL, i_loc, o);
                    if (oi != 0 && (i_loc == 0 || ok < a_key || (ok == a_key && oi < i_loc))) { a_key = ok; a_loc = oa; i_loc = oi; }
                }
                if (moved) { imv = i_loc; alpha = a_loc; }
            }
            if (!moved) break;
            dual_flag = true;
            #pragma unroll 1
            for (int i = 1 + lane; i <= nsetp; i += 32) {
                int ix = s.idx[i - 1] - 1;
                s.x[ix] = fma(alpha, s.zz[i - 1] - s.x[ix], s.x[ix]);
            }
            __syncwarp();
            // move coefficient imv (and any infeasible ones) from set P to set Z
            #pragma unroll 1
            for (int guard = 0; guard <= n; ++guard) {
                if (lane == 0) s.x[s.idx[imv - 1] - 1] = 0.0;
                __syncwarp();
                if (imv != nsetp) {
                    #pragma unroll 1
                    for (int i = imv + 1; i <= nsetp; ++i) {
                        const ShD ci = s.C + (s.idx[i - 1] - 1) * s.lda;
                        double a = ci[i - 2], bb = ci[i - 1];
                        double sg = jl_hypot(a, bb);
                        // both rotation coefficients and 1 / sg in one division, a lane each
                        const double qd = (lane == 0 ? a : (lane == 1 ? bb : 1.0)) / sg;
                        const double cc = bcast(qd, 0), ss = bcast(qd, 1);
                        __syncwarp();
                        const int pi = s.idx[i - 1] - 1;
                        // the other columns, and b as column n
                        #pragma unroll 1
                        for (int pj = lane; pj <= n; pj += 32) {
                            if (pj == pi) continue;
                            const ShD cj = pj < n ? s.C + pj * s.lda : s.b;
                            double p = cj[i - 2], r = cj[i - 1];
                            cj[i - 2] = fma(cc, p, __dmul_rn(ss, r));
                            cj[i - 1] = fma(-ss, p, __dmul_rn(cc, r));
                        }
                        if (lane == 2) {
                            ci[i - 2] = sg;
                            ci[i - 1] = 0.0;
                            s.rdiag[pi] = qd;
                        }
                        __syncwarp();
                    }
                    // move logical column imv to position nsetp (idx rotation; no data moves)
                    if (lane == 0) {
                        int t = s.idx[imv - 1];
                        #pragma unroll 1
                        for (int j = imv; j <= nsetp - 1; ++j) {
                            s.idx[j - 1] = s.idx[j];
                            s.posof[s.idx[j - 1] - 1] = j;
                        }
                        s.idx[nsetp - 1] = t;
                        s.posof[t - 1] = nsetp;
                    }
                    __syncwarp();
                }
                nsetp -= 1;
                // first remaining infeasible coefficient, if any
                int bad = 0;
                #pragma unroll 1
                for (int ib = 1; ib <= nsetp; ib += 32) {
                    int i = ib + lane;
                    bool neg = (i <= nsetp) && nonpos_bits(s.x[s.idx[i - 1] - 1]);
                    unsigned msk = __ballot_sync(FULL, neg);
                    if (msk) { bad = ib + __ffs(msk) - 1; break; }
                }
                if (bad == 0) break;
                imv = bad;
            }
            warp_solve_tri(s, nsetp);
        }
        if (terminated) break;
        if (dual_flag) warp_compute_dual(s, n, nsetp + 1, m);
        #pragma unroll 1
        for (int i = 1 + lane; i <= nsetp; i += 32) s.x[s.idx[i - 1] - 1] = s.zz[i - 1];
        __syncwarp();
    }
    // residual norm over the remaining rows (all padded rows for the Tikhonov form)
    const int rows = tikh ? M : m;
    double part = 0.0;
    if (nsetp < rows) {
        #pragma unroll 1
        for (int i = nsetp + 1 + lane; i <= rows; i += 32) part = fma(s.b[i - 1], s.b[i - 1], part);
    } else {
        #pragma unroll 1
        for (int j = lane; j < n; j += 32) s.w[j] = 0.0;
    }
    __syncwarp();
    NnlsResult r;
    r.rnorm = sqrt(wsum(part));
    r.nsetp = nsetp;
    r.mode = mode;
    return r;
}

// Warm start of solve!(::NNLSProblem, A, b) (src/lsqnonneg.jl:30-84) and of
// its Tikhonov form (src/lsqnonneg.jl:86-164): copy A (global, m x n) into
// the workspace, seed the dual with column n, then run the NNLS loops.
// `data` is the (shared-memory) right-hand side; it is not modified.
// Not inlined: every caller shares one copy of the NNLS code (instruction
// cache), and the workspace views travel in registers.
static __device__ __noinline__ NnlsResult warp_lsq(const NnlsWS s, const double *A, int m, int n, const ShD data,
                                            bool tikh, double mu) {
    const int lane = threadIdx.x & 31;
    const int M = tikh ? m + n : m;
    // C[:, j] = A[:, j] (coalesced, asynchronous: all copies in flight at once),
    // padded rows zeroed
    #pragma unroll 1
    for (int j = 0; j < n; ++j) {
        const double *aj = A + (size_t)j * m;
        const ShD cj = s.C + j * s.lda;
        #pragma unroll 1
        for (int i = lane; i < m; i += 32) copy_async(cj + i, aj + i);
        #pragma unroll 1
        for (int i = m + lane; i < M; i += 32) row_set<true>(s, j, i + 1, 0.0);
    }
    #pragma unroll 1
    for (int i = lane; i < M; i += 32) s.b[i] = (i < m) ? data[i] : 0.0;
    #pragma unroll 1
    for (int j = lane; j < n; j += 32) {
        s.x[j] = 0.0;
        s.idx[j] = j + 1;
        s.posof[j] = j + 1;
        s.diag[j] = 0;
    }
    copy_async_wait();
    const ShD an = s.C + (n - 1) * s.lda;
    double part = 0.0;
    #pragma unroll 1
    for (int i = lane; i < m; i += 32) part = __dadd_rn(part, __dmul_rn(an[i], an[i]));
    double den = wsum(part);
    if (tikh) den = __dadd_rn(den, __dmul_rn(mu, mu));
    const double rden = 1.0 / den;
    part = 0.0;
    #pragma unroll 1
    for (int i = lane; i < m; i += 32) part = __dadd_rn(part, __dmul_rn(mdiv(an[i], den, rden), data[i]));
    double xj = wsum(part);
    #pragma unroll 1
    for (int i = lane; i < m; i += 32) s.zz[i] = __dsub_rn(data[i], __dmul_rn(an[i], xj));
    __syncwarp();
    bool pos = false;
    #pragma unroll 1
    for (int jb = 0; jb < n - 1; jb += 32) {
        int j = jb + lane;
        if (j < n - 1) {
            const ShD cj = s.C + j * s.lda;
            double wj = 0.0;
            #pragma unroll 8
            for (int i = 0; i < m; ++i) wj = __dadd_rn(wj, __dmul_rn(cj[i], s.zz[i]));
            s.w[j] = wj;
            pos |= !nonpos_bits(wj);
        }
    }
    bool anypos = __any_sync(FULL, pos);
    if (lane == 0) s.w[n - 1] = anypos ? 0.0 : 1.0;
    __syncwarp();
    return warp_nnls(s, M, n, m, tikh, mu, 3 * n);
}

// sum(abs2, positive_solution): ||x||^2 over the active set in set-P order.
static __device__ double warp_seminorm_sq(const NnlsWS &s, int nsetp) {
    const int lane = threadIdx.x & 31;
    double part = 0.0;
    #pragma unroll 1
    for (int i = lane; i < nsetp; i += 32) {
        double v = s.x[s.idx[i] - 1];
        part = __dadd_rn(part, __dmul_rn(v, v));
    }
    return wsum(part);
}

}  // namespace dk
