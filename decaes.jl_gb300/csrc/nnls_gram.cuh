// nnls_gram.cuh -- Lawson-Hanson NNLS on the normal equations, one warp per
// problem: the solver of the mixed-precision method (DECAES_PREC_MIXED).
//
// The plain method factors the (m+n) x n Tikhonov-padded basis by Householder
// QR on every solve (src/NNLS.jl).  Here each basis gets its Gram matrix
// G = A'A and right-hand side f = A'b once; a Tikhonov solve at any mu then
// works on H = G + mu^2 I restricted to the passive set P:
//   * the passive set grows and shrinks exactly as in Lawson-Hanson (add the
//     column with the largest positive dual w = f - H x, step back to
//     feasibility when the unconstrained solution on P leaves the orthant);
//   * H_PP is held as an LDL' factorization (unit lower L, pivots D),
//     extended by one bordered row per added column and refactored
//     (right-looking) after a removal or a change of mu;
//   * every solve may start from the previous solve's passive set (the
//     problem is strictly convex for mu > 0, so any start reaches the same
//     minimizer): successive mu's of the regularizer searches share most of
//     their support, which cuts the number of column additions about 7x.
// All arithmetic is FP64 (the Gram matrix squares the basis condition number,
// so single precision is not enough for it); the saving is in operation count:
// per added column O(k) warp instructions on k <= n passive columns instead of
// O((m+n)(n-k)) for a Householder step.
//
// FP64 results take ~64 cycles to come back on this part, so the factorization
// avoids square roots and divisions on its dependency chain: LDL' instead of
// Cholesky, reciprocals seeded in FP32 and finished with one cubic Newton
// step, unit-diagonal substitutions (one shuffle + one FMA per step), and the
// trailing update of the factorization as independent FMAs.
//
// Storage (shared memory, packed to keep more warps resident): G as its upper
// triangle by columns, G(i,j) = Gp[j(j+1)/2 + i] for i <= j; L strictly lower
// by rows, L(r,q) = Lp[r(r-1)/2 + q] for q < r.  Passive rows r live on lanes
// r and r+32 (n <= 64).
#pragma once
#include "nnls_warp.cuh"

namespace dk {

constexpr int kGramMaxN = 64;
constexpr double kGramDepTol = 1e-12;  // reject a column when its pivot <= tol * H_tt

__device__ __forceinline__ int tri(int j) { return (j * (j + 1)) >> 1; }
// packed symmetric G: entry (i, j)
__device__ __forceinline__ int gidx(int i, int j) { return i <= j ? tri(j) + i : tri(i) + j; }

struct GramWS {
    ShD G;     // packed upper triangle of the Gram matrix, n(n+1)/2
    ShD L;     // packed strictly-lower unit factor of H_PP = L D L'
    int nL;    // doubles at L
    ShD f;     // A'b
    ShD y;     // L^{-1} f_P
    ShD dd;    // factorization scratch: the running diagonal, or a scaled pivot column
    ShD dinv;  // 1 / D
    ShD xp;    // x on P (xp[r] = x[P[r]])
    ShI P;     // passive columns, 0-based, k entries; kept for the next solve's warm start
    int lastk;
    double bb;     // b'b
};

// 1/d for normal d: the hardware's approximate FP64 reciprocal (rcp.approx,
// relative error below 2^-20) refined by one cubic Newton step
// r(1 + e + e^2), e = 1 - d r, whose error e^3 is below FP64 rounding.
__device__ __forceinline__ double fast_rcp(double d) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
    const double e = fma(-d, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

__device__ __forceinline__ double lane_pick(double v0, double v1, int i) {
    // value held for row i (rows i < 32 in v0, rows >= 32 in v1) broadcast from its lane
    return __shfl_sync(FULL, i < 32 ? v0 : v1, i & 31);
}

// An FP32 value as FP64 by moving its exponent and mantissa fields (integer
// pipes; exact for zero and normal numbers, the only values an EPG curve takes
// here).
__device__ __forceinline__ double widen(float f) {
    const unsigned u = __float_as_uint(f);
    const unsigned e = (u >> 23) & 0xffu;
    const unsigned long long sgn = (unsigned long long)(u >> 31) << 63;
    const unsigned long long mag = e == 0 ? 0ull
                                          : ((unsigned long long)(e + (1023 - 127)) << 52) | ((unsigned long long)(u & 0x7fffffu) << 29);
    return __longlong_as_double((long long)(sgn | mag));
}
// The same for a value with its sign bit clear (an EPG curve is an absolute
// value), in half the instructions.
__device__ __forceinline__ double widen_abs(float f) {
    const unsigned u = __float_as_uint(f);
    return __hiloint2double(u < 0x800000u ? 0 : (int)((u >> 3) + 0x38000000u), u < 0x800000u ? 0 : (int)(u << 29));
}

// Tile of the factorization: the lower triangle of the matrix still to be
// factored with the right-hand side as a row below it, in one run of shared
// memory.  Rows and columns count from the end -- rho = k - r for matrix row r,
// 0 for the right-hand side; gamma = k - c -- and element (rho, gamma), rho <=
// gamma, has number gamma (gamma + 1) / 2 + rho.  So the trailing elements of
// every step, of any k, are the first numbers.  gamma of a number is the count
// of triangular numbers up to it: those before its block of 32 numbers, and a
// bit mask of those in the block (one constant load, one population count).
struct TileBlocks {
    unsigned mask[66];  // triangular numbers in block s, and how many (of 1, 3, 6, ...) come before it
    int below[66];
    constexpr TileBlocks() : mask(), below() {
        for (int s = 0; s < 66; ++s)
            for (int g = 1; g * (g + 1) / 2 < 32 * s + 32; ++g)
                if (g * (g + 1) / 2 < 32 * s) below[s] = g;
                else mask[s] |= 1u << (g * (g + 1) / 2 - 32 * s);
    }
};
static __constant__ const TileBlocks kTile;
// element e = 32 s + lane (also entry (rho, gamma) of the packed Gram matrix)
__device__ __forceinline__ void tile_element(int s, int e, unsigned lanes_le, int &rho, int &gamma) {
    gamma = kTile.below[s] + __popc(kTile.mask[s] & lanes_le);
    rho = e - tri(gamma);
}

// b'b.
static __device__ void gram_bb(GramWS &g, int m, const ShD b) {
    const int lane = threadIdx.x & 31;
    double part = 0.0;
    #pragma unroll 1
    for (int i = lane; i < m; i += 32) part = fma(b[i], b[i], part);
    g.bb = wsum(part);
}

// f = A'b from a row-major (transposed, m x n) basis in global memory: a lane
// per column and row parity (the even and the odd rows have sums of their own,
// added at the end), so 40 columns take 3 rounds of 24 rows instead of 2 of 48;
// four loads are in flight.
static __device__ __noinline__ void gram_rhs_t(GramWS &g, const double *AT, int m, int n, const ShD b) {
    const int lane = threadIdx.x & 31, par = lane & 1;
    #pragma unroll 1
    for (int t = lane; t - lane < 2 * n; t += 32) {
        const int j = t >> 1;
        double s = 0.0;
        if (j < n) {
            const double *a = AT + j;
            #pragma unroll 4
            for (int i = par; i < m; i += 2) s = fma(__ldg(a + (long)i * n), b[i], s);
        }
        __syncwarp();
        s = s + __shfl_xor_sync(FULL, s, 1);
        if (par == 0 && j < n) g.f[j] = s;
    }
    __syncwarp();
}

// f = A'b from a precomputed row of products held as float pairs (hi, lo)
// (the tensor-core grid products of the voxel), times their scale to the
// normalized decay.
static __device__ __noinline__ void gram_rhs_f32(GramWS &g, const float *F, int n, double scale, int m,
                                                 const ShD b) {
    const int lane = threadIdx.x & 31;
    #pragma unroll 1
    for (int j = lane; j < n; j += 32) {
        const float2 v = __ldg(reinterpret_cast<const float2 *>(F) + j);
        g.f[j] = (widen(v.x) + widen(v.y)) * scale;
    }
    __syncwarp();
}

// f = A'b and G = A'A from a basis staged in shared memory as FP32 values
// (column-major, odd leading dimension lda).  The staged values are the FP32
// EPG curves themselves, so the products are exact in FP64 and G is the Gram
// matrix of the basis to FP64 rounding.  Lanes over columns for f and over the
// n(n+1)/2 upper-triangle entries for G.
static __device__ __noinline__ void gram_build_f32(GramWS &g, const Sh<float> As, int lda, int m, int n, const ShD b) {
    const int lane = threadIdx.x & 31;
    #pragma unroll 1
    for (int j = lane; j < n; j += 32) {
        const Sh<float> aj = As + j * lda;
        double s0 = 0.0, s1 = 0.0;
        int i = 0;
        #pragma unroll 1
        for (; i + 1 < m; i += 2) {
            s0 = fma(widen_abs(aj[i]), b[i], s0);
            s1 = fma(widen_abs(aj[i + 1]), b[i + 1], s1);
        }
        if (i < m) s0 = fma(widen_abs(aj[i]), b[i], s0);
        g.f[j] = s0 + s1;
    }
    // 32 entries at a time from the last: As reaches into G from below, and an
    // entry overwrites only columns that none before it reads
    const unsigned lanes_le = (2u << lane) - 1u;
    #pragma unroll 1
    for (int b0 = (tri(n) - 1) >> 5; b0 >= 0; --b0) {
        const int p = 32 * b0 + lane;
        double s0 = 0.0, s1 = 0.0;
        if (p < tri(n)) {
            int i, j;
            tile_element(b0, p, lanes_le, i, j);
            const Sh<float> ai = As + i * lda, aj = As + j * lda;
            int r = 0;
            #pragma unroll 1
            for (; r + 1 < m; r += 2) {
                s0 = fma(widen_abs(ai[r]), widen_abs(aj[r]), s0);
                s1 = fma(widen_abs(ai[r + 1]), widen_abs(aj[r + 1]), s1);
            }
            if (r < m) s0 = fma(widen_abs(ai[r]), widen_abs(aj[r]), s0);
        }
        __syncwarp();
        if (p < tri(n)) g.G[p] = s0 + s1;
        __syncwarp();
    }
}

// Starts the copy of G from a precomputed packed Gram matrix in global memory;
// copy_async_wait before it is read.  Asynchronous copies need no registers, so
// all of them are in flight at once, behind the right-hand side's products.
static __device__ __noinline__ void gram_load(GramWS &g, const double *Gg, int n) {
    const int lane = threadIdx.x & 31;
    const int np = tri(n);
#pragma unroll 4
    for (int q = lane; q < np; q += 32) copy_async(g.G + q, Gg + q);
}

// LDL' factorization of H_PP = G_PP + mu2 I from scratch (right-looking) for k
// <= 32, with y = L^{-1} f_P carried along as an extra row, on a tile held
// behind the factor (k^2 doubles for both).  Per pivot: one reciprocal, the
// column scaled by the lanes of its rows, and the trailing update of 32 tile
// elements at a time; the elements of the next pivot column also go to a
// buffer of their own.  gram_refactor_large's update finds each element's row
// and column by a square root and both operands in the packed factor, ~45
// instructions a round against ~16 here.  The loops are kept small on purpose:
// the same tile held in registers (no loads or stores of its elements, 15-30
// KB of unrolled code) ran 3-35% slower, all of the kernel with it, waiting for
// instructions.  Returns false when a pivot is not positive relative to its
// diagonal (numerically dependent set).  Until the results are written, y and
// dd hold a pivot column and its scaled copy.
static __device__ __forceinline__ bool gram_refactor_tile(const GramWS g, int k, double mu2) {
    const int lane = threadIdx.x & 31;
    ShD col = g.xp, nxt = g.y;
    const ShD lb = g.dd, Lr = g.L + tri(lane - 1), T = g.L + tri(k - 1);
    double th = 0.0, yv = 0.0, dv = 0.0;  // lane r: row r's pivot threshold tol * H_rr, y and reciprocal pivot
    if (lane < k) {
        const int p = g.P[lane];
        th = kGramDepTol * (g.G[tri(p) + p] + mu2);
    }
    const unsigned lanes_le = (2u << lane) - 1u;
    #pragma unroll 1
    for (int s = 0, e = lane; e < tri(k + 1); ++s, e += 32) {  // the first pivot column goes to its buffer
        int rho, gamma;
        tile_element(s, e, lanes_le, rho, gamma);
        if (gamma == 0) continue;  // (0, 0) is no element
        const int pc = g.P[k - gamma];
        double h;
        if (rho == 0) {
            h = g.f[pc];
        } else {
            h = g.G[gidx(g.P[k - rho], pc)];
            if (rho == gamma) h = h + mu2;
        }
        if (gamma == k) col[rho] = h;
        else T[e] = h;
    }
    __syncwarp();
    #pragma unroll 1
    for (int gp = k; gp > 0; --gp) {  // gamma of the pivot column j = k - gp
        const int j = k - gp;
        const double d = col[gp];
        if (__any_sync(FULL, lane == j && !gt_nonneg_bits(d, th))) return false;  // d > tol * H_jj
        const double rd = fast_rcp(d);
        if (lane == j) { yv = col[0]; dv = rd; }
        if (lane > j && lane < k) {
            const double l = col[k - lane] * rd;
            lb[k - lane] = l;
            Lr[j] = l;
        }
        __syncwarp();
        const int trail = gp > 1 ? tri(gp) : 0;
        #pragma unroll 1
        for (int s = 0, e = lane; e < trail; ++s, e += 32) {
            int rho, gamma;
            tile_element(s, e, lanes_le, rho, gamma);
            const double h = fma(-col[rho], lb[gamma], T[e]);
            T[e] = h;
            if (gamma == gp - 1) nxt[rho] = h;
        }
        const ShD s = col; col = nxt; nxt = s;
        __syncwarp();
    }
    if (lane < k) { g.y[lane] = yv; g.dinv[lane] = dv; }
    __syncwarp();
    return true;
}

// LDL' factorization of H_PP = G_PP + mu2 I from scratch (right-looking)
// for any k, with y = L^{-1} f_P carried along as an extra column.  Per pivot: one
// reciprocal, the column scaled by the lanes of its rows, and the trailing
// update -- diagonal included -- spread over lanes by (row, column) pair, so a
// step costs ~(k-j)^2/64 FMA instructions instead of k-j.  Returns false when
// a pivot is not positive relative to its diagonal (numerically dependent set).
static __device__ __noinline__ bool gram_refactor_large(GramWS g, int k, double mu2) {
    const int lane = threadIdx.x & 31;
    const int r0 = lane, r1 = lane + 32;
    const int p0 = r0 < k ? g.P[r0] : 0, p1 = r1 < k ? g.P[r1] : 0;
    const ShD L0 = g.L + tri(r0 - 1), L1 = g.L + tri(r1 - 1);
    const ShD cu = g.xp;  // unscaled pivot column of the current step
    // strictly lower triangle and diagonal of H_PP, one row per lane, and each
    // row's pivot threshold tol * H_rr
    double th0 = 0.0, th1 = 0.0;
    if (r0 < k) {
        #pragma unroll 1
        for (int c = 0; c < r0; ++c) L0[c] = g.G[gidx(p0, g.P[c])];
        const double h = g.G[tri(p0) + p0] + mu2;
        g.dd[r0] = h;
        th0 = kGramDepTol * h;
    }
    if (r1 < k) {
        #pragma unroll 1
        for (int c = 0; c < r1; ++c) L1[c] = g.G[gidx(p1, g.P[c])];
        const double h = g.G[tri(p1) + p1] + mu2;
        g.dd[r1] = h;
        th1 = kGramDepTol * h;
    }
    double v0 = r0 < k ? g.f[p0] : 0.0, v1 = r1 < k ? g.f[p1] : 0.0;
    __syncwarp();
    #pragma unroll 1
    for (int j = 0; j < k; ++j) {
        const double d = g.dd[j];
        if (!gt_nonneg_bits(d, lane_pick(th0, th1, j))) return false;  // d > tol * H_jj
        const double rd = fast_rcp(d);
        const double yj = lane_pick(v0, v1, j);
        if (r0 > j && r0 < k) {
            const double c0 = L0[j], l0 = c0 * rd;
            L0[j] = l0;
            cu[r0] = c0;
            v0 = fma(-l0, yj, v0);
        }
        if (r1 > j && r1 < k) {
            const double c1 = L1[j], l1 = c1 * rd;
            L1[j] = l1;
            cu[r1] = c1;
            v1 = fma(-l1, yj, v1);
        }
        if (lane == 0) g.dinv[j] = rd;
        __syncwarp();
        // trailing lower entries (r, c), j < c <= r < k, one per lane: the
        // strictly-lower ones in L and the running diagonal (c == r) in dd
        const int t = k - 1 - j, npair = t * (t + 1) / 2;
        #pragma unroll 1
        for (int q = lane; q < npair; q += 32) {
            int a = (int)((sqrtf(8.0f * (float)q + 1.0f) - 1.0f) * 0.5f);
            while (a * (a + 1) / 2 > q) --a;
            while ((a + 1) * (a + 2) / 2 <= q) ++a;
            const int r = j + 1 + a, c = j + 1 + (q - a * (a + 1) / 2);
            const ShD e = c == r ? g.dd + r : g.L + tri(r - 1) + c;
            *e = fma(-cu[r], g.L[tri(c - 1) + j], *e);
        }
        __syncwarp();
    }
    if (r0 < k) g.y[r0] = v0;
    if (r1 < k) g.y[r1] = v1;
    __syncwarp();
    return true;
}

__device__ __forceinline__ bool gram_refactor(const GramWS &g, int k, double mu2) {
    return k <= 32 && k * k <= g.nL ? gram_refactor_tile(g, k, mu2) : gram_refactor_large(g, k, mu2);
}

// Extends the factorization by column t (k -> k+1): u = L^{-1} H[P,t],
// w = D^{-1} u, delta = H_tt - u'w, y_t = f_t - w'y.  Rejects t when delta is
// not positive relative to H_tt or when its coefficient y_t / delta in the
// unconstrained solution on P + {t} is not positive (the guards of the
// reference's Householder step).  Returns true when t was added.
static __device__ __forceinline__ bool gram_append(const GramWS g, int k, int t, double mu2) {
    const int lane = threadIdx.x & 31;
    const int r0 = lane, r1 = lane + 32;
    double v0 = r0 < k ? g.G[gidx(g.P[r0], t)] : 0.0, v1 = 0.0;
    const ShD L0 = g.L + tri(r0 - 1);
    if (k <= 32) {
        #pragma unroll 1
        for (int i = 0; i < k; ++i) {
            const double ui = bcast(v0, i);
            if (r0 > i && r0 < k) v0 = fma(-L0[i], ui, v0);
        }
    } else {
        const ShD L1 = g.L + tri(r1 - 1);
        if (r1 < k) v1 = g.G[gidx(g.P[r1], t)];
        #pragma unroll 1
        for (int i = 0; i < k; ++i) {
            const double ui = lane_pick(v0, v1, i);
            if (r0 > i) v0 = fma(-L0[i], ui, v0);
            if (r1 > i && r1 < k) v1 = fma(-L1[i], ui, v1);
        }
    }
    double w0 = 0.0, w1 = 0.0, pl = 0.0, py = 0.0;
    if (r0 < k) { w0 = v0 * g.dinv[r0]; pl = fma(v0, w0, pl); py = fma(w0, g.y[r0], py); }
    if (r1 < k) { w1 = v1 * g.dinv[r1]; pl = fma(v1, w1, pl); py = fma(w1, g.y[r1], py); }
    double ll, ly;
    wsum2(pl, py, ll, ly);
    const double htt = g.G[tri(t) + t] + mu2;
    const double delta = htt - ll;
    if (!gt_nonneg_bits(delta, kGramDepTol * htt)) return false;
    const double yt = g.f[t] - ly;
    if (!pos_bits(yt)) return false;
    const double rd = fast_rcp(delta);
    const ShD Lk = g.L + tri(k - 1);
    if (r0 < k) Lk[r0] = w0;
    if (r1 < k) Lk[r1] = w1;
    if (lane == 0) {
        g.dinv[k] = rd;
        g.y[k] = yt;
        g.P[k] = t;
    }
    __syncwarp();
    return true;
}

// z = L^{-T} D^{-1} y (unit upper back substitution, lanes over rows);
// z returned in (z0, z1).
static __device__ __forceinline__ double2 gram_back(const GramWS g, int k) {
    const int lane = threadIdx.x & 31;
    const int r0 = lane, r1 = lane + 32;
    double u0 = r0 < k ? g.y[r0] * g.dinv[r0] : 0.0, u1 = 0.0;
    int i = k - 1;
    if (k > 32) {
        if (r1 < k) u1 = g.y[r1] * g.dinv[r1];
        #pragma unroll 1
        for (; i >= 32; --i) {
            const double zi = bcast(u1, i & 31);
            const ShD Li = g.L + tri(i - 1);
            u0 = fma(-Li[r0], zi, u0);
            if (r1 < i) u1 = fma(-Li[r1], zi, u1);
        }
    }
    #pragma unroll 1
    for (; i > 0; --i) {
        const double zi = bcast(u0, i);
        if (r0 < i) u0 = fma(-g.L[tri(i - 1) + r0], zi, u0);
    }
    return make_double2(u0, u1);
}

// Singular values of the basis for GCV, as square roots of the eigenvalues of
// its Gram matrix (the mixed method's stand-in for svdvals(A)):
//   1. Householder tridiagonalization of G in a packed lower working copy W
//      (W(r,c) = W[r(r+1)/2 + c], c <= r: the same packing as G's upper
//      triangle by columns, so the copy is a straight one), lanes over rows;
//   2. eigenvalues of the tridiagonal matrix by bisection, one eigenvalue per
//      lane, counting sign changes of the Sturm sequence p_j = (d_j - x)
//      p_{j-1} - e_{j-1}^2 p_{j-2} (no divisions on the chain; rescaled by
//      powers of two when its exponent leaves +-400).
// Only eigenvalues above tau = 1e-14 * (Gershgorin bound) are resolved: GCV's
// mu is at least exp(-8), so smaller ones enter its dof sum as 1 either way
// (error <= tau / mu^2 per eigenvalue).  Eigenvalues are resolved to an
// absolute 1e-15 * bound.  Writes the min(m,n) largest square roots in
// descending order to gam (zeros for the unresolved ones).  Uses y, xp, dd and
// dinv as scratch (free before the first solve) and W (tri(n) doubles).
static __device__ __noinline__ void gram_svdvals(GramWS g, const ShD W, int m, int n, double *gam) {
    const int lane = threadIdx.x & 31;
    const int np = tri(n);
#pragma unroll 1
    for (int q = lane; q < np; q += 32) W[q] = g.G[q];
    __syncwarp();
    const ShD d = g.dd, e = g.dinv, u = g.y, qv = g.xp;
    const unsigned lanes_le = (2u << lane) - 1u;
    // 1. tridiagonalization (Householder from the left and right, column k)
#pragma unroll 1
    for (int k = 0; k + 2 < n; ++k) {
        double part = 0.0;
#pragma unroll 1
        for (int r = k + 2 + lane; r < n; r += 32) { const double x = W[tri(r) + k]; part = fma(x, x, part); }
        const double sigma = wsum(part);
        const double x1 = W[tri(k + 1) + k];
        if (lane == 0) d[k] = W[tri(k) + k];
        if (!(sigma > 0)) {  // column already reduced
            if (lane == 0) e[k] = x1;
            __syncwarp();
            continue;
        }
        const double nrm = sqrt(fma(x1, x1, sigma));
        const double alpha = x1 >= 0 ? -nrm : nrm;
        const double u1 = x1 - alpha;
        const double beta = 2.0 / fma(u1, u1, sigma);
        if (lane == 0) e[k] = alpha;
#pragma unroll 1
        for (int r = k + 1 + lane; r < n; r += 32) u[r] = (r == k + 1) ? u1 : W[tri(r) + k];
        __syncwarp();
        // p = beta W22 u on rows r > k (W symmetric: W(r,c) from row max(r,c))
        double pk = 0.0;
#pragma unroll 1
        for (int r = k + 1 + lane; r < n; r += 32) {
            const int br = tri(r);
            double s0 = 0.0, s1 = 0.0;
            int c = k + 1;
#pragma unroll 1
            for (; c + 1 < n; c += 2) {
                s0 = fma(W[c <= r ? br + c : tri(c) + r], u[c], s0);
                s1 = fma(W[c + 1 <= r ? br + c + 1 : tri(c + 1) + r], u[c + 1], s1);
            }
            if (c < n) s0 = fma(W[c <= r ? br + c : tri(c) + r], u[c], s0);
            const double pr = beta * (s0 + s1);
            qv[r] = pr;
            pk = fma(u[r], pr, pk);
        }
        const double K = 0.5 * beta * wsum(pk);
        __syncwarp();
#pragma unroll 1
        for (int r = k + 1 + lane; r < n; r += 32) qv[r] = fma(-K, u[r], qv[r]);
        __syncwarp();
        // W22 -= u q' + q u' (lower triangle), lanes over its entries
        const int t = n - k - 1;
        #pragma unroll 1
        for (int s = 0, e = lane; e < tri(t); ++s, e += 32) {
            int c, r;
            tile_element(s, e, lanes_le, c, r);
            c += k + 1;
            r += k + 1;
            const int w = tri(r) + c;
            W[w] = fma(-u[r], qv[c], fma(-qv[r], u[c], W[w]));
        }
        __syncwarp();
    }
    if (lane == 0) {
        if (n >= 2) {
            d[n - 2] = W[tri(n - 2) + n - 2];
            e[n - 2] = W[tri(n - 1) + n - 2];
        }
        d[n - 1] = W[tri(n - 1) + n - 1];
    }
    __syncwarp();
    // squared off-diagonals (reuse W) and the Gershgorin bound
    double bnd = 0.0;
#pragma unroll 1
    for (int j = lane; j < n; j += 32) {
        const double a = j > 0 ? fabs(e[j - 1]) : 0.0, b = j + 1 < n ? fabs(e[j]) : 0.0;
        bnd = fmax(bnd, fabs(d[j]) + a + b);
        if (j + 1 < n) W[j] = e[j] * e[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) bnd = fmax(bnd, __shfl_xor_sync(FULL, bnd, o));
    __syncwarp();
    const ShD e2 = W;
    const double tau = 1e-14 * bnd, atol = 1e-15 * bnd;
    // Sturm count: eigenvalues of the tridiagonal matrix below x
    auto count_below = [&](double x) {
        double p2 = 1.0, p1 = d[0] - x;
        bool neg = sturm_neg(p1, false);  // (p_0 = +1)
        int c = neg;
#pragma unroll 2
        for (int j = 1; j < n; ++j) {
            const double p = fma(d[j] - x, p1, -e2[j - 1] * p2);
            const bool pneg = sturm_neg(p, neg);
            c += (pneg != neg);
            neg = pneg;
            p2 = p1;
            p1 = p;
            sturm_rescale(p1, p2);
        }
        return c;
    };
    const int nz = count_below(tau);  // eigenvalues below tau: left at zero
    const int kk = m < n ? m : n;
    const int nres = n - nz;  // resolved eigenvalues (the largest)
    warp_bisect(count_below, n, nres, tau, bnd, atol, u, qv, [&](int t, double a, double b) {
        if (t < kk) gam[t] = sqrt(0.5 * (a + b));
    });
#pragma unroll 1
    for (int t = nres + lane; t < kk; t += 32) gam[t] = 0.0;
    __syncwarp();
}

// NNLS on H = G + mu2 I with right-hand side f (prepared by gram_rhs_t /
// gram_build_f32 / gram_load, which also set b'b).  On return x (dense, n)
// holds the solution, nsetp the size of its passive set (in g.P, from where
// the next solve of the voxel starts: *lastk_io entries, 0: from scratch),
// rnorm^2 = ||A x - b||^2 + mu2 ||x||^2 and xx = ||x||^2 as warp_seminorm_sq
// sums it.  mode = 1 when max_iter was reached (the reference's cap 3n).
//
// x on the passive set lives on the lanes of its rows (x0, x1); the free
// columns' duals, compacted, in wv with their columns in fc.  The factorization,
// the append and the back substitution are inlined at their one call site each:
// a solve makes ~10 of these short calls, and their argument passing cost 4.5%
// of a 48-echo L-curve voxel and 7% of a chi2 one (240x240x1 53.0 -> 50.6 ms,
// 240x240x4 87.7 -> 81.4 ms).
static __device__ __noinline__ NnlsResult gram_nnls(const GramWS g, const ShD x, const ShD wv, const ShI fc, int n, double mu2,
                                             int max_iter, int *lastk_io) {
    const int lane = threadIdx.x & 31;
    const int r0 = lane, r1 = lane + 32;
    const unsigned below = (1u << lane) - 1u;
    double x0 = 0.0, x1 = 0.0;
    int k = *lastk_io, nf = 0, iters = 0, mode = 0;
    // warm start: the previous passive set, pruned until its unconstrained
    // solution is positive
    bool warm = k > 0, dual_stale = true;
    unsigned long long rejected = 0ull;  // free columns (positions in fc) refused since the last change of P
    #pragma unroll 1
    for (int outer = warm ? -1 : 0;; ++outer) {
        if (!warm) {
            if (outer > 4 * max_iter) { mode = 1; break; }
            // dual w_j = f_j - sum_r G[j, P_r] x_{P_r} on the free columns j: in
            // column order, so that up to 32 of them take one round of lanes
            if (dual_stale) {
                const int p0 = r0 < k ? g.P[r0] : -1, p1 = r1 < k ? g.P[r1] : -1;
                unsigned in0 = 0u, in1 = 0u;  // passive columns 0-31, 32-63
                if (p0 >= 0) { if (p0 < 32) in0 = 1u << p0; else in1 = 1u << (p0 - 32); }
                if (p1 >= 0) { if (p1 < 32) in0 |= 1u << p1; else in1 |= 1u << (p1 - 32); }
                in0 = __reduce_or_sync(FULL, in0);
                in1 = __reduce_or_sync(FULL, in1);
                const unsigned b0 = ~in0 & (n >= 32 ? ~0u : (1u << n) - 1u), b1 = n > 32 ? ~in1 & (~0u >> (64 - n)) : 0u;
                if (b0 >> lane & 1u) fc[__popc(b0 & below)] = r0;
                if (b1 >> lane & 1u) fc[__popc(b0) + __popc(b1 & below)] = r1;
                nf = __popc(b0) + __popc(b1);
                if (r0 < k) g.xp[r0] = x0;
                if (r1 < k) g.xp[r1] = x1;
                __syncwarp();
                #pragma unroll 1
                for (int i = lane; i < nf; i += 32) {
                    const int j = fc[i];
                    double s = g.f[j], s2 = 0.0;
                    int r = 0;
                    #pragma unroll 1
                    for (; r + 1 < k; r += 2) {
                        s = fma(-g.G[gidx(j, g.P[r])], g.xp[r], s);
                        s2 = fma(-g.G[gidx(j, g.P[r + 1])], g.xp[r + 1], s2);
                    }
                    if (r < k) s = fma(-g.G[gidx(j, g.P[r])], g.xp[r], s);
                    wv[i] = s + s2;
                }
                __syncwarp();
                dual_stale = false;
            }
            if (k >= n) break;
            // entering column: largest positive dual among the unrefused ones, first column on ties
            unsigned long long best = 0;
            int bi = 0;
            #pragma unroll 1
            for (int i = lane; i < nf; i += 32) {
                const double w = wv[i];
                const unsigned long long key = (unsigned long long)__double_as_longlong(w);
                if (pos_bits(w) && !(rejected >> i & 1ull) && key > best) { best = key; bi = i; }
            }
            best = warp_bitsmax(best, bi);
            if (best == 0) break;
            if (!gram_append(g, k, fc[bi], mu2)) {
                rejected |= 1ull << bi;
                continue;
            }
            if (r0 == k) x0 = 0.0;
            if (r1 == k) x1 = 0.0;
            k += 1;
            rejected = 0ull;
        }
        // move toward the unconstrained solution on P (a warm start: drop the
        // columns whose coefficients in it are not positive)
        bool factored = !warm;
        #pragma unroll 1
        for (;;) {
            if (!factored && !gram_refactor(g, k, mu2)) { k = 0; break; }  // numerically dependent: from the empty set
            const double2 zz = gram_back(g, k);
            const double z0 = zz.x, z1 = zz.y;
            const bool pos0 = !(r0 < k) || pos_bits(z0), pos1 = !(r1 < k) || pos_bits(z1);
            if (__all_sync(FULL, pos0 && pos1)) { x0 = z0; x1 = z1; break; }
            double nx0 = z0, nx1 = z1;
            if (!warm) {
                if (++iters > max_iter) { mode = 1; break; }
                // alpha = min over z_r <= 0 of x_r / (x_r - z_r), first row on ties (bit
                // patterns of non-negative values order like the values)
                double a0 = CUDART_INF, a1 = CUDART_INF;
                if (!pos0) { const double dz = x0 - z0; a0 = pos_bits(dz) ? x0 * fast_rcp(dz) : 0.0; }
                if (!pos1) { const double dz = x1 - z1; a1 = pos_bits(dz) ? x1 * fast_rcp(dz) : 0.0; }
                unsigned long long ka = (unsigned long long)__double_as_longlong(a0);
                const unsigned long long ka1 = (unsigned long long)__double_as_longlong(a1);
                int ia = r0;
                if (ka1 < ka) { ka = ka1; ia = r1; }
                const double alpha = __longlong_as_double((long long)warp_bitsmin(ka, ia));
                nx0 = r0 == ia ? 0.0 : fma(alpha, z0 - x0, x0);
                nx1 = r1 == ia ? 0.0 : fma(alpha, z1 - x1, x1);
            }
            const bool keep0 = r0 < k && pos_bits(nx0), keep1 = r1 < k && pos_bits(nx1);
            const unsigned m0 = __ballot_sync(FULL, keep0), m1 = __ballot_sync(FULL, keep1);
            const int p0 = r0 < k ? g.P[r0] : 0, p1 = r1 < k ? g.P[r1] : 0;
            __syncwarp();
            if (keep0) { const int d = __popc(m0 & below); g.P[d] = p0; g.xp[d] = nx0; }
            if (keep1) { const int d = __popc(m0) + __popc(m1 & below); g.P[d] = p1; g.xp[d] = nx1; }
            k = __popc(m0) + __popc(m1);
            __syncwarp();
            if (r0 < k) x0 = g.xp[r0];
            if (r1 < k) x1 = g.xp[r1];
            __syncwarp();
            factored = false;
        }
        if (mode) break;
        warm = false;
        dual_stale = true;
    }

    *lastk_io = k;
    #pragma unroll 1
    for (int j = lane; j < n; j += 32) x[j] = 0.0;
    __syncwarp();
    // ||A x - b||^2 = b'b - f'x - mu^2 ||x||^2 at the solution ((G + mu^2 I)_PP x_P
    // = f_P); the cancellation costs ~eps * b'b, far below the noise floor
    double fx = 0.0, xx = 0.0;
    if (r0 < k) { const int p = g.P[r0]; x[p] = x0; fx = fma(g.f[p], x0, 0.0); xx = x0 * x0; }
    double xs = xx;
    if (r1 < k) { const int p = g.P[r1]; x[p] = x1; fx = fma(g.f[p], x1, fx); xx = fma(x1, x1, xx); xs = xs + x1 * x1; }
    wsum2(fx, xx, fx, xx);  // the same pairings as wsum, both sums in one butterfly
    const double res = fmax(g.bb - fx - mu2 * xx, 0.0);
    NnlsResult out;
    out.nsetp = k;
    out.mode = mode;
    out.rnorm = sqrt(fma(mu2, xx, res));
    out.xx = k <= 32 ? xx : wsum(xs);  // (one term per lane: the same sum)
    __syncwarp();
    return out;
}

}  // namespace dk
