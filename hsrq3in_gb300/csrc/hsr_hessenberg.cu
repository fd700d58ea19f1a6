// hsr_hessenberg.cu -- reduction of a dense matrix to upper-Hessenberg form
// on the device, and application of its orthogonal factor.
//
// The input step of the solver: the reference's problem generator reduces
// Q T Q^T with LAPACK dgehrd (problemgenerator.c:344), and dense requests
// need the same reduction before inverse iteration.  The layout and the
// reflector convention are LAPACK's (dgehd2 with dlarfg and dlarf): on exit
// the upper-Hessenberg part of A holds H, the entries below the subdiagonal
// of column k hold v_k(k+2 : n-1) with v_k(k+1) = 1 implied, and
// A_in = Q H Q^T with Q = H_0 H_1 ... H_{n-3}, H_k = I - tau_k v_k v_k^T.
//
// Blocked as LAPACK dgehrd/dlahr2 do it, in panels of kHbNb reflectors.  For
// a panel starting at column k0, Q_p = H_k0 ... H_{k0+nb-1} = I - V T V^T
// (compact WY, T upper triangular) and Y = A V T over the panel-start A.
// Column j = k0 + i of the panel is first brought up to date with the
// panel's earlier reflectors, a_j - Y V(j,:)^T from the right and
// (I - V T^T V^T) from the left; then its reflector is generated, and
// Y(:, i) = tau (A v - Y (V^T v)), T(:, i) = -tau T (V^T v), T(i,i) = tau.
// All columns of a panel run in one cooperative launch (k_hb_panel); only
// where the rows do not fit its shared memory (n above about 25,000), or the
// device refuses such a launch, three launches per column do the same:
//   k_hb_step    rows in parallel: finishes the previous column (Y, V and T
//                columns, its reflector into A) and starts this one,
//                c = a_j - Y V(j,:)^T, with partial V^T c; the last block to
//                finish reduces them and forms w' = T^T V^T c
//   k_hb_larfg   rows in parallel: c -= V w' (rows > k0), the H entries of
//                column j, partial three-accumulator norms; the last block
//                runs dlarfg (with its safe-minimum rescaling)
//   k_hb_gemv    A(:, j+1 : n-1) v in column chunks, and partial V^T v
// After the panel the trailing columns c1 = k0 + nb ... get both sides of
// the block reflector: in one rank-128 product by digits on the tensor cores
// (hb_trailing), or with FP64 GEMMs (k_hb_plain, DFMA, 64x64 tiles):
//   A(:, c1:) -= Y V(c1:, :)^T;  W = T^T V^T A(k0+1:, c1:);  A(k0+1:, c1:) -= V W
// Digits and fixed point hold an entry by a window below the largest one of its
// row or column, FP64 by 53 bits of its own.  They are for matrices whose
// entries are of like size (k_hb_even decides, on the device); where rows or
// columns differ, the reduction in FP64 keeps the small ones accurate, and it
// runs in FP64 throughout.
// The "last block" reductions use a completion counter and a fixed summation
// order: no block waits for another, and results are reproducible run to run.
#include "../../include/hsrq3in_gb300.h"
#include "hsr_device.cuh"
#include "hsr_digits.cuh"
#include "hsr_scratch.h"

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <cuda_runtime.h>
#include <type_traits>

namespace hsr {
namespace {


__device__ __forceinline__ double block_sum3(double v, double *red) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < nw; ++i) t += red[i];   // fixed order, every thread
    return t;
}

// dlapy2 (LAPACK >= 3.10): sqrt(x^2 + y^2) without overflow; NaN propagates.
__device__ __forceinline__ double lapy2(double x, double y) {
    if (x != x) return x;
    if (y != y) return y;
    const double xa = fabs(x), ya = fabs(y);
    const double w = fmax(xa, ya), z = fmin(xa, ya);
    if (z == 0.0 || w > DBL_MAX) return w;
    const double q = z / w;
    return w * sqrt(1.0 + q * q);
}


constexpr int kHbNb = 64;         // reflectors per panel
constexpr int kHbRows = 256;      // rows per CTA of the row-parallel kernels
constexpr int kHbChunk = 64;      // columns per CTA of the panel GEMV
constexpr int kHbMaxSplit = 8;    // split-K factor of the thin left-update GEMM

// Device state of one reduction.  Y, V: n x kHbNb (leading dimension n);
// T: kHbNb x kHbNb; c: the working column; part / part2: per-block partial
// sums [nblk][kHbNb]; partn: per-block norm accumulators [nblk][3]; gpart:
// GEMV partials [nchunk][n]; sc[0 .. kHbNb): w', sc[kHbNb]: the reflector's
// scale 1/(alpha - beta), sc[kHbNb+1]: tau; cnt: completion counters.
struct HbState {
    double *A;
    long long lda;
    int n;
    double *Y, *V, *T, *c, *part, *part2, *partn, *gpart, *sc, *tau;
    unsigned int *cnt;
};

// True in the block that finished last; its partial sums see every other
// block's (threadfence before the count).
__device__ __forceinline__ bool last_block(unsigned int *counter) {
    __shared__ bool am_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) am_last = atomicAdd(counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (am_last) __threadfence();
    return am_last;
}

// Sum over the 256 rows of a block of V(r, q) * cs[r - r0] for q < i, a warp
// per q; writes out[q].
__device__ __forceinline__ void block_vdot(const HbState &S, int r0, int i, const double *cs, double *out) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int q = warp; q < i; q += kHbRows / 32) {
        double s = 0.0;
        for (int t = lane; t < kHbRows; t += 32) {
            const int r = r0 + t;
            if (r < S.n) s = fma(S.V[r + (size_t)q * S.n], cs[t], s);
        }
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) out[q] = s;
    }
}

// v(r) of the current reflector: 1 at j+1, c(r) * rs below, 0 above.
__device__ __forceinline__ double hb_v(const HbState &S, int j, double rs, int r) {
    return r == j + 1 ? 1.0 : (r >= j + 2 ? S.c[r] * rs : 0.0);
}

// Sum_{q < m} x[q * stride] * w[q] in four interleaved fma chains, combined
// in a fixed order (independent chains hide the FP64 latency).
__device__ __forceinline__ double dot4(const double *x, long long stride, const double *w, int m) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int q = 0;
    for (; q + 3 < m; q += 4) {
        s0 = fma(x[(size_t)q * stride], w[q], s0);
        s1 = fma(x[(size_t)(q + 1) * stride], w[q + 1], s1);
        s2 = fma(x[(size_t)(q + 2) * stride], w[q + 2], s2);
        s3 = fma(x[(size_t)(q + 3) * stride], w[q + 3], s3);
    }
    for (; q < m; ++q) s0 = fma(x[(size_t)q * stride], w[q], s0);
    return (s0 + s1) + (s2 + s3);
}

// The same with eight chains, for the panel GEMV: eight independent loads in
// flight per thread.
__device__ __forceinline__ double dot8(const double *x, long long stride, const double *w, int m) {
    double s[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    int q = 0;
    for (; q + 7 < m; q += 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) s[u] = fma(x[(size_t)(q + u) * stride], w[q + u], s[u]);
    }
    for (; q < m; ++q) s[0] = fma(x[(size_t)q * stride], w[q], s[0]);
    return ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
}

// Sum of m partials p[ch * stride], four chains in a fixed order.
__device__ __forceinline__ double sum4(const double *p, long long stride, int m) {
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int q = 0;
    for (; q + 3 < m; q += 4) {
        s0 += p[(size_t)q * stride];
        s1 += p[(size_t)(q + 1) * stride];
        s2 += p[(size_t)(q + 2) * stride];
        s3 += p[(size_t)(q + 3) * stride];
    }
    for (; q < m; ++q) s0 += p[(size_t)q * stride];
    return (s0 + s1) + (s2 + s3);
}

// T(0:ip, ip) = -tau T(0:ip, 0:ip) vv, T(ip, ip) = tau, by one block.
__device__ __forceinline__ void hb_tcol(const HbState &S, int ip, double t, const double *vv) {
    for (int p = threadIdx.x; p < ip; p += blockDim.x) {
        double s = 0.0;
        for (int q = p; q < ip; ++q) s = fma(S.T[p + (size_t)q * kHbNb], vv[q], s);
        S.T[p + (size_t)ip * kHbNb] = -t * s;
    }
    if (threadIdx.x == 0) S.T[ip + (size_t)ip * kHbNb] = t;
}

// One launch between two reflectors.  Phase A (ip >= 0) finishes column
// jp = k0 + ip: Y(:, ip) = tau (A v - Y (V^T v)), V(:, ip), the reflector
// into A, T(:, ip).  Phase B (i >= 0) starts column j = k0 + i: c = a_j -
// Y V(j,:)^T and the partial sums of V^T c, reduced by the last block into
// w' = T^T V^T c.  Row r of both phases is one thread's, so phase B reads the
// Y(r, ip) that phase A just wrote; V(j, ip) = v_jp(jp + 1) is 1.
__global__ void __launch_bounds__(kHbRows) k_hb_step(HbState S, int k0, int ip, int i, int nchp) {
    __shared__ double vv[kHbNb], vrow[kHbNb], cs[kHbRows], ws[kHbNb];
    const int tid = threadIdx.x, r0 = blockIdx.x * kHbRows, r = r0 + tid, n = S.n;
    const int nblk = gridDim.x;
    if (ip >= 0) {
        const int jp = k0 + ip;
        for (int q = tid; q < ip; q += blockDim.x) {
            double s = 0.0;
            for (int b = 0; b < nblk; ++b) s += S.part2[(size_t)b * kHbNb + q];
            vv[q] = s;
        }
        __syncthreads();
        const double t = S.sc[kHbNb + 1], rs = S.sc[kHbNb];
        if (r < n) {
            const double av = sum4(S.gpart + r, n, nchp);
            const double y = av - dot4(S.Y + r, n, vv, ip);
            S.Y[r + (size_t)ip * n] = t * y;
            if (r >= jp + 1) {
                const double v = hb_v(S, jp, rs, r);
                S.V[r + (size_t)ip * n] = v;
                if (r >= jp + 2) S.A[r + (size_t)jp * S.lda] = v;
            }
        }
        if (i < 0) {
            if (blockIdx.x == 0) hb_tcol(S, ip, t, vv);
            return;
        }
    }
    const int j = k0 + i;
    for (int q = tid; q < i; q += blockDim.x) vrow[q] = (q == i - 1) ? 1.0 : S.V[j + (size_t)q * n];
    __syncthreads();
    double x = 0.0;
    if (r < n) {
        x = S.A[r + (size_t)j * S.lda] - dot4(S.Y + r, n, vrow, i);
        S.c[r] = x;
    }
    if (i == 0) return;
    cs[tid] = (r < n && r >= k0 + 1) ? x : 0.0;
    __syncthreads();
    block_vdot(S, r0, i, cs, S.part + (size_t)blockIdx.x * kHbNb);
    if (!last_block(&S.cnt[0])) return;
    hb_tcol(S, ip, S.sc[kHbNb + 1], vv);
    __syncthreads();
    for (int q = tid; q < i; q += blockDim.x) {
        double w = 0.0;
        for (int b = 0; b < nblk; ++b) w += S.part[(size_t)b * kHbNb + q];
        ws[q] = w;
    }
    __syncthreads();
    for (int p = tid; p < i; p += blockDim.x) {            // (T^T w)_p = sum_{q <= p} T(q, p) w_q
        double t = 0.0;
        for (int q = 0; q <= p; ++q) t = fma(S.T[q + (size_t)p * kHbNb], ws[q], t);
        S.sc[p] = t;
    }
    if (tid == 0) S.cnt[0] = 0;
}

__global__ void __launch_bounds__(kHbRows) k_hb_larfg(HbState S, int k0, int i, int j) {
    __shared__ double red[32];
    const int tid = threadIdx.x, r = blockIdx.x * kHbRows + tid, n = S.n;
    double x = 0.0;
    if (r < n) {
        x = S.c[r];
        if (r >= k0 + 1 && i > 0) {
            x = x - dot4(S.V + r, n, S.sc, i);
            S.c[r] = x;
        }
        if (r <= j) S.A[r + (size_t)j * S.lda] = x;          // final entries of H above the subdiagonal
    }
    Nrm3 acc;
    acc.init();
    if (r < n && r >= j + 2) acc.add(x);
    const double a0 = block_sum3(acc.asml, red), a1 = block_sum3(acc.amed, red), a2 = block_sum3(acc.abig, red);
    if (tid == 0) {
        S.partn[(size_t)blockIdx.x * 3] = a0;
        S.partn[(size_t)blockIdx.x * 3 + 1] = a1;
        S.partn[(size_t)blockIdx.x * 3 + 2] = a2;
    }
    if (!last_block(&S.cnt[1])) return;
    // dlarfg on alpha = c(j+1), x = c(j+2 : n-1), as the reference's LAPACK.
    double *xv = S.c + (j + 2);
    const int nx = n - j - 2;
    Nrm3 tot;
    tot.init();
    for (int b = 0; b < (int)gridDim.x; ++b) {
        tot.asml += S.partn[(size_t)b * 3];
        tot.amed += S.partn[(size_t)b * 3 + 1];
        tot.abig += S.partn[(size_t)b * 3 + 2];
    }
    double xnorm = tot.finish();
    double alpha = S.c[j + 1];
    double t = 0.0, rs = 1.0, beta = alpha;
    if (xnorm != 0.0) {
        const double safmin = 0x1p-969;                        // dlamch('S') / dlamch('E')
        const double rsafmn = 0x1p+969;
        beta = -copysign(lapy2(alpha, xnorm), alpha);
        int knt = 0;
        if (fabs(beta) < safmin) {
            do {
                ++knt;
                __syncthreads();
                for (int q = tid; q < nx; q += blockDim.x) xv[q] = xv[q] * rsafmn;
                beta = beta * rsafmn;
                alpha = alpha * rsafmn;
            } while (fabs(beta) < safmin && knt < 20);
            __syncthreads();
            Nrm3 a;
            a.init();
            for (int q = tid; q < nx; q += blockDim.x) a.add(xv[q]);
            Nrm3 s2;
            s2.asml = block_sum3(a.asml, red);
            s2.amed = block_sum3(a.amed, red);
            s2.abig = block_sum3(a.abig, red);
            xnorm = s2.finish();
            beta = -copysign(lapy2(alpha, xnorm), alpha);
        }
        t = (beta - alpha) / beta;
        rs = 1.0 / (alpha - beta);
        for (int q = 0; q < knt; ++q) beta = beta * safmin;
    }
    if (tid == 0) {
        S.tau[j] = t;
        S.A[(j + 1) + (size_t)j * S.lda] = beta;
        S.sc[kHbNb] = rs;
        S.sc[kHbNb + 1] = t;
        S.cnt[1] = 0;
    }
}

__global__ void __launch_bounds__(kHbRows) k_hb_gemv(HbState S, int k0, int i, int j) {
    __shared__ double vs[kHbChunk], cs[kHbRows];
    const int tid = threadIdx.x, n = S.n;
    const double rs = S.sc[kHbNb];
    const int c0 = j + 1 + blockIdx.y * kHbChunk, c1 = min(n, c0 + kHbChunk);
    for (int t = tid; t < c1 - c0; t += blockDim.x) vs[t] = hb_v(S, j, rs, c0 + t);
    __syncthreads();
    const int r0 = blockIdx.x * kHbRows, r = r0 + tid;
    if (r < n) S.gpart[(size_t)blockIdx.y * n + r] = dot8(S.A + r + (size_t)c0 * S.lda, S.lda, vs, c1 - c0);
    if (blockIdx.y != 0 || i == 0) return;
    cs[tid] = r < n ? hb_v(S, j, rs, r) : 0.0;
    __syncthreads();
    block_vdot(S, r0, i, cs, S.part2 + (size_t)blockIdx.x * kHbNb);
}

// --------------------------------------------------- panel in one launch
// The same column steps as the three kernels above, for all columns of a
// panel in one cooperative launch.  The first CTAs own R rows each for the
// vector work and keep their rows of Y and V, and a copy of T, in shared
// memory; a sum over all rows is left in global memory as one partial per
// CTA, and after a grid barrier every CTA that needs it adds all of them up
// in the same order.  Three barriers a column: after the partial V^T c (CTAs
// with rows only), after the partial norms, and after A v.  All CTAs share
// A v, a row tile of rpc rows and a share of the columns each.  T's new
// column is formed while a barrier is awaited, the next column and the first
// entries of A for A v are loaded ahead of one.
//
// Bound for small orders by the L2 round trips of the barriers and sums and
// by FP64 issue (a warp's instruction takes 64 clocks of its sub-partition):
// 35,000 clocks a column at n = 700, of which A v 4,000; for large ones by the
// memory in A v (fixed point, below; with FMAs by the FP64 pipe).  Against the
// three launches a column on n / 256 CTAs: n = 700 39.4 ms before, 13.4 now;
// n = 6000 691 and 316; n = 10 354 us and 225.
constexpr int kHbThreads = 512;
constexpr int kHbPiece = 1024;         // columns of v staged at a time (two per thread)
constexpr int kHbAhead = 8;            // entries of A per thread loaded before v is known
constexpr int kHbPanelSmem = 220 * 1024;
constexpr unsigned kHbSpin = 1u << 23; // polls of a barrier before it gives up and says so
constexpr unsigned kHbDead = 1u << 30; // ... by this bit of both counters

struct HbPanel {
    HbState S;
    int k0, ib, R, own;                // CTAs 0 .. own-1 have rows, R each
    int rpc, tiles, shares;            // A v: row tiles of rpc rows, CTAs (column shares) per tile
    unsigned *bar;                     // arrivals since the reduction began: of all CTAs, of those with rows
    const int2 *F;                     // A's columns k0+1 .. in fixed point, n entries each (kFix)
    const unsigned *top;               // their rows' largest high words, sign off (kFix)
    const int *uneven;                 // k_hb_panel<true> runs where it is 0, <false> where it is not (null: runs)
};
__host__ __device__ constexpr int hb_pitch(int R) { return R | 1; }     // odd: columns fall on different banks
__host__ __device__ constexpr size_t hb_panel_smem(int R) {
    return sizeof(double) * ((size_t)2 * kHbNb * hb_pitch(R) + kHbNb * (kHbNb + 1) + 2 * (size_t)R + 4 * kHbNb +
                             2 * kHbThreads + kHbPiece + 16);
}
// Sum of x over the lanes of an aligned group of g (a power of two), in every lane.
__device__ __forceinline__ double group_sum(double x, int g) {
    for (int o = g >> 1; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// A v on the integer pipe.  The FP64 pipe gives two products a clock and SM,
// 16 bytes of A, where the memory gives 24; so for large n the panel first
// puts A's remaining columns into fixed point, 58 bits below the largest
// entry of the row (v, at most 1, likewise: 58 bits below 1), as a high part
// of 29 bits and a signed low part of 30 in eight bytes, what the double took.
// A product is then four 32 x 32 -> 64 bit ones, exact, in three sums:
// high x high (2^56 at most, turned to FP64 every 64), high x low and low x
// high, low x low (2^58 at most, carried up every 16).  So the entries are
// rounded once, to 2^-59 of their row's largest, and the sum over 64 columns
// once, where the FMAs round at every column.
//
// Then the memory bounds A v (6.3 TB/s of A).  The two passes that make the
// copy cost 24 bytes of traffic an entry once in 64 products.  n = 6000: a
// panel's column 70 us at the start and 24 at the end, the reduction 380 ->
// 316 ms; n = 3000 94 -> 87.  At n = 2000 both take 52.5 ms (the matrix lies
// in L2, and the steps around A v are most of a column); below, the copy costs
// more than it gives (n = 1000 19.9 -> 21.0).
constexpr int kHbFixN = 2048;
constexpr int kFixLow = 30, kFixBits = 58;
// x 2^58 / 2^e to the nearest, for |x| < 2^e or a little above; parts as above.
__device__ __forceinline__ int2 fix_parts(double x, int e) {
    const unsigned long long u = ubits(x);
    const int f = (int)(u >> 52) & 0x7ff;
    const unsigned long long m = ((u & 0xfffffffffffffULL) | (f ? 0x10000000000000ULL : 0ULL)) << 10;
    const int sh = min(62 - kFixBits - (max(f, 1) - 1023 - e), 63);          // m = |x| 2^(62 - exponent)
    long long q = (long long)((m + (1ULL << (sh - 1))) >> sh);
    q = u >> 63 ? -q : q;
    const long long hi = (q + (1LL << (kFixLow - 1))) >> kFixLow;
    return make_int2((int)hi, (int)(q - (hi << kFixLow)));
}
// The exponent e of fix_parts for a row whose largest high word is `top`.
__device__ __forceinline__ int fix_exp(unsigned top) { return max((int)(top >> 20), 1) - 1022; }
struct FixSum {
    double s = 0.0;
    long long hh = 0, hl = 0, ll = 0;
    __device__ __forceinline__ void add(int2 a, int2 v) {
        hh += (long long)a.x * v.x;
        hl += (long long)a.x * v.y;
        hl += (long long)a.y * v.x;
        ll += (long long)a.y * v.y;
    }
    __device__ __forceinline__ void carry() {                    // after at most 16 products
        constexpr long long mask = (1LL << kFixLow) - 1;
        hl += ll >> kFixLow;
        ll &= mask;
        hh += hl >> kFixLow;
        hl &= mask;
    }
    __device__ __forceinline__ void flush() {                    // after at most 64
        s += (double)hh;
        hh = 0;
    }
    // The sum, over 2^(e - 56).
    __device__ __forceinline__ double value() {
        carry();
        flush();
        return fma((double)(int)hl, 0x1p-30, s);
    }
};
// Largest high word of each row over the columns k0+1 .. n-1.
constexpr int kFixCols = 64;
__global__ void __launch_bounds__(256) k_hb_fix_top(int n, const double *A, long long lda, int c0, unsigned *top,
                                                    const int *uneven) {
    if (dg_off(uneven)) return;
    const int r = blockIdx.x * 256 + threadIdx.x, ca = c0 + blockIdx.y * kFixCols, ce = min(ca + kFixCols, n);
    if (r >= n) return;
    unsigned m = 0;
#pragma unroll 16
    for (int c = ca; c < ce; ++c) m = max(m, (unsigned)(ubits(A[r + (size_t)c * lda]) >> 32) & 0x7fffffffu);
    atomicMax(top + r, m);
}
__global__ void __launch_bounds__(256) k_hb_fix(int n, const double *A, long long lda, int c0, const unsigned *top, int2 *F,
                                                const int *uneven) {
    if (dg_off(uneven)) return;
    const int r = blockIdx.x * 256 + threadIdx.x, ca = c0 + blockIdx.y * kFixCols, ce = min(ca + kFixCols, n);
    if (r >= n) return;
    const int e = fix_exp(top[r]);
#pragma unroll 8
    for (int c = ca; c < ce; ++c) F[r + (size_t)(c - c0) * n] = fix_parts(A[r + (size_t)c * lda], e);
}

template <bool kFix>
__global__ void __launch_bounds__(kHbThreads, 1) k_hb_panel(HbPanel P) {
    extern __shared__ double hsm[];
    __shared__ int dead;
    if (P.uneven && (*P.uneven != 0) == kFix) return;            // uniform over the grid, ahead of every barrier
    const HbState &S = P.S;
    const int tid = threadIdx.x, n = S.n, k0 = P.k0, R = P.R, Rp = hb_pitch(R), G = gridDim.x, b = blockIdx.x;
    double *const Ys = hsm, *const Vs = Ys + kHbNb * Rp, *const Ts = Vs + kHbNb * Rp;      // T(p, q) at p + 65 q
    double *const cs = Ts + kHbNb * (kHbNb + 1), *const aj = cs + R, *const vv = aj + R, *const wv = vv + kHbNb;
    double *const w2 = wv + kHbNb, *const vrow = w2 + kHbNb, *const red = vrow + kHbNb, *const gred = red + kHbThreads;
    double *const vst = gred + kHbThreads, *const sc = vst + kHbPiece;
    const int rt = b / P.shares, share = b - rt * P.shares;      // place in A v
    const bool has = b < P.own;
    const int r0 = min(b * R, n), nr = has ? min(R, n - r0) : 0; // own rows
    const int rlo = min(max(k0 + 1 - r0, 0), nr);                // first own row that the reflectors touch
    // A warp's FP64 instruction takes 64 clocks of its sub-partition whether
    // one lane or all are at work, so the dots below use the fewest warps that
    // fill four of them, and warps without work stay out.
    int tpr = 1;                                                 // threads per row
    while (tpr < 32 && R * tpr * 2 <= 128) tpr *= 2;
    const int rgrp = kHbThreads / tpr, rs = tid & (tpr - 1), rofs = tid / tpr, wofs = (tid & ~31) / tpr;

    unsigned target[2] = {0, 0};
    if (tid == 0) {
        // Arrivals of this launch cannot complete a round before this CTA's own.
        target[0] = (*reinterpret_cast<volatile unsigned *>(P.bar) & ~kHbDead) / G * G;
        target[1] = (*reinterpret_cast<volatile unsigned *>(P.bar + 1) & ~kHbDead) / P.own * P.own;
        dead = 0;
    }
    auto arrive = [&](int which) {                               // 0: all CTAs, 1: those with rows
        __syncthreads();
        if (tid == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(P.bar + which) : "memory");
            target[which] += which ? P.own : G;
        }
    };
    auto wait = [&](int which) {                                 // false once a barrier gave up
        if (tid == 0) {
            unsigned it = 0, v;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(P.bar + which) : "memory");
            } while (!(v & kHbDead) && (int)(v - target[which]) < 0 && ++it < kHbSpin);
            if (it >= kHbSpin) {
                atomicOr(P.bar, kHbDead);
                atomicOr(P.bar + 1, kHbDead);
            }
            if (it >= kHbSpin || (v & kHbDead)) dead = 1;
        }
        __syncthreads();
        return dead == 0;
    };
    // out[q] = f * sum over the CTAs of part[c][q], q < cnt, in a fixed order:
    // four or (many CTAs) eight threads per q, up to 13 loads of each in
    // flight at a time.
    auto reduce_parts = [&](const double *part, int cnt, double *out, double f) {
        const int lq = cnt <= 32 ? 5 : 6, q = tid & ((1 << lq) - 1), s = tid >> lq, ns = P.own > 52 ? 8 : 4;
        if (s < ns) {
            double a = 0.0;
            if (q < cnt) {
                for (int c = s; c < P.own; c += 13 * ns) {
                    double x[13];
#pragma unroll
                    for (int e = 0; e < 13; ++e) x[e] = c + e * ns < P.own ? __ldcg(part + (size_t)(c + e * ns) * kHbNb + q) : 0.0;
#pragma unroll
                    for (int e = 0; e < 13; ++e)
                        if (c + e * ns < P.own) a += x[e];       // uniform over the warp
                }
            }
            red[tid] = a;
        }
        __syncthreads();
        if (tid < cnt) {
            double u = (red[tid] + red[tid + (1 << lq)]) + (red[tid + (2 << lq)] + red[tid + (3 << lq)]);
            if (ns == 8) u += (red[tid + (4 << lq)] + red[tid + (5 << lq)]) + (red[tid + (6 << lq)] + red[tid + (7 << lq)]);
            out[tid] = f * u;
        }
        __syncthreads();
    };
    // Threads per column for `cnt` column dots: as with the rows.
    auto per_col = [&](int cnt) { return cnt <= 16 ? 8 : cnt <= 32 ? 4 : 2; };
    // part[b][q] = sum over own rows of V(r, q) x(r), q < cnt.
    auto col_dots = [&](const double *x, int cnt, double *part) {
        const int tq = per_col(cnt), q = tid / tq, s = tid & (tq - 1);
        if ((tid & ~31) / tq >= cnt) return;
        double a = 0.0;
        if (q < cnt)
            for (int r = rlo + s; r < nr; r += tq) a = fma(Vs[q * Rp + r], x[r], a);
        a = group_sum(a, tq);
        if (s == 0 && q < cnt) __stcg(part + (size_t)b * kHbNb + q, a);
    };
    // Norm accumulators of c(j+2 :): this CTA's rows to partn, later all CTAs'.
    auto norms_out = [&](int j, double *out) {
        Nrm3 acc;
        acc.init();
        for (int r = tid; r < nr; r += kHbThreads)
            if (r0 + r >= j + 2) acc.add(cs[r]);
        const int warps = min(kHbThreads / 32, (nr + 31) / 32), w = tid >> 5;
        const bool ends = __syncthreads_or(acc.asml != 0.0 || acc.abig != 0.0);
        if (w < warps) {
            const double m = group_sum(acc.amed, 32);
            if ((tid & 31) == 0) red[w] = m;
            if (ends) {
                const double lo = group_sum(acc.asml, 32), hi = group_sum(acc.abig, 32);
                if ((tid & 31) == 0) {
                    red[32 + w] = lo;
                    red[64 + w] = hi;
                }
            }
        }
        __syncthreads();
        if (tid < 3) {                                           // asml, amed, abig
            double u = 0.0;
            const int at = tid == 0 ? 32 : tid == 1 ? 0 : 64;
            if (tid == 1 || ends)
                for (int z = 0; z < warps; ++z) u += red[at + z];
            __stcg(out + (size_t)b * 3 + tid, u);
        }
    };
    // xnorm (or, as good a test for 0, its square) to sc[0], alpha to sc[1],
    // beta to sc[2], 1 / (alpha - beta) to sc[4].  With all of c(j+1 :) in the middle range beta is one
    // square root of the sum of squares.  `again`: after the rescaling, whose
    // caller needs xnorm itself and has an alpha that is not the stored one.
    auto norms_in = [&](int j, const double *in, bool again) {
        if (tid < 32) {
            double x[3][5];
            Nrm3 tot;
            tot.init();
            const double alpha = __ldcg(S.c + j + 1);
            for (int c = tid; c < P.own; c += 160) {
#pragma unroll
                for (int e = 0; e < 5; ++e)
#pragma unroll
                    for (int k = 0; k < 3; ++k) x[k][e] = c + 32 * e < P.own ? __ldcg(in + (size_t)(c + 32 * e) * 3 + k) : 0.0;
#pragma unroll
                for (int e = 0; e < 5; ++e)
                    if ((c & ~31) + 32 * e < P.own) tot.amed += x[1][e];
#pragma unroll
                for (int e = 0; e < 5; ++e) {
                    if (mag(x[0][e]) != 0) tot.asml = add_rare(tot.asml, x[0][e]);
                    if (mag(x[2][e]) != 0) tot.abig = add_rare(tot.abig, x[2][e]);
                }
            }
            const bool ends = __any_sync(0xffffffffu, mag(tot.asml) != 0 || mag(tot.abig) != 0);
            tot.amed = group_sum(tot.amed, 32);
            if (ends) {
                tot.asml = group_sum(tot.asml, 32);
                tot.abig = group_sum(tot.abig, 32);
            }
            if (tid == 0) {
                const unsigned long long ma = mag(alpha);
                double xn = tot.amed, beta = alpha;
                if (!again && !ends && (ma == 0 || (ma > pow2_bits(-500) && ma < pow2_bits(486))) && mag(xn) > pow2_bits(-900)) {
                    beta = sqrt(fma(alpha, alpha, xn));
                    beta = ubits(alpha) >> 63 ? beta : neg(beta);
                } else {
                    xn = tot.finish();
                    if (xn != 0.0) beta = -copysign(lapy2(alpha, xn), alpha);
                }
                sc[0] = xn;
                sc[1] = alpha;
                sc[2] = beta;
                sc[4] = xn != 0.0 ? 1.0 / (alpha - beta) : 1.0;
            }
        }
        __syncthreads();
    };
    // T(0 : ip, ip) = -tau T vv, T(ip, ip) = tau, in shared memory (vv holds -V^T v).
    auto t_column = [&](int ip, double t) {
        const int tq = per_col(ip + 1), p = tid / tq, s = tid & (tq - 1);
        if ((tid & ~31) / tq > ip) return;
        double a = 0.0;
        for (int q = p + s; q < ip; q += tq) a = fma(Ts[p + q * (kHbNb + 1)], vv[q], a);
        a = group_sum(a, tq);
        if (s == 0 && p <= ip) Ts[p + ip * (kHbNb + 1)] = p < ip ? t * a : t;
    };
    // sum_q M(r, q) w[q] over q < cnt for row r, in the row's lanes; `more` is
    // each lane's own part of something to add.
    auto row_dot = [&](const double *M, const double *w, int cnt, int r, double more) {
        double a = more;
        if (r < nr)
            for (int q = rs; q < cnt; q += tpr) a = fma(M[q * Rp + r], w[q], a);
        return group_sum(a, tpr);
    };

    for (int e = tid; e < kHbNb * (kHbNb + 1); e += kHbThreads) Ts[e] = 0.0;
    for (int r = tid; r < nr; r += kHbThreads) aj[r] = S.A[r0 + r + (size_t)k0 * S.lda];
    double t = 0.0;
    bool ok = true;
    __syncthreads();
    for (int i = 0; i <= P.ib; ++i) {
        const int j = k0 + i, ip = i - 1;
        if (i == P.ib && !has) break;
        if (has) {
            if (i > 0) {
                // Y(:, ip) = tau (A v - Y (V^T v)).
                if (tid < i) vrow[tid] = tid == ip ? 1.0 : __ldcg(S.V + j + (size_t)tid * n);
                double g0[4];                                    // the first row's parts, beside the sums' loads
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    g0[e] = rofs < nr && rs + e * tpr < P.shares ? __ldcg(S.gpart + (size_t)(rs + e * tpr) * n + r0 + rofs) : 0.0;
                reduce_parts(S.part2, ip, vv, -1.0);                 // -V^T v
                for (int base = 0; base + wofs < nr; base += rgrp) {
                    const int r = base + rofs;
                    double av = 0.0;
                    if (r < nr) {
                        for (int c = rs; c < P.shares; c += 4 * tpr) {
                            double x[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                x[e] = base == 0 && c == rs      ? g0[e]
                                       : c + e * tpr < P.shares ? __ldcg(S.gpart + (size_t)(c + e * tpr) * n + r0 + r)
                                                                : 0.0;
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (c - rs + e * tpr < P.shares) av += x[e];     // uniform over the warp
                        }
                    }
                    const double y = t * row_dot(Ys, vv, ip, r, av);
                    if (r < nr && rs == 0) {
                        Ys[ip * Rp + r] = y;
                        S.Y[r0 + r + (size_t)ip * n] = y;
                    }
                }
                if (i == P.ib) break;
                __syncthreads();
            }
            // c = a_j - Y V(j, :)^T.
            for (int base = 0; base + wofs < nr; base += rgrp) {
                const int r = base + rofs;
                const double a = row_dot(Ys, vrow, i, r, 0.0);
                if (r < nr && rs == 0) cs[r] = aj[r] - a;
            }
            __syncthreads();
            if (i > 0) {
                // c -= V T^T V^T c.
                col_dots(cs, i, S.part);
                arrive(1);
                t_column(ip, t);
                ok = wait(1);
                if (!ok) break;
                reduce_parts(S.part, i, wv, 1.0);
                {                                                    // T^T of it
                    const int tq = per_col(i), p = tid / tq, s = tid & (tq - 1);
                    if ((tid & ~31) / tq < i) {
                        double a = 0.0;
                        if (p < i)
                            for (int q = s; q <= p; q += tq) a = fma(Ts[q + p * (kHbNb + 1)], wv[q], a);
                        a = group_sum(a, tq);
                        if (s == 0 && p < i) w2[p] = a;
                    }
                }
                __syncthreads();
                for (int base = rlo; base + wofs < nr; base += rgrp) {
                    const int r = base + rofs;
                    const double a = row_dot(Vs, w2, i, r, 0.0);
                    if (r < nr && rs == 0) cs[r] -= a;
                }
                __syncthreads();
            }
            for (int r = tid; r < nr; r += kHbThreads) {
                const int g = r0 + r;
                if (g <= j) S.A[g + (size_t)j * S.lda] = cs[r];      // final entries of H
                else __stcg(S.c + g, cs[r]);
            }
            norms_out(j, S.partn);
        }
        arrive(0);
        if (has && i + 1 < P.ib)                                 // the next column, unchanged since the panel began
            for (int r = tid; r < nr; r += kHbThreads) aj[r] = S.A[r0 + r + (size_t)(j + 1) * S.lda];
        // This CTA's share of A v: columns [ca, ce) after j + 1 for its row tile.
        // The first of A are loaded ahead of the barrier, the first of c ahead
        // of the norm.
        const int w = n - j - 1, len = (w + P.shares - 1) / P.shares, ca = min(w, share * len), ce = min(w, ca + len);
        const int rl = tid & (P.rpc - 1), sub = tid / P.rpc, nsub = kHbThreads / P.rpc, r = rt * P.rpc + rl;
        const bool work = rt < P.tiles && r < n;
        const int pl0 = min(ce - ca, kHbPiece), sl0 = (pl0 + nsub - 1) / nsub, qa = min(sub * sl0, pl0), qb = min(qa + sl0, pl0);
        using Entry = std::conditional_t<kFix, int2, double>;
        const Entry *const Ap = kFix ? reinterpret_cast<const Entry *>(P.F) - (size_t)(k0 + 1) * n
                                     : reinterpret_cast<const Entry *>(S.A);
        const size_t ld = kFix ? (size_t)n : (size_t)S.lda;
        Entry y0[kHbAhead];
        double cpre[2];
#pragma unroll
        for (int e = 0; e < kHbAhead; ++e)
            y0[e] = work && qa + e < qb ? Ap[r + (size_t)(j + 1 + ca + qa + e) * ld] : Entry{};
        ok = wait(0);
        if (!ok) break;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int c = tid + e * kHbThreads;
            cpre[e] = rt < P.tiles && c < pl0 ? __ldcg(S.c + j + 1 + ca + c) : 0.0;
        }
        // dlarfg, the same in every CTA.
        norms_in(j, S.partn, false);
        double xnorm = sc[0], alpha = sc[1], beta = sc[2];
        const double safmin = 0x1p-969, rsafmn = 0x1p+969;       // dlamch('S') / dlamch('E')
        int knt = 0;
        if (xnorm != 0.0 && fabs(beta) < safmin) {
            do {
                ++knt;
                for (int r = tid; r < nr; r += kHbThreads)
                    if (r0 + r >= j + 2) cs[r] = cs[r] * rsafmn;
                beta = beta * rsafmn;
                alpha = alpha * rsafmn;
            } while (fabs(beta) < safmin && knt < 20);
            for (int r = tid; r < nr; r += kHbThreads)
                if (r0 + r >= j + 2) __stcg(S.c + r0 + r, cs[r]);
            double *const again = S.partn + (size_t)3 * P.own;       // the first sums may still be read
            if (has) norms_out(j, again);
            arrive(0);
            ok = wait(0);
            if (!ok) break;
            norms_in(j, again, true);
            xnorm = sc[0];
            beta = -copysign(lapy2(alpha, xnorm), alpha);
            __syncthreads();
            if (tid == 0) sc[4] = 1.0 / (alpha - beta);
            __syncthreads();
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int c = tid + e * kHbThreads;
                if (rt < P.tiles && c < pl0) cpre[e] = __ldcg(S.c + j + 1 + ca + c);
            }
        }
        const double rsc = sc[4];
        if (tid == 32) sc[3] = xnorm != 0.0 ? (beta - alpha) / beta : 0.0;       // tau, for after the product
        if (b == 0 && tid == 0) {
            for (int q = 0; q < knt; ++q) beta = beta * safmin;
            S.A[(j + 1) + (size_t)j * S.lda] = beta;
        }
        for (int r = tid; r < nr; r += kHbThreads) {
            const int g = r0 + r;
            const double v = g == j + 1 ? 1.0 : (g >= j + 2 ? cs[r] * rsc : 0.0);
            Vs[i * Rp + r] = v;
            if (g >= j + 1) S.V[g + (size_t)i * n] = v;
            if (g >= j + 2) S.A[g + (size_t)j * S.lda] = v;
        }
        // A v
        if (rt < P.tiles) {
            double x = 0.0;                                      // one chain: four warps share a sub-partition
            FixSum fx;
            bool bad = false;                                    // v not finite (kFix)
            Entry *const ve = reinterpret_cast<Entry *>(vst);
            for (int p0 = ca; p0 < ce; p0 += kHbPiece) {
                const int pl = min(ce - p0, kHbPiece), c0 = j + 1 + p0;
                if (p0 > ca) __syncthreads();
                for (int c = tid, e = 0; c < pl; c += kHbThreads, ++e) {
                    const int g = c0 + c;
                    const double v = g == j + 1 ? 1.0 : (p0 == ca ? cpre[e & 1] : __ldcg(S.c + g)) * rsc;
                    if constexpr (kFix) {
                        ve[c] = fix_parts(v, 0);
                        bad = bad || mag(v) >= pow2_bits(1);
                    } else {
                        ve[c] = v;
                    }
                }
                if (kFix) bad = __syncthreads_or(bad);
                else __syncthreads();
                const int sl = (pl + nsub - 1) / nsub, q0 = min(sub * sl, pl), q1 = min(q0 + sl, pl);
                if (r < n) {
                    int q = q0;
                    const auto add = [&](Entry a, Entry v) {
                        if constexpr (kFix) fx.add(a, v);
                        else x = fma(a, v, x);
                    };
                    if (p0 == ca) {
#pragma unroll
                        for (int e = 0; e < kHbAhead; ++e)
                            if (q + e < q1) add(y0[e], ve[q + e]);
                        q = min(q + kHbAhead, q1);
                        if constexpr (kFix) fx.carry();
                    }
                    const Entry *a = Ap + r + (size_t)(c0 + q) * ld;
                    for (int z = 0; q + 15 < q1; q += 16, a += 16 * ld) {
                        Entry y[16];
#pragma unroll
                        for (int e = 0; e < 16; ++e) y[e] = a[(size_t)e * ld];
#pragma unroll
                        for (int e = 0; e < 16; ++e) add(y[e], ve[q + e]);
                        if constexpr (kFix) {
                            fx.carry();
                            if ((++z & 1) == 0) fx.flush();      // with the 8 ahead and the 15 left, never 64
                        }
                    }
                    if (q < q1) {                                // the rest, its loads in flight together too
                        Entry y[15];
#pragma unroll
                        for (int e = 0; e < 15; ++e) y[e] = q + e < q1 ? a[(size_t)e * ld] : Entry{};
#pragma unroll
                        for (int e = 0; e < 15; ++e)
                            if (q + e < q1) add(y[e], ve[q + e]);
                    }
                    if constexpr (kFix) {
                        fx.carry();
                        fx.flush();
                    }
                }
            }
            if constexpr (kFix) {
                const unsigned top = r < n ? P.top[r] : 0u;
                x = top >= 0x7ff00000u || bad ? dg_nan() : scalbn(fx.value(), fix_exp(top) - 2 * (kFixBits - kFixLow));
            }
            if (nsub > 1) {
                gred[tid] = x;
                __syncthreads();
                int left = nsub;                                 // by fours, then what is left
                if (left > 4) {
                    left /= 4;
                    if (sub < left) {
                        x = (x + gred[(sub + left) * P.rpc + rl]) + (gred[(sub + 2 * left) * P.rpc + rl] + gred[(sub + 3 * left) * P.rpc + rl]);
                        gred[tid] = x;
                    }
                    __syncthreads();
                }
                if (sub == 0)
                    for (int z = 1; z < left; ++z) x += gred[z * P.rpc + rl];
            }
            if (sub == 0 && r < n) __stcg(S.gpart + (size_t)share * n + r, x);
        }
        __syncthreads();
        t = sc[3];
        if (b == 0 && tid == 0) S.tau[j] = t;
        if (has && i > 0) col_dots(Vs + i * Rp, i, S.part2);     // V^T v
        arrive(0);
        ok = wait(0);
        if (!ok) break;
    }
    if (!ok) {                                                   // a barrier gave up: results say so
        if (b == 0) {
            for (int q = tid; q < n; q += kHbThreads) S.tau[q] = dg_nan();
            for (int q = tid; q < kHbNb * kHbNb; q += kHbThreads) S.T[q] = dg_nan();
        }
        return;
    }
    if (b == 0) {
        __syncthreads();
        t_column(P.ib - 1, t);
        __syncthreads();
        for (int e = tid; e < kHbNb * kHbNb; e += kHbThreads) S.T[e] = Ts[(e % kHbNb) + (e / kHbNb) * (kHbNb + 1)];
    }
}

// C(i, j) = beta C(i, j) + alpha sum_k A(i, k) B(k, j), with A(i, k) =
// A[i*sai + k*sak], B(k, j) = B[k*sbk + j*sbj] (one of each pair of strides is
// 1: loads coalesce along it) and C(i, j) = C[i + j*ldc + z*cz], where part z
// of nz takes k = z kc .. .  64x64 tiles, 256 threads with a 4x4 block each, K
// in chunks of 16 through shared memory; the sum over k is one fma chain in k
// order.  CTA c takes tiles c, c + gridDim.x, ...
constexpr int kHbTm = 64, kHbTk = 16;
struct HbGemm {
    int M, N, K, nz, kc;
    double alpha;
    const double *A;
    long long sai, sak;
    const double *B;
    long long sbk, sbj;
    double beta;
    double *C;
    long long ldc, cz;
};
// Parts of K for `split` of them at most, in whole chunks.
__host__ __device__ __forceinline__ int hb_kc(int K, int split) {
    return ((K + split - 1) / split + kHbTk - 1) / kHbTk * kHbTk;
}
__host__ __device__ __forceinline__ int hb_parts(int K, int split) {
    const int kc = hb_kc(K, split);
    return (K + kc - 1) / kc;
}
struct HbTiles {
    __align__(16) double A[kHbTk][kHbTm + 2];
    __align__(16) double B[kHbTk][kHbTm + 2];
};
__device__ __forceinline__ void hb_gemm_tile(const HbGemm &g, int bx, int by, int bz, HbTiles &sm) {
    double (&As)[kHbTk][kHbTm + 2] = sm.A, (&Bs)[kHbTk][kHbTm + 2] = sm.B;
    const int tid = threadIdx.x;
    const int i0 = bx * kHbTm, j0 = by * kHbTm;
    const int kb = bz * g.kc, ke = min(g.K, kb + g.kc);
    const int tr = tid >> 4, tc = tid & 15;
    double acc[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = 0.0;
    const bool a_i = g.sai == 1;                 // A contiguous along i (else along k)
    const bool b_k = g.sbk == 1;                 // B contiguous along k (else along j)
    for (int k = kb; k < ke; k += kHbTk) {
        double ra[4], rb[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            int ii, kk;
            if (a_i) { ii = tid & 63; kk = (tid >> 6) + 4 * e; }
            else { kk = tid & 15; ii = (tid >> 4) + 16 * e; }
            const int gi = i0 + ii, gk = k + kk;
            ra[e] = (gi < g.M && gk < ke) ? g.A[(size_t)gi * g.sai + (size_t)gk * g.sak] : 0.0;
            int jj, kq;
            if (b_k) { kq = tid & 15; jj = (tid >> 4) + 16 * e; }
            else { jj = tid & 63; kq = (tid >> 6) + 4 * e; }
            const int gj = j0 + jj, gq = k + kq;
            rb[e] = (gj < g.N && gq < ke) ? g.B[(size_t)gq * g.sbk + (size_t)gj * g.sbj] : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (a_i) As[(tid >> 6) + 4 * e][tid & 63] = ra[e];
            else As[tid & 15][(tid >> 4) + 16 * e] = ra[e];
            if (b_k) Bs[tid & 15][(tid >> 4) + 16 * e] = rb[e];
            else Bs[(tid >> 6) + 4 * e][tid & 63] = rb[e];
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kHbTk; ++kk) {
            const double2 a01 = *reinterpret_cast<const double2 *>(&As[kk][4 * tr]);
            const double2 a23 = *reinterpret_cast<const double2 *>(&As[kk][4 * tr + 2]);
            const double2 b01 = *reinterpret_cast<const double2 *>(&Bs[kk][4 * tc]);
            const double2 b23 = *reinterpret_cast<const double2 *>(&Bs[kk][4 * tc + 2]);
            const double av[4] = {a01.x, a01.y, a23.x, a23.y};
            const double bv[4] = {b01.x, b01.y, b23.x, b23.y};
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) acc[a][b] = fma(av[a], bv[b], acc[a][b]);
        }
    }
    double *Cz = g.C + (size_t)bz * g.cz;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const int gj = j0 + 4 * tc + b;
        if (gj >= g.N) continue;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const int gi = i0 + 4 * tr + a;
            if (gi >= g.M) continue;
            double *cp = Cz + gi + (size_t)gj * g.ldc;
            const double v = g.alpha * acc[a][b];
            *cp = g.beta == 0.0 ? v : fma(g.beta, *cp, v);
        }
    }
}
__host__ __device__ __forceinline__ int hb_gemm_tiles(const HbGemm &g) {
    return g.M <= 0 || g.N <= 0 ? 0 : ((g.M + kHbTm - 1) / kHbTm) * ((g.N + kHbTm - 1) / kHbTm) * g.nz;
}
// `skip`: tiles of another product handed out just before.
__device__ __forceinline__ void hb_gemm_run(const HbGemm &g, HbTiles &sm, int skip = 0) {
    const int mt = (g.M + kHbTm - 1) / kHbTm, nt = (g.N + kHbTm - 1) / kHbTm, total = hb_gemm_tiles(g);
    for (int t = (blockIdx.x + gridDim.x - skip % gridDim.x) % gridDim.x; t < total; t += gridDim.x) {
        const int z = t / (mt * nt), r = t - z * mt * nt, by = r / mt;
        hb_gemm_tile(g, r - by * mt, by, z, sm);
        __syncthreads();                                         // before the next tile's first chunk
    }
}
// W(q, j) = sum over z of Wp[z](q, j), in order.
__device__ __forceinline__ void hb_sum_parts(int M, int N, int nz, const double *Wp, long long ldw, long long cz, double *W) {
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < (long long)M * N; e += (long long)gridDim.x * blockDim.x) {
        const long long q = e % M, j = e / M;
        double s = 0.0;
        for (int z = 0; z < nz; ++z) s += Wp[(size_t)z * cz + q + (size_t)j * ldw];
        W[q + (size_t)j * ldw] = s;
    }
}

// A grid barrier for kernels launched cooperatively, as in k_hb_panel: `word`
// counts arrivals since it was zeroed, in whole rounds: every launch that uses
// the word has the same grid.
// False once one gave up after kHbSpin polls.
struct GridBar {
    unsigned *word, target, G;
    __device__ __forceinline__ GridBar(unsigned *w) : word(w), target(0), G(gridDim.x) {
        // Arrivals of this launch cannot complete a round before this CTA's own.
        if (threadIdx.x == 0) target = (*reinterpret_cast<volatile unsigned *>(w) & ~kHbDead) / G * G;
    }
    __device__ __forceinline__ bool meet() {
        bool dead = false;
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(word) : "memory");
            target += G;
            unsigned it = 0, v;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
            } while (!(v & kHbDead) && (int)(v - target) < 0 && ++it < kHbSpin);
            if (it >= kHbSpin) atomicOr(word, kHbDead);
            dead = it >= kHbSpin || (v & kHbDead);
        }
        return __syncthreads_or(dead) == 0;
    }
};

// The trailing columns c1 .. n-1 of panel k0 in FP64, five phases: A(:, c1:)
// -= Y V(c1:, :)^T; the parts of V^T A(k0+1:, c1:); their sums W; T^T W; and
// A(k0+1:, c1:) -= V (T^T W).  One cooperative launch for all (first = 0, last
// = 5), so that a panel whose product runs by digits passes over it in one
// launch and not in five, or one launch a phase.
struct HbPlain {
    HbState S;
    int k0, ib, c1, split;
    double *Wp, *W, *W2;
    unsigned *bar;
    const int *uneven;                 // runs where it is not 0 (null: runs)
};
constexpr int kHbPlainPhases = 5;
__global__ void __launch_bounds__(256, 2) k_hb_plain(HbPlain P, int first, int last) {
    __shared__ HbTiles sm;
    if (P.uneven && *P.uneven == 0) return;
    const HbState &S = P.S;
    const long long n = S.n, nb = kHbNb, m = n - P.c1, kr = n - P.k0 - 1;
    double *const A1 = S.A + (size_t)P.c1 * S.lda, *const A2 = A1 + (P.k0 + 1);
    const double *const V = S.V + (P.k0 + 1);
    GridBar bar(P.bar);
    for (int ph = first; ph < last; ++ph) {
        if (ph == 2) {
            hb_sum_parts(P.ib, (int)m, hb_parts((int)kr, P.split), P.Wp, nb, nb * m, P.W);
        } else {
            HbGemm g;
            if (ph == 0) g = HbGemm{(int)n, (int)m, P.ib, 1, P.ib, -1.0, S.Y, 1, n, S.V + P.c1, n, 1, 1.0, A1, S.lda, 0};
            if (ph == 1)
                g = HbGemm{P.ib, (int)m, (int)kr, hb_parts((int)kr, P.split), hb_kc((int)kr, P.split), 1.0, V, n, 1, A2, 1,
                           S.lda, 0.0, P.Wp, nb, nb * m};
            if (ph == 3) g = HbGemm{P.ib, (int)m, P.ib, 1, P.ib, 1.0, S.T, nb, 1, P.W, 1, nb, 0.0, P.W2, nb, 0};
            if (ph == 4) g = HbGemm{(int)kr, (int)m, P.ib, 1, P.ib, -1.0, V, 1, n, P.W2, 1, nb, 1.0, A2, S.lda, 0};
            hb_gemm_run(g, sm);
        }
        if (ph + 1 < last && !bar.meet()) {
            if (blockIdx.x == 0)
                for (int q = threadIdx.x; q < n; q += blockDim.x) S.tau[q] = dg_nan();
            return;
        }
    }
}
// A cooperative launch that this device, or what is left of it, cannot take.
bool refused(cudaError_t e) { return e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported; }
// HSR_HESS_PANEL=steps: do without cooperative launches (read per call: tests
// switch it).
bool without_cooperative() {
    const char *env = getenv("HSR_HESS_PANEL");
    return env && !strcmp(env, "steps");
}
// All phases of a kernel k(P, first, last) in one cooperative launch, or, where
// the device refuses that, one by one.
template <class Params>
cudaError_t launch_phases(void (*kernel)(Params, int, int), Params P, int phases, int grid, cudaStream_t st) {
    int first = 0;
    void *args[] = {&P, &first, &phases};
    if (!without_cooperative()) {
        const cudaError_t e =
            cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(kernel), dim3(grid), dim3(256), args, 0, st);
        if (!refused(e)) return e;
        cudaGetLastError();
    }
    for (; first < phases; ++first) kernel<<<grid, 256, 0, st>>>(P, first, first + 1);
    return cudaGetLastError();
}

// Whether the sizes of A's entries allow digits and fixed point: in every row
// but the first (no reflector touches it) and in every column, three fifths of
// the entries lie within 2^8 of the largest of all.  Then every reflector mixes
// entries of like size, and FP64 itself leaves errors of the size of the
// largest entry's rounding everywhere.  Measured, n = 160, Q^T A Q - H in extended
// precision, by digits over FP64, median and largest ratio of the root mean
// squares of its columns, against the bits a matrix needs: N(0,1) entries (4) 0.83,
// 1.8; Z H Z^T, Z orthogonal (3) 0.87, 1.3; G G^T (5) 0.93, 1.7; G + 100 D (9) 0.98,
// 2.5; a Hessenberg matrix between two reflectors (10) 0.96, 3.1; Cauchy entries
// (16) 0.86, 5.3, cubed (49) 1.4, 38.  D G D scaled by 1 / (d_i d_j), relative to
// G, FP64 / digits, n = 160 (4000): d from 1 to 2^-8 (14) 7.2e-15 / 6.8e-15
// (2.3e-14 / 2.1e-14), to 2^-16 (27) 2.9e-14 / 7.5e-14 (7.3e-14 / 3.1e-13), to
// 1e-16 4.6e-13 / 3e-4.  The check reads A once: n = 700 13.35 -> 13.38 ms with
// the launches that do nothing, n = 4000 138.2 -> 139.3, n = 6000 317.0 -> 318.0.
// Refused, d to 1e-12: n = 700 16.4 ms, n = 4000 324.
constexpr int kHbEvenBits = 8;
__device__ __forceinline__ bool hb_few(int low, int of) { return 5 * low <= 2 * of; }
// Counts of entries by row, low[r], and by column, low[n + c]: a warp takes 32 x
// 32 of them, a lane a row, its 32 loads in flight together, and its lane c ends
// with column c's count; warps side by side take rows below one another.
// get(r, c): an entry; limit(c): what the lane of column c contributes to
// small(x, r, c, limit), which tells whether it counts.  Above the diagonal of
// c = r + below there is nothing to count.  Bound by the latency of the loads,
// with 16 warps an SM: V of n = 5000 (100 MB) 52 us; with the loads under the
// conditions 120, with block-wide counts in shared memory 90 to 115.
constexpr int kEvenTile = 32;
template <class Get, class Limit, class Small>
__device__ __forceinline__ void even_count(int n, int r0, int rows, int cols, int below, const Get &get, const Limit &limit,
                                           const Small &small, int *low) {
    const int lane = threadIdx.x & 31, nr = (rows + kEvenTile - 1) / kEvenTile, nc = (cols + kEvenTile - 1) / kEvenTile;
    const int warps = gridDim.x * (blockDim.x >> 5);
    for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < nr * nc; t += warps) {
        const int c0 = t / nr * kEvenTile, ra = r0 + t % nr * kEvenTile, r = ra + lane;
        if (c0 > ra + kEvenTile - 1 + below) continue;
        double x[kEvenTile];
#pragma unroll
        for (int c = 0; c < kEvenTile; ++c) x[c] = get(min(r, n - 1), min(c0 + c, cols - 1));   // unconditional loads
        const int lim = c0 + lane < cols ? limit(c0 + lane) : 0;
        int mine = 0, ours = 0;
#pragma unroll
        for (int c = 0; c < kEvenTile; ++c) {
            const int l = __shfl_sync(0xffffffffu, lim, c);      // by all lanes, also those past the last row
            const bool s = r < n && c0 + c < cols && small(x[c], r, c0 + c, l);
            const unsigned b = __ballot_sync(0xffffffffu, s);
            if (lane == c) ours = __popc(b);
            mine += s;
        }
        if (mine) atomicAdd(&low[r], mine);
        if (ours) atomicAdd(&low[n + c0 + lane], ours);
    }
}
int even_grid(int rows, int cols, int sms) {                     // CTAs of 256 threads
    const long long tiles = (long long)((rows + kEvenTile - 1) / kEvenTile) * ((cols + kEvenTile - 1) / kEvenTile);
    return (int)std::min<long long>(2 * sms, (tiles + 7) / 8);
}
// The CTA that counted last sees all counts.
__device__ __forceinline__ bool even_last(unsigned *cnt) {
    __shared__ bool am_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) am_last = atomicAdd(cnt, 1u) == gridDim.x - 1;
    __syncthreads();
    if (am_last) __threadfence();
    return am_last;
}
// cex: exponents of A's columns over rows 1 ..; low: 2 n counts, zeroed, of the
// rows' and the columns' smaller (or non-finite) entries; cnt: a counter, zeroed.
__global__ void __launch_bounds__(256) k_hb_even(int n, const double *A, long long lda, const int *cex, int *low, unsigned *cnt,
                                                 int *uneven) {
    __shared__ int red[8];
    const int tid = threadIdx.x;
    int top = kDgZero;
    for (int c = tid; c < n; c += 256) top = dg_bad(cex[c]) ? top : max(top, cex[c]);
    top = __reduce_max_sync(0xffffffffu, top);
    if ((tid & 31) == 0) red[tid >> 5] = top;
    __syncthreads();
    for (int w = 0; w < 8; ++w) top = max(top, red[w]);
    even_count(n, 1, n - 1, n, n, [&](int r, int c) { return A[r + (size_t)c * lda]; }, [](int) { return 0; },
               [&](double x, int, int, int) {
                   const int e = dg_exp(x);
                   return e < top - kHbEvenBits || dg_bad(e);
               }, low);
    if (!even_last(cnt)) return;
    bool bad = false;
    for (int q = tid; q < n; q += 256) bad = bad || !hb_few(__ldcg(&low[n + q]), n - 1) || (q > 0 && !hb_few(__ldcg(&low[q]), n));
    bad = __syncthreads_or(bad);
    if (tid == 0) *uneven = bad;
}

// Back-transform Q X in FP64, blocked like LAPACK dormhr ('L', 'N'): the panels
// of the reduction in reverse order, X(k0+1:, :) -= V (T (V^T X(k0+1:, :))),
// with V rebuilt from the reflectors stored in A and T from V and tau (dlarft:
// T(0:i, i) = -tau_i T(0:i, 0:i) (V^T V)(0:i, i), T(i, i) = tau_i).  Six phases a
// panel: V; the parts of V^T V and V^T X; their sums G and W; T; T W; X.  One
// cooperative launch for all panels, so that a call which the digits take
// passes over it in one launch.
struct HqPlain {
    int n, ncols;
    const double *A;
    long long lda;
    const double *tau;
    double *X;
    long long ldx;
    double *V, *T, *G, *Gp, *W, *Wp, *W2;
    int splitg, splitw;                // parts of the sums over rows, at most
    unsigned *bar;
    const int *uneven;                 // runs where it is not 0 (null: runs)
};
constexpr int kHqPlainPhases = 6;
__global__ void __launch_bounds__(256, 2) k_hq_plain(HqPlain P, int first, int last) {
    __shared__ HbTiles sm;
    if (P.uneven && *P.uneven == 0) return;
    const long long n = P.n, nb = kHbNb, nc = P.ncols;
    const int panels = (P.n - 3) / kHbNb + 1;
    GridBar bar(P.bar);
    for (int ph = first; ph < last; ++ph) {
        const int k0 = (panels - 1 - ph / kHqPlainPhases) * kHbNb, ib = min(kHbNb, P.n - 2 - k0), kr = P.n - k0 - 1;
        const double *const V = P.V + (k0 + 1);
        double *const X = P.X + (k0 + 1);
        const int zg = hb_parts(kr, P.splitg), zw = hb_parts(kr, P.splitw);
        switch (ph % kHqPlainPhases) {
        case 0:
            for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < n * ib; e += (long long)gridDim.x * blockDim.x) {
                const int i = (int)(e / n), r = (int)(e - i * n), j = k0 + i;
                P.V[e] = r == j + 1 ? 1.0 : (r >= j + 2 ? P.A[r + (size_t)j * P.lda] : 0.0);
            }
            break;
        case 1:
            {
                const HbGemm w{ib, P.ncols, kr, zw, hb_kc(kr, P.splitw), 1.0, V, n, 1, X, 1, P.ldx, 0.0, P.Wp, nb, nb * nc};
                hb_gemm_run(w, sm);
                hb_gemm_run(HbGemm{ib, ib, kr, zg, hb_kc(kr, P.splitg), 1.0, V, n, 1, V, 1, n, 0.0, P.Gp, nb, nb * ib}, sm,
                            hb_gemm_tiles(w));
            }
            break;
        case 2:
            hb_sum_parts(ib, ib, zg, P.Gp, nb, nb * ib, P.G);
            hb_sum_parts(ib, P.ncols, zw, P.Wp, nb, nb * nc, P.W);
            break;
        case 3:
            for (int i = 0; blockIdx.x == 0 && i < ib; ++i) {
                const double t = P.tau[k0 + i];
                for (int p = threadIdx.x; p < i; p += blockDim.x) {
                    double s = 0.0;
                    for (int q = p; q < i; ++q) s = fma(P.T[p + (size_t)q * kHbNb], P.G[q + (size_t)i * kHbNb], s);
                    P.T[p + (size_t)i * kHbNb] = -t * s;
                }
                for (int p = i + threadIdx.x; p < kHbNb; p += blockDim.x) P.T[p + (size_t)i * kHbNb] = p == i ? t : 0.0;
                __syncthreads();
            }
            break;
        case 4:
            hb_gemm_run(HbGemm{ib, P.ncols, ib, 1, ib, 1.0, P.T, 1, nb, P.W, 1, nb, 0.0, P.W2, nb, 0}, sm);
            break;
        default:
            hb_gemm_run(HbGemm{kr, P.ncols, ib, 1, ib, -1.0, V, 1, n, P.W2, 1, nb, 1.0, X, P.ldx, 0}, sm);
        }
        if (ph + 1 < last && !bar.meet()) {
            if (blockIdx.x == 0)
                for (long long e = threadIdx.x; e < (n - 1) * nc; e += blockDim.x) P.X[1 + e % (n - 1) + (e / (n - 1)) * P.ldx] = dg_nan();
            return;
        }
    }
}

// ------------------------------------------------ back-transform by digits
// The same back-transform with the products on the bf16 tensor cores
// (hsr_digits.cuh), in blocks of kHqNb = 128 reflectors, one row block of
// digits.  Blocks are taken in groups whose digits of V fit kHqVBytes: for a
// group, the digits, the Gram matrices V^T V and the factors T of all its
// blocks at once (they do not depend on X), then per block W = V^T X, T W and
// X -= V (T W).
constexpr int kHqNb = 128;
// Smallest order: a reflector of the DFMA form costs about 5.5 us (three thin
// products and a serial factor per 64), this form 240 us and 0.5 us each
// (n = 32: 139 us as DFMA; 64: 360 against 249; 300: 1,665 against 411; 4000
// with 2000 columns: 85.7 ms against 5.2).  The DFMA form also stays for
// reflectors that are not even and for a scratch buffer that cannot be had.
constexpr int kHqDigitsN = 40;
// Most scratch for digits of X's columns and of V (three layouts) at a time.
constexpr size_t kHqXBytes = (size_t)1 << 30, kHqVBytes = (size_t)4 << 30;   // (V of n = 10,000: 2.5 GB)
constexpr int kHqMaxSplit = 16;

// Whether the reflectors allow digits.  A column of X is held by a window below
// its largest entry in rows 1 ..; that loses nothing where the reflectors carry
// an entry of that size into every row, whose rounding in FP64 is then as large.
// So in every column of V with kHqEvenMin entries below its 1, and in every row
// with as many, three fifths of the entries have to be at least 2^-3 / sqrt(m),
// m the length of the column (a reflector's norm is at most sqrt(2) and that of
// a random one's entries about 1 / sqrt(m)), and tau not near 0.  Reflectors of
// D G D on columns D G', G and G' of N(0,1) entries, error row by row relative
// to the row's largest, root mean square, in FP64 / by digits, n = 160 (500): d
// from 1 to 2^-6 3.7e-16 / 3.0e-16 (4.0e-16 / 2.3e-16), to 2^-8, which is
// refused, 3.5e-16 / 5.4e-16 (3.8e-16 / 2.9e-16), to 2^-16 3.3e-16 / 2.3e-14
// (3.9e-16 / 1.3e-14); d to 1e-12 (n = 300), the largest, 3.3e-15 / 2.3e-7.
// Random reflectors need 2^-2 at most.  The check reads V once: n = 64
// 236 -> 250 us, n = 700 625 -> 640, n = 5000 with 2500 columns 8.54 -> 8.63 ms.
// Refused, n = 700 with 350 columns 4.0 ms, n = 4000 with 2000 89.
constexpr int kHqEvenBits = 3, kHqEvenMin = 32;
// low: 2 n counts, zeroed, of the rows' and the columns' smaller entries; cnt: a
// counter, zeroed.
__global__ void __launch_bounds__(256) k_hq_even(int n, const double *A, long long lda, const double *tau, int *low, unsigned *cnt,
                                                 int *uneven) {
    const int tid = threadIdx.x;
    even_count(n, 2, n - 2, n - 2, -2, [&](int r, int c) { return A[r + (size_t)c * lda]; },
               [&](int c) {                                      // smallest exponent of column c that counts
                   const unsigned long long t = ubits(tau[c]);   // mixing: 0.5 <= tau, no NaN
                   return t < pow2_bits(-1) || t >= kInfBits ? INT_MAX : 1022 - kHqEvenBits - ((32 - __clz(n - 1 - c)) >> 1);
               },
               [&](double x, int r, int c, int least) {
                   const int e = dg_exp(x);
                   return r >= c + 2 && (e < least || dg_bad(e));
               }, low);
    if (!even_last(cnt)) return;
    bool bad = false;
    for (int q = tid; q < n; q += 256) {
        const int below = n - 2 - q, left = q - 1;               // entries of column q and of row q
        bad = bad || (below >= kHqEvenMin && !hb_few(__ldcg(&low[n + q]), below)) ||
              (left >= kHqEvenMin && !hb_few(__ldcg(&low[q]), left));
    }
    bad = __syncthreads_or(bad);
    if (tid == 0) *uneven = bad;
}

// The blocks of a group, last first: block g of the group begins at reflector
// k0(g) and has rows k0 + 1 .. n - 1.  Its row blocks of 128 count from the
// bottom, so that block g has g more of them than block 0 and places are
// sums: `rb0` row blocks in block 0.
struct HqGroup {
    const double *A;
    long long lda;
    int n, klast, rb0;                                           // klast: k0 of block 0
    const int *off;
    __host__ __device__ __forceinline__ int k0(int g) const { return klast - g * kHqNb; }
    __host__ __device__ __forceinline__ int rblocks(int g) const { return rb0 + g; }
    __host__ __device__ __forceinline__ long long before(int g) const {      // row blocks of blocks 0 .. g-1
        return (long long)g * rb0 + (long long)g * (g - 1) / 2;
    }
    // V(i, q) of block g.
    __device__ __forceinline__ double at(int g, int i, int q) const {
        const int j = k0(g) + q;
        if (j >= n - 2 || i >= n || i < j + 1) return 0.0;
        return i == j + 1 ? 1.0 : A[i + (size_t)j * lda];
    }
};
// Exponents of V's columns (row g * 128 + q: column q of block g).
struct HqVCols {
    HqGroup h;
    __device__ __forceinline__ double operator()(int r, int k) const {
        const int g = r / kHqNb;
        return h.at(g, h.k0(g) + 1 + k, r % kHqNb);
    }
};
// Digits of V's columns as row blocks of RB (128: the A side, 64: the B
// side): block (x, y) = eight columns and 256 rows of block z of the group.
template <int RB>
__global__ void __launch_bounds__(256) k_hq_vcols(HqGroup h, const int *ex, unsigned char *out) {
    const int t = threadIdx.x, g = blockIdx.z, r = blockIdx.x * 8 + (t & 7), c8 = blockIdx.y * 32 + (t >> 3);
    const int steps = h.rblocks(g) * (kHqNb / kDgBK);
    if (dg_off(h.off)) return;
    if (c8 >= 2 * steps) return;
    const int base = max(ex[g * kHqNb + r], kDgZero) - 9, i0 = h.k0(g) + 1 + c8 * 8;
    unsigned long long u[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) u[e] = dg_digits(h.at(g, i0 + e, r), base);
    dg_store8(u, out + (size_t)h.before(g) * kHqNb * kHqNb * kDgDigits * 2 + dg_place(r, c8, RB, steps), RB * kDgBK * 2);
}
// Exponents and digits of V's rows: 32 rows of one block of the group.
__global__ void __launch_bounds__(512) k_hq_vrows(HqGroup h, int *ex, unsigned char *out) {
    __shared__ int red[32][17];
    const int t = threadIdx.x, g = blockIdx.y, rr = t & 31, c8 = t >> 5, r = blockIdx.x * 32 + rr;
    if (dg_off(h.off) || r - rr >= h.rblocks(g) * kHqNb) return; // uniform over the block
    double x[8];
    int m = kDgZero;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        x[e] = h.at(g, h.k0(g) + 1 + r, c8 * 8 + e);
        m = max(m, dg_exp(x[e]));
    }
    red[rr][c8] = m;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; ++q) m = max(m, red[rr][q]);
    const size_t row = (size_t)h.before(g) * kHqNb + r;
    if (c8 == 0) ex[row] = m;
    unsigned long long u[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) u[e] = dg_digits(x[e], m - 9);
    dg_store8(u, out + (size_t)h.before(g) * kHqNb * kHqNb * kDgDigits * 2 + dg_place(r, c8, kDgBM, kHqNb / kDgBK),
              kDgBM * kDgBK * 2);
}
// Gram matrices of a group: part z of block g to S[(g * nz + z)].
struct HqGram {
    using Sum = DgTwo<16>;
    static constexpr int kWarps = 16;
    HqGroup h;
    int nz;
    const int *ex;
    double *S;
    __device__ __forceinline__ DgTile tile(int t) const {
        const int g = t / (2 * nz), r = t - g * 2 * nz, z = r >> 1, by = r & 1;
        const int steps = h.rblocks(g) * (kHqNb / kDgBK), per = (steps + nz - 1) / nz, s0 = min(z * per, steps);
        const long long at = h.before(g) * (kHqNb / kDgBK);
        return DgTile{g, by, z, at + s0, 2 * at + (long long)by * steps + s0, min(steps - s0, per)};
    }
    __device__ __forceinline__ void finish(const DgTile &q, int i, int j0, const Sum &sum) const {
        const int p = i - q.bx * kDgBM, lane = threadIdx.x & 31;
        const int ecl = max(ex[q.bx * kHqNb + j0 + (lane & 15)], kDgZero), er = max(ex[q.bx * kHqNb + p], kDgZero);
        double *o = S + ((size_t)q.bx * nz + q.bz) * kHqNb * kHqNb + p + (size_t)j0 * kHqNb;
#pragma unroll
        for (int c = 0; c < Sum::kCols; ++c) {
            const int ec = __shfl_sync(0xffffffffu, ecl, c);
            const double v = sum.value(c, er + ec - 2044);
            o[(size_t)c * kHqNb] = dg_bad(er) || dg_bad(ec) ? dg_nan() : v;
        }
    }
    // The group's block 0, which the back-transform takes first and whose rows
    // every later block mixes into all of X.
    __device__ void poison(int thread, int threads) const {
        for (int e = thread; e < nz * kHqNb * kHqNb; e += threads) S[e] = dg_nan();
    }
};
// Rows of the operand are columns of a column-major matrix.
struct HqCols {
    const double *X;
    long long ld;
    int cols, rows;
    __device__ __forceinline__ double operator()(int r, int k) const {
        return r < cols && k < rows ? X[k + (size_t)r * ld] : 0.0;
    }
    __device__ __forceinline__ int first(int) const { return 0; }
};
// W(:, j) as the sum of nz partial products, in order.
struct HqSum {
    const double *Wp;
    int nz;
    long long cz;
    __device__ __forceinline__ double operator()(int r, int k) const {
        double s = 0.0;
        for (int z = 0; z < nz; ++z) s += Wp[(size_t)z * cz + k + (size_t)r * kHqNb];
        return s;
    }
};
// Factors T of all blocks, stacked (row r of the operand: row r % 128 of block r / 128).
struct HqT {
    const double *T;
    __device__ __forceinline__ double operator()(int r, int k) const {
        return T[(size_t)(r / kHqNb) * kHqNb * kHqNb + (r % kHqNb) + (size_t)k * kHqNb];
    }
};

// dlarft of a block of 128 in three parts, from S = V^T V (summed from its
// partial products): the factors T11 and T22 of its halves, T(0:i, i) =
// -tau_i T(0:i, 0:i) S(0:i, i), T(i, i) = tau_i, by one CTA each, four threads
// per row; then T12 = -T11 S12 T22, eight columns per CTA.  Bound by the FP64
// pipe of the SMs that take part (a warp's FMA 64 clocks): one CTA for the
// whole block 254 us, this form 79 + 50 us, for any number of blocks.
constexpr int kHqHalf = kHqNb / 2;
__device__ __forceinline__ int hq_packed(int p, int i) { return p + i * (i + 1) / 2; }
__device__ __forceinline__ double hq_gram(const double *S, int nz, int p, int i) {
    double s = 0.0;
#pragma unroll 4
    for (int z = 0; z < nz; ++z) s += S[(size_t)z * kHqNb * kHqNb + p + (size_t)i * kHqNb];
    return s;
}
__global__ void __launch_bounds__(4 * kHqHalf) k_hq_thalf(HqGroup h, const double *tau, const double *Sp, int nz, double *T) {
    __shared__ double ts[kHqHalf * (kHqHalf + 1) / 2], ss[kHqHalf * (kHqHalf + 1) / 2], part[4][kHqHalf];
    if (dg_off(h.off)) return;
    const int p = threadIdx.x % kHqHalf, w = threadIdx.x / kHqHalf, o = blockIdx.y * kHqHalf;
    const int k0 = h.k0(blockIdx.x) + o, ib = max(0, min(kHqHalf, h.n - 2 - k0));
    const double *S = Sp + (size_t)blockIdx.x * nz * kHqNb * kHqNb + o + (size_t)o * kHqNb;
    double *To = T + (size_t)blockIdx.x * kHqNb * kHqNb + o + (size_t)o * kHqNb;
    for (int i = w; i < kHqHalf; i += 4) {
        if (p < i) ss[hq_packed(p, i)] = hq_gram(S, nz, p, i);
        if (p > i || i >= ib) To[p + (size_t)i * kHqNb] = 0.0;
    }
    for (int i = 0; i < ib; ++i) {
        __syncthreads();                                         // S, T(:, i - 1)
        double a = 0.0;
        for (int q = p + w; q < i; q += 4) a = fma(ts[hq_packed(p, q)], ss[hq_packed(q, i)], a);
        part[w][p] = a;
        __syncthreads();
        if (w == 0 && p <= i) {
            const double t = tau[k0 + i];
            const double v = p < i ? -t * ((part[0][p] + part[1][p]) + (part[2][p] + part[3][p])) : t;
            ts[hq_packed(p, i)] = v;
            To[p + (size_t)i * kHqNb] = v;
        }
    }
}
__global__ void __launch_bounds__(8 * kHqHalf) k_hq_tcross(HqGroup h, const double *Sp, int nz, double *T) {
    __shared__ double s12[kHqHalf][kHqHalf + 1], t22[kHqHalf][8], u[kHqHalf][8];
    if (dg_off(h.off)) return;
    const int p = threadIdx.x % kHqHalf, c = threadIdx.x / kHqHalf, col = blockIdx.y * 8 + c;
    const double *S = Sp + (size_t)blockIdx.x * nz * kHqNb * kHqNb + (size_t)kHqHalf * kHqNb;   // S(0.., 64..)
    double *To = T + (size_t)blockIdx.x * kHqNb * kHqNb;
    for (int r = c; r < kHqHalf; r += 8) s12[r][p] = hq_gram(S, nz, p, r);       // S12(p, r)
    t22[p][c] = To[kHqHalf + p + (size_t)(kHqHalf + col) * kHqNb];
    __syncthreads();
    double a0 = 0.0, a1 = 0.0;
    for (int r = 0; r <= col; r += 2) {                          // T22 is zero below its diagonal
        a0 = fma(s12[r][p], t22[r][c], a0);
        a1 = fma(s12[r + 1][p], t22[r + 1][c], a1);
    }
    u[p][c] = a0 + a1;
    __syncthreads();
    a0 = a1 = 0.0;
    for (int q = p & ~31; q < kHqHalf; q += 2) {                 // T11 likewise
        a0 = fma(To[p + (size_t)q * kHqNb], u[q][c], a0);
        a1 = fma(To[p + (size_t)(q + 1) * kHqNb], u[q + 1][c], a1);
    }
    To[p + (size_t)(kHqHalf + col) * kHqNb] = -(a0 + a1);
    To[kHqHalf + p + (size_t)col * kHqNb] = 0.0;                 // T21
}

// Scratch of the digit form, laid out once.
struct HqDigits {
    unsigned char *XN, *VM, *VN, *VA, *TM, *WN;
    double *S, *T, *Wp, *W2;
    int *exX, *exW, *exVA, *exV, *exT, *low;                     // low: k_hq_even's counts, a counter, the result and
                                                                 // k_hq_plain's barrier
    int nblk, cch, gmax;                                         // blocks of reflectors, columns at a time, blocks of a group
};
constexpr size_t kHqVBlock = (size_t)kHqNb * kHqNb * kDgDigits * 2, kHqSmall = (size_t)kHqNb * kDgDigits * 2;
size_t hq_digits_layout(int n, int ncols, unsigned char *base, HqDigits &D) {
    D.nblk = (n - 3) / kHqNb + 1;
    const int rbmax = (n - 1 + kHqNb - 1) / kHqNb;               // row blocks of the first one
    const size_t per_row = (size_t)rbmax * kHqNb * kDgDigits * 2;
    const size_t fit = std::max<size_t>(1, kHqXBytes / (per_row * kDgBN)) * kDgBN;
    D.cch = (int)std::min<size_t>(fit, (size_t)((ncols + kDgBN - 1) / kDgBN) * kDgBN);
    // Row blocks of a group, at most: the g first blocks have rbmax, rbmax - 1, ... of them.
    const auto rows_of = [&](size_t g) { return g * rbmax - g * (g - 1) / 2; };
    D.gmax = 1;
    while (D.gmax < D.nblk && 3 * kHqVBlock * rows_of(D.gmax + 1) <= kHqVBytes) ++D.gmax;
    const size_t vrb = rows_of(D.gmax);
    size_t off = 0;
    const auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) / 256 * 256;
        return base + o;
    };
    D.XN = take((size_t)D.cch * per_row);
    D.VM = take(vrb * kHqVBlock);
    D.VN = take(vrb * kHqVBlock);
    D.VA = take(vrb * kHqVBlock);
    D.TM = take((size_t)D.gmax * kHqNb * kHqSmall);
    D.WN = take((size_t)D.cch * kHqSmall);
    D.S = reinterpret_cast<double *>(take((size_t)D.gmax * kHqMaxSplit * kHqNb * kHqNb * 8));
    D.T = reinterpret_cast<double *>(take((size_t)D.gmax * kHqNb * kHqNb * 8));
    D.Wp = reinterpret_cast<double *>(take((size_t)kHqMaxSplit * kHqNb * D.cch * 8));
    D.W2 = reinterpret_cast<double *>(take((size_t)kHqNb * D.cch * 8));
    D.exX = reinterpret_cast<int *>(take(((size_t)ncols + D.cch + vrb * kHqNb + (size_t)2 * D.gmax * kHqNb + 2 * n + 3) * sizeof(int)));
    D.exW = D.exX + ncols;
    D.exVA = D.exW + D.cch;
    D.exV = D.exVA + vrb * kHqNb;
    D.exT = D.exV + D.gmax * kHqNb;
    D.low = D.exT + D.gmax * kHqNb;
    return off;
}
// Enqueues the digit form, which does nothing where *uneven (set here) is not 0.
cudaError_t hq_digits(const HqDigits &D, int n, const double *dA, int lda, const double *dtau, int ncols, double *dX, int ldx,
                      int sms, cudaStream_t st, const int **uneven) {
    constexpr int ksteps = kHqNb / kDgBK;
    constexpr size_t vblock = kHqVBlock, small = kHqSmall;
    const int nblk = D.nblk, cch = D.cch, gmax = D.gmax;
    unsigned char *const XN = D.XN, *VM = D.VM, *VN = D.VN, *VA = D.VA, *TM = D.TM, *WN = D.WN;
    double *S = D.S, *T = D.T, *Wp = D.Wp, *W2 = D.W2;
    int *exX = D.exX, *exW = D.exW, *exVA = D.exVA, *exV = D.exV, *exT = D.exT, *low = D.low, *gate = low + 2 * n + 1;
    cudaError_t e = cudaMemsetAsync(low, 0, (size_t)(2 * n + 3) * sizeof(int), st);
    if (e != cudaSuccess) return e;
    *uneven = gate;
    k_hq_even<<<even_grid(n, n - 2, sms), 256, 0, st>>>(
        n, dA, lda, dtau, low, reinterpret_cast<unsigned *>(low + 2 * n), gate);
    // Over the rows that reflectors touch: row 0 stays what it is.
    k_dg_exp_k<<<ncols, 256, 0, st>>>(HqCols{dX + 1, ldx, ncols, n - 1}, n - 1, nullptr, 0, exX);
    for (int last = nblk - 1; last >= 0; last -= gmax) {
        const int ng = std::min(gmax, last + 1);
        const HqGroup h{dA, lda, n, last * kHqNb, (n - 1 - last * kHqNb + kHqNb - 1) / kHqNb, gate};
        const int rmax = h.rblocks(ng - 1), gz = std::min(kHqMaxSplit, std::max(1, 2 * sms / (2 * ng)));
        k_dg_exp_k<<<ng * kHqNb, 256, 0, st>>>(HqVCols{h}, n - h.k0(ng - 1) - 1, nullptr, 0, exV);
        const dim3 gv(kHqNb / 8, (unsigned)((2 * rmax * ksteps + 31) / 32), ng);
        k_hq_vcols<kDgBM><<<gv, 256, 0, st>>>(h, exV, VM);
        k_hq_vcols<kDgBN><<<gv, 256, 0, st>>>(h, exV, VN);
        k_hq_vrows<<<dim3(rmax * (kHqNb / 32), ng), 512, 0, st>>>(h, exVA, VA);
        if ((e = dg_gemm(2 * gz * ng, sms, VM, VN, HqGram{h, gz, exV, S}, gate, st)) != cudaSuccess) return e;
        k_hq_thalf<<<dim3(ng, 2), 4 * kHqHalf, 0, st>>>(h, dtau, S, gz, T);
        k_hq_tcross<<<dim3(ng, kHqHalf / 8), 8 * kHqHalf, 0, st>>>(h, S, gz, T);
        k_dg_small<HqT, true><<<ng * (kHqNb / 32), 512, 0, st>>>(HqT{T}, kDgBM, ng * kHqNb, ng * kHqNb, kHqNb, nullptr, 0,
                                                                exT, TM);
        for (int c0 = 0; c0 < ncols; c0 += cch) {
            const int cols = std::min(cch, ncols - c0), cb = (cols + kDgBN - 1) / kDgBN;
            for (int g = 0; g < ng; ++g) {
                const int k0 = h.k0(g), kr = n - k0 - 1, rb = h.rblocks(g), steps = rb * ksteps;
                const long long at = h.before(g);
                double *X = dX + (size_t)c0 * ldx + k0 + 1;
                k_dg_split<HqCols, false><<<dim3(cb * (kDgBN / 8), (unsigned)((2 * steps + 31) / 32)), 256, 0, st>>>(
                    HqCols{X, ldx, cols, kr}, kDgBN, cb * kDgBN, steps, exX + c0, nullptr, 0, cols, kr, XN);
                int per = 0;
                const int nz = dg_parts(cb, sms, kHqMaxSplit, steps, per);
                const DgStoreLong e1{1, cb, steps, per, kHqNb, cols, exV + g * kHqNb, exX + c0, Wp, 1, kHqNb,
                                     (long long)kHqNb * cols};
                if ((e = dg_gemm(cb * nz, sms, VM + (size_t)at * vblock, XN, e1, gate, st)) != cudaSuccess) return e;
                k_dg_small<HqSum, false><<<cb * (kDgBN / 8), 128, 0, st>>>(HqSum{Wp, nz, (long long)kHqNb * cols}, kDgBN,
                                                                         cols, cb * kDgBN, kHqNb, nullptr, 0, exW, WN);
                const DgStoreShort e2{1, cb, ksteps, ksteps, kHqNb, cols, exT + g * kHqNb, exW, W2, 1, kHqNb, 0};
                if ((e = dg_gemm(cb, sms, TM + (size_t)g * kHqNb * small, WN, e2, gate, st)) != cudaSuccess) return e;
                k_dg_small<HqSum, false><<<cb * (kDgBN / 8), 128, 0, st>>>(HqSum{W2, 1, 0}, kDgBN, cols, cb * kDgBN, kHqNb,
                                                                         nullptr, 0, exW, WN);
                const DgUpdate e3{rb, ksteps, kr, cols, exVA + at * kHqNb, exW, X, ldx, exX + c0, 0};
                if ((e = dg_gemm(rb * cb, sms, VA + (size_t)at * vblock, WN, e3, gate, st)) != cudaSuccess) return e;
            }
        }
    }
    return cudaGetLastError();
}

// ------------------------------------------------ trailing update by digits
// Both sides of a panel's block reflector in one rank-128 product: with Y =
// A V T and W0 = V^T A(k0+1:, c1:) over the panel-start A,
//   (I - V T^T V^T) (A - Y V^T) = A - Y V^T - V Z,
//   Z = T^T W0 - T^T (V^T Y) V(c1:, :)^T,
// so the trailing columns are read once for W0 and read and written once for
// A -= [Y V] [V(c1:, :)^T; Z], where the two sides one after the other pass
// over them five times.  V^T Y comes with W0 (Y's columns follow A's).
constexpr size_t kHbDigitBytes = (size_t)2 << 30;   // most scratch for digits of A's columns at a time (or 8 n^2 bytes, below)
constexpr int kHbParts = 16;
// Smallest order: the DFMA form's thin products take about 65 us each on the
// few SMs they fill (n = 10, no trailing product worth the name: 331 us
// against 354; 40: 1,729 against 1,664; 700: 41.4 ms against 39.4; 6000: 1,130
// against 691, the rest of it the panels).  The DFMA form also stays for a
// scratch buffer that cannot be had.
constexpr int kHbDigitsN = 32;

// Columns c0 + r of A, then Y's; rows k0 + 1 + k.
struct HbTrail {
    const double *A, *Y;
    long long lda;
    int n, k0, c0;
    __device__ __forceinline__ double operator()(int r, int k) const {
        const int i = k0 + 1 + k, c = c0 + r;
        if (i >= n || c >= n + kHbNb) return 0.0;
        return c < n ? A[i + (size_t)c * lda] : Y[i + (size_t)(c - n) * n];
    }
    __device__ __forceinline__ int first(int) const { return 0; }
};
// Columns of [Y V] (rows k0 + 1 + k), for their exponents, and V's alone.
struct HbPanelCols {
    const double *Y, *V;
    int n, k0;
    __device__ __forceinline__ double operator()(int r, int k) const {
        const int i = k0 + 1 + k;
        if (i >= n) return 0.0;
        return r < kHbNb ? Y[i + (size_t)r * n] : V[i + (size_t)(r - kHbNb) * n];
    }
};
struct HbVCols {
    const double *V;
    int n, k0;
    __device__ __forceinline__ double operator()(int r, int k) const {
        const int i = k0 + 1 + k;
        return i < n ? V[i + (size_t)r * n] : 0.0;
    }
    __device__ __forceinline__ int first(int) const { return 0; }
};
// [T^T, -T^T (V^T Y)], 64 x 128.
struct HbM1 {
    const double *M;
    __device__ __forceinline__ double operator()(int r, int k) const { return M[r + k * kHbNb]; }
};
// Column j of [W0; V(c1:, :)^T].
struct HbB1 {
    const double *Wp, *V;
    int nz, n, c1;
    long long cz;
    __device__ __forceinline__ double operator()(int r, int k) const {
        if (k >= kHbNb) return V[c1 + r + (size_t)(k - kHbNb) * n];
        double s = 0.0;
        for (int z = 0; z < nz; ++z) s += Wp[(size_t)z * cz + k + (size_t)r * kHbNb];
        return s;
    }
};
// Row i of [Y V], column j of [V(c1:, :)^T; Z].
struct HbA2 {
    const double *Y, *V;
    int n;
    __device__ __forceinline__ double operator()(int r, int k) const {
        return k < kHbNb ? Y[r + (size_t)k * n] : V[r + (size_t)(k - kHbNb) * n];
    }
};
struct HbB2 {
    const double *V, *Z;
    int n, c1;
    __device__ __forceinline__ double operator()(int r, int k) const {
        return k < kHbNb ? V[c1 + r + (size_t)k * n] : Z[k - kHbNb + (size_t)r * kHbNb];
    }
};

// M1 = [T^T, -T^T VY] (VY: the last 64 columns of W0), eight columns per CTA,
// and their exponents.
__global__ void __launch_bounds__(8 * kHbNb) k_hb_m1(const double *T, const double *VYp, int nz, long long cz, double *M,
                                                     int *dk) {
    __shared__ double vy[8][kHbNb];
    __shared__ int red[8][2];
    const int q = threadIdx.x % kHbNb, c = threadIdx.x / kHbNb, k = blockIdx.x * 8 + c;
    double v;
    if (k < kHbNb) {
        v = T[k + q * kHbNb];
    } else {
        double s = 0.0;
#pragma unroll 4
        for (int z = 0; z < nz; ++z) s += VYp[(size_t)z * cz + q + (size_t)(k - kHbNb) * kHbNb];
        vy[c][q] = s;
    }
    __syncthreads();
    if (k >= kHbNb) {
        double a0 = 0.0, a1 = 0.0;
        for (int p = 0; p < kHbNb; p += 2) {
            a0 = fma(T[p + q * kHbNb], vy[c][p], a0);
            a1 = fma(T[p + 1 + q * kHbNb], vy[c][p + 1], a1);
        }
        v = -(a0 + a1);
    }
    M[q + k * kHbNb] = v;
    const int m = __reduce_max_sync(0xffffffffu, dg_exp(v));
    if ((q & 31) == 0) red[c][q >> 5] = m;
    __syncthreads();
    if (q == 0) dk[k] = max(red[c][0], red[c][1]);
}

// The scratch of one reduction, laid out once.
struct HbDigits {
    unsigned char *AD, *VN, *M1, *B1, *A2, *B2;
    double *Wp, *M, *Z;
    unsigned *top;                                               // rows' largest high words
    int *low, *uneven;                                           // k_hb_even's counts and result
    int *cex, *exM1, *exB, *exA2, *dk1;                          // cex: n columns of A, then [Y V]
    int cch;
};
size_t hb_digits_layout(int n, bool fix, unsigned char *base, HbDigits &D) {
    const size_t rows16 = (size_t)((n + kDgBK - 1) / kDgBK) * kDgBK * kDgDigits * 2;   // bytes of one column's digits
    const size_t all = (size_t)(n + kHbNb + kDgBM - 1) / kDgBM * kDgBM;
    const size_t fit = std::max<size_t>(1, kHbDigitBytes / (rows16 * kDgBM)) * kDgBM;
    D.cch = (int)std::min(all, fit);
    const size_t small = (size_t)2 * kHbNb * kDgDigits * 2;      // bytes of one 128-column row's digits
    size_t off = 0;
    const auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) / 256 * 256;
        return base + o;
    };
    // The same place serves A's columns in fixed point while a panel runs (fix:
    // 8 n^2 bytes, 5 GB at the largest order whose panel is one launch).
    D.AD = take(std::max((size_t)D.cch * rows16, fix ? (size_t)n * n * sizeof(int2) : 0));
    D.VN = take((size_t)kDgBN * rows16);
    D.M1 = take((size_t)kDgBM * small);
    D.B1 = take(all * small);
    D.A2 = take(all * small);
    D.B2 = take(all * small);
    D.Wp = reinterpret_cast<double *>(take((size_t)kHbParts * kHbNb * all * 8));
    D.M = reinterpret_cast<double *>(take((size_t)2 * kHbNb * kHbNb * 8));
    D.Z = reinterpret_cast<double *>(take((size_t)kHbNb * all * 8));
    D.cex = reinterpret_cast<int *>(take((size_t)(n + 2 * kHbNb) * sizeof(int)));
    D.exM1 = reinterpret_cast<int *>(take((size_t)kDgBM * sizeof(int)));
    D.exB = reinterpret_cast<int *>(take(all * sizeof(int)));
    D.exA2 = reinterpret_cast<int *>(take(all * sizeof(int)));
    D.dk1 = reinterpret_cast<int *>(take((size_t)2 * kHbNb * sizeof(int)));
    D.top = reinterpret_cast<unsigned *>(take((size_t)n * sizeof(unsigned)));
    D.low = reinterpret_cast<int *>(take((size_t)(2 * n + 2) * sizeof(int)));   // the last two: counter, result
    D.uneven = D.low + 2 * n + 1;
    return off;
}
// The trailing columns c1 .. n-1 of panel k0, where the matrix is even.
cudaError_t hb_trailing(const HbState &S, const HbDigits &D, int k0, int c1, int sms, cudaStream_t st) {
    const int n = S.n, m = n - c1, kr = n - k0 - 1, total = m + kHbNb;
    const int steps = (kr + kDgBK - 1) / kDgBK;
    constexpr int ksteps = 2 * kHbNb / kDgBK;
    const int *exY = D.cex + n, *exV = exY + kHbNb;
    k_dg_exp_k<<<2 * kHbNb, 256, 0, st>>>(HbPanelCols{S.Y, S.V, n, k0}, kr, nullptr, 0, D.cex + n);
    k_dg_split<HbVCols, false><<<dim3(kDgBN / 8, (unsigned)((2 * steps + 31) / 32)), 256, 0, st>>>(
        HbVCols{S.V, n, k0}, kDgBN, kDgBN, steps, exV, nullptr, 0, kHbNb, kr, D.VN);
    int per = 0;
    const int tiles = (std::min(total, D.cch) + kDgBM - 1) / kDgBM;
    const int nz = dg_parts(tiles, sms, kHbParts, steps, per);
    const long long cz = (long long)kHbNb * total;
    for (int c = 0; c < total; c += D.cch) {
        const int cols = std::min(D.cch, total - c), mb = (cols + kDgBM - 1) / kDgBM;
        k_dg_split<HbTrail, false><<<dim3(mb * (kDgBM / 8), (unsigned)((2 * steps + 31) / 32)), 256, 0, st>>>(
            HbTrail{S.A, S.Y, S.lda, n, k0, c1 + c}, kDgBM, mb * kDgBM, steps, D.cex + c1 + c, nullptr, 0, cols, kr, D.AD);
        const DgStoreLong e{mb, 1, steps, per, cols, kHbNb, D.cex + c1 + c, exV, D.Wp + (size_t)kHbNb * c, kHbNb, 1, cz};
        const cudaError_t err = dg_gemm(mb * nz, sms, D.AD, D.VN, e, D.uneven, st);
        if (err != cudaSuccess) return err;
    }
    k_hb_m1<<<2 * kHbNb / 8, 8 * kHbNb, 0, st>>>(S.T, D.Wp + (size_t)kHbNb * m, nz, cz, D.M, D.dk1);
    k_dg_small<HbM1, true><<<kDgBM / 32, 512, 0, st>>>(HbM1{D.M}, kDgBM, kHbNb, kDgBM, 2 * kHbNb, D.dk1, -1, D.exM1, D.M1);
    const int nb = (m + kDgBN - 1) / kDgBN, rb = (n + kDgBM - 1) / kDgBM;
    k_dg_small<HbB1, false><<<nb * (kDgBN / 8), 128, 0, st>>>(HbB1{D.Wp, S.V, nz, n, c1, cz}, kDgBN, m, nb * kDgBN,
                                                              2 * kHbNb, D.dk1, 1, D.exB, D.B1);
    const DgStoreShort ez{1, nb, ksteps, ksteps, kHbNb, m, D.exM1, D.exB, D.Z, 1, kHbNb, 0};
    cudaError_t err = dg_gemm(nb, sms, D.M1, D.B1, ez, D.uneven, st);
    if (err != cudaSuccess) return err;
    k_dg_small<HbA2, true><<<rb * (kDgBM / 32), 512, 0, st>>>(HbA2{S.Y, S.V, n}, kDgBM, n, rb * kDgBM, 2 * kHbNb, D.cex + n,
                                                              -1, D.exA2, D.A2);
    k_dg_small<HbB2, false><<<nb * (kDgBN / 8), 128, 0, st>>>(HbB2{S.V, D.Z, n, c1}, kDgBN, m, nb * kDgBN, 2 * kHbNb,
                                                              D.cex + n, 1, D.exB, D.B2);
    const DgUpdate eu{rb, ksteps, n, m, D.exA2, D.exB, S.A + (size_t)c1 * S.lda, S.lda, D.cex + c1, k0 + 1};
    err = dg_gemm(rb * nb, sms, D.A2, D.B2, eu, D.uneven, st);
    return err != cudaSuccess ? err : cudaGetLastError();
}

}  // namespace
}  // namespace hsr

using namespace hsr;

extern "C" int hsr_hessenberg_device(int n, double *dA, int lda, double *dtau, void *stream) {
    if (n <= 0 || lda < n || !dA || !dtau) return HSR_ERR_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(dtau, 0, (size_t)n * sizeof(double), st) != cudaSuccess) return HSR_ERR_CUDA;
    if (n <= 2) return HSR_OK;
    static thread_local Scratch sc;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return HSR_ERR_CUDA;
    const int nblk = (n + kHbRows - 1) / kHbRows;
    const int maxch = (n + kHbChunk - 1) / kHbChunk;
    const size_t nb = kHbNb;
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // The one-launch panel: CTAs, rows per CTA, rows per tile of A v.
    // Rows: every CTA with rows adds one part to the sums that each of them
    // forms, 48 clocks of the FP64 pipe a column, and its own rows cost 80.
    const int ctas = std::max(1, std::min(sms, (n + 3) / 4));
    const int R = std::max((n + ctas - 1) / ctas, (int)(n / (1.3 * std::sqrt((double)n)))), own = (n + R - 1) / R;
    // The lowest row tile that keeps nearly as many CTAs busy as the best one:
    // fewer column shares, whose parts each row adds up.
    const auto busy = [&](int h) {
        const int rt = (n + h - 1) / h;
        return rt <= ctas ? (long long)(ctas / rt) * n / h : 0LL;
    };
    int rpc = 32;
    long long best = 0;
    for (int h = 32; h <= kHbThreads; h *= 2) best = std::max(best, busy(h));
    while (rpc < kHbThreads && 10 * busy(rpc) < 9 * best) rpc *= 2;
    const int rtiles = (n + rpc - 1) / rpc, shares = std::max(1, ctas / rtiles);
    bool one = !without_cooperative() && rtiles <= ctas && hb_panel_smem(R) <= kHbPanelSmem &&
                     cudaFuncSetAttribute(k_hb_panel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kHbPanelSmem) == cudaSuccess &&
                     cudaFuncSetAttribute(k_hb_panel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kHbPanelSmem) == cudaSuccess;
    const size_t need = 2 * (size_t)n * nb           // Y, V
                        + nb * nb                     // T
                        + (size_t)n                   // c
                        + 2 * (size_t)std::max(nblk, ctas) * nb   // part, part2
                        + 6 * (size_t)std::max(nblk, ctas)        // partn
                        + std::max((size_t)maxch, (size_t)shares) * n   // gpart
                        + nb + 8                      // sc
                        + (size_t)(kHbMaxSplit + 2) * nb * n   // W partials, W, W2
                        + 4;                          // counters
    // The digits' part behind it, where there is memory for it.
    const size_t plain = (need * sizeof(double) + 255) / 256 * 256;
    HbDigits D{};
    const bool fixes = one && n >= kHbFixN;
    const ScratchUse use(sc, n >= kHbDigitsN ? plain + hb_digits_layout(n, fixes, nullptr, D) : plain, plain, dev, st);
    if (!use) return HSR_ERR_NOMEM;
    const bool digits = use.bytes() > plain;
    HbState S{};
    S.A = dA;
    S.lda = lda;
    S.n = n;
    double *p = reinterpret_cast<double *>(use.get());
    S.Y = p; p += (size_t)n * nb;
    S.V = p; p += (size_t)n * nb;
    S.T = p; p += nb * nb;
    S.c = p; p += n;
    S.part = p; p += (size_t)std::max(nblk, ctas) * nb;
    S.part2 = p; p += (size_t)std::max(nblk, ctas) * nb;
    S.partn = p; p += 6 * (size_t)std::max(nblk, ctas);
    S.gpart = p; p += std::max((size_t)maxch, (size_t)shares) * n;
    S.sc = p; p += nb + 8;
    double *Wp = p; p += (size_t)kHbMaxSplit * nb * n;
    double *W = p; p += nb * (size_t)n;
    double *W2 = p; p += nb * (size_t)n;
    S.cnt = reinterpret_cast<unsigned int *>(p);
    S.tau = dtau;
    if (cudaMemsetAsync(S.cnt, 0, 4 * sizeof(double), st) != cudaSuccess) return HSR_ERR_CUDA;
    if (digits) {
        hb_digits_layout(n, fixes, use.get() + plain, D);
        // Exponents of A's columns over the rows that reflectors touch.
        k_dg_exp_k<<<n, 256, 0, st>>>(HqCols{dA + 1, lda, n, n - 1}, n - 1, nullptr, 0, D.cex);
        if (cudaMemsetAsync(D.low, 0, (size_t)(2 * n + 2) * sizeof(int), st) != cudaSuccess) return HSR_ERR_CUDA;
        k_hb_even<<<even_grid(n - 1, n, sms), 256, 0, st>>>(
            n, dA, lda, D.cex, D.low, reinterpret_cast<unsigned *>(D.low + 2 * n), D.uneven);
    }
    for (int k0 = 0; k0 < n - 2; k0 += kHbNb) {
        const int ib = std::min(kHbNb, n - 2 - k0);
        if (cudaMemsetAsync(S.V, 0, (size_t)n * nb * sizeof(double), st) != cudaSuccess ||
            cudaMemsetAsync(S.T, 0, nb * nb * sizeof(double), st) != cudaSuccess)
            return HSR_ERR_CUDA;
        if (ib < kHbNb &&                                        // columns a short panel leaves unwritten
            cudaMemsetAsync(S.Y + (size_t)ib * n, 0, (size_t)(kHbNb - ib) * n * sizeof(double), st) != cudaSuccess)
            return HSR_ERR_CUDA;
        if (one) {
            const bool fix = digits && fixes;
            HbPanel pp{S, k0, ib, R, own, rpc, rtiles, shares, S.cnt + 2, reinterpret_cast<const int2 *>(D.AD), D.top,
                       fix ? D.uneven : nullptr};
            void *args[] = {&pp};
            const auto panel = [&](const void *fn) {
                return cudaLaunchCooperativeKernel(fn, dim3(ctas), dim3(kHbThreads), args, hb_panel_smem(R), st);
            };
            // (First: where it is refused, neither form runs.)
            const cudaError_t e = panel(reinterpret_cast<const void *>(k_hb_panel<false>));
            if (refused(e)) {
                cudaGetLastError();
                one = false;
            } else if (e != cudaSuccess) {
                return HSR_ERR_CUDA;
            } else if (fix) {
                const dim3 g((unsigned)(n + 255) / 256, (unsigned)((n - k0 - 1 + kFixCols - 1) / kFixCols));
                if (cudaMemsetAsync(D.top, 0, (size_t)n * sizeof(unsigned), st) != cudaSuccess) return HSR_ERR_CUDA;
                k_hb_fix_top<<<g, 256, 0, st>>>(n, dA, lda, k0 + 1, D.top, D.uneven);
                k_hb_fix<<<g, 256, 0, st>>>(n, dA, lda, k0 + 1, D.top, reinterpret_cast<int2 *>(D.AD), D.uneven);
                if (panel(reinterpret_cast<const void *>(k_hb_panel<true>)) != cudaSuccess) return HSR_ERR_CUDA;
            }
        }
        if (!one) {
            int nchp = 0;
            for (int i = 0; i < ib; ++i) {
                const int j = k0 + i;
                const int nch = (n - j - 1 + kHbChunk - 1) / kHbChunk;
                k_hb_step<<<nblk, kHbRows, 0, st>>>(S, k0, i - 1, i, nchp);
                k_hb_larfg<<<nblk, kHbRows, 0, st>>>(S, k0, i, j);
                k_hb_gemv<<<dim3(nblk, nch), kHbRows, 0, st>>>(S, k0, i, j);
                nchp = nch;
            }
            k_hb_step<<<nblk, kHbRows, 0, st>>>(S, k0, ib - 1, -1, nchp);
        }
        const int c1 = k0 + ib, m = n - c1;
        if (m <= 0) continue;
        if (digits && hb_trailing(S, D, k0, c1, sms, st) != cudaSuccess) return HSR_ERR_CUDA;
        // In FP64, where the matrix is not even or there are no digits.
        const int kr = n - k0 - 1, mt = (m + kHbTm - 1) / kHbTm;
        const int split = std::max(1, std::min((2 * sms + mt - 1) / mt, std::min(kHbMaxSplit, (kr + kHbTk - 1) / kHbTk)));
        const HbPlain hp{S, k0, ib, c1, split, Wp, W, W2, S.cnt + 4, digits ? D.uneven : nullptr};
        const int nt = (n + kHbTm - 1) / kHbTm;
        const int grid = std::min(sms, nt * std::max(nt, kHbMaxSplit));   // the same for all panels (GridBar)
        if (launch_phases(k_hb_plain, hp, kHbPlainPhases, grid, st) != cudaSuccess) return HSR_ERR_CUDA;
    }
    return cudaGetLastError() == cudaSuccess ? HSR_OK : HSR_ERR_CUDA;
}

extern "C" int hsr_hessenberg_apply_q_device(int n, const double *dA, int lda, const double *dtau, int ncols,
                                             double *dX, int ldx, void *stream) {
    if (n <= 0 || lda < n || ncols < 0 || ldx < n || !dA || !dtau || (ncols > 0 && !dX)) return HSR_ERR_ARG;
    if (ncols == 0 || n <= 2) return HSR_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    static thread_local Scratch sc;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return HSR_ERR_CUDA;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t nb = kHbNb;
    const size_t need = (size_t)n * nb + 2 * nb * nb + (size_t)kHbMaxSplit * nb * nb +
                        (size_t)(kHbMaxSplit + 2) * nb * ncols + 1;
    const size_t plain = (need * sizeof(double) + 255) / 256 * 256;
    HqDigits D{};
    const ScratchUse use(sc, n >= kHqDigitsN ? plain + hq_digits_layout(n, ncols, nullptr, D) : plain, plain, dev, st);
    if (!use) return HSR_ERR_NOMEM;
    const int *uneven = nullptr;
    if (use.bytes() > plain) {
        hq_digits_layout(n, ncols, use.get() + plain, D);
        if (hq_digits(D, n, dA, lda, dtau, ncols, dX, ldx, sms, st, &uneven) != cudaSuccess) return HSR_ERR_CUDA;
    }
    // In FP64, where the reflectors are not even or there are no digits.
    HqPlain P{};
    P.n = n, P.ncols = ncols, P.A = dA, P.lda = lda, P.tau = dtau, P.X = dX, P.ldx = ldx, P.uneven = uneven;
    P.V = reinterpret_cast<double *>(use.get()), P.G = P.V + (size_t)n * nb, P.T = P.G + nb * nb, P.Gp = P.T + nb * nb;
    P.Wp = P.Gp + (size_t)kHbMaxSplit * nb * nb, P.W = P.Wp + (size_t)kHbMaxSplit * nb * ncols;
    P.W2 = P.W + nb * (size_t)ncols;
    P.bar = reinterpret_cast<unsigned *>(P.W2 + nb * (size_t)ncols);
    const int ct = (ncols + kHbTm - 1) / kHbTm, rt = (n + kHbTm - 1) / kHbTm;
    P.splitg = std::min(2 * sms, kHbMaxSplit);
    P.splitw = std::max(1, std::min((2 * sms + ct - 1) / ct, kHbMaxSplit));
    if (uneven) P.bar = reinterpret_cast<unsigned *>(D.low + 2 * n + 2);         // zeroed with the counts
    if ((!uneven && cudaMemsetAsync(P.bar, 0, sizeof(double), st) != cudaSuccess) ||
        launch_phases(k_hq_plain, P, kHqPlainPhases * ((n - 3) / kHbNb + 1), std::min(sms, ct * std::max(rt, kHbMaxSplit)), st) !=
            cudaSuccess)
        return HSR_ERR_CUDA;
    return cudaGetLastError() == cudaSuccess ? HSR_OK : HSR_ERR_CUDA;
}
