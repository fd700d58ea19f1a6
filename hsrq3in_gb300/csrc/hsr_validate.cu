// hsr_validate.cu -- residuals of computed eigenpairs on the device.
//
// For every column k:  res_k = ||H x_k - lambda_k x_k||_2 / (||H||_F ||x_k||_2),
// the bound form of validation.c:145-166 (without |lambda| in the denominator,
// which makes it the stricter of the two).  Only the Hessenberg part of H
// (i <= j+1) enters, as in the solver.  Inputs of any magnitude are safe:
// H is scaled by 2^-e(max|H|) and each x_k by 2^-e(max|x_k|) before anything
// is multiplied, so every product and partial sum stays below 4n; the ratio
// is invariant under those exact power-of-two scalings.  A non-finite entry
// of H or x_k gives NaN for the column, a zero x_k gives +Inf.
//
// Launches on the caller's stream, no synchronisation:
//   k_val_max    max |H_ij| over the Hessenberg part and max |x_ik| per column
//   k_val_sums   sum of squares of the scaled H and of each scaled x_k
//   then r = H x - lambda x and its sum of squares per column, either
//   k_dg_exp_*, k_dg_split, k_val_cols, k_dg_gemm   on the bf16 tensor cores
//                by digits (hsr_digits.cuh), or
//   k_val_gemm   on 64 x 32 tiles (DFMA, K in chunks of 32 from the
//                subdiagonal on)
//   k_val_final  the ratio
// The digit product takes over at order 128 (kValDigitsN), for any number of
// columns: below, its seven more launches cost more than the product (n = 64:
// 69 us against 60; n = 128: 76 against 93; n = 1000 with 1000 columns: 173
// against 2,127; n = 5000 with 5000 columns: 4.22 ms against 114.7).  The DFMA
// form also stays for a scratch buffer that cannot be had.  Error of the
// residuals against a double-double evaluation, n = 3000: 1.4e-13 relative,
// DFMA 1.1e-12.
// The sums use floating-point atomics, so the last bits of a residual may
// differ between runs; the residual is a diagnostic, not a solver output.
#include "../../include/hsrq3in_gb300.h"
#include "hsr_device.cuh"
#include "hsr_digits.cuh"
#include "hsr_scratch.h"

#include <algorithm>
#include <cmath>
#include <cuda_runtime.h>

namespace hsr {
namespace {

constexpr int kValDigitsN = 128;      // smallest order of the digit product
// Most scratch for digits of H's rows and of x's columns at a time.
constexpr size_t kValHBytes = (size_t)2 << 30, kValXBytes = (size_t)1 << 30;
constexpr int kValRows = 64, kValCols = 32, kValK = 32;

__device__ __forceinline__ unsigned long long block_umax(unsigned long long v, unsigned long long *red) {
    for (int o = 16; o; o >>= 1) v = umax64(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        v = lane < nw ? red[lane] : 0ULL;
        for (int o = 16; o; o >>= 1) v = umax64(v, __shfl_xor_sync(0xffffffffu, v, o));
    }
    return v;   // valid in warp 0
}

__device__ __forceinline__ double block_sum(double v, double *red) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        v = lane < nw ? red[lane] : 0.0;
        for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    return v;   // valid in warp 0
}

// |x| bit pattern with NaN kept above +Inf (any non-finite value wins).
__device__ __forceinline__ unsigned long long mag_bits(double x) { return mag(x); }

// 2^-e(m) for the largest magnitude m (as bits): the exact power of two that
// brings m into [1, 2), at most 2^1022 (a subnormal m stays below 1); 1 for
// m = 0 or a non-finite m.
__device__ __forceinline__ double inv_pow2_of(unsigned long long m) {
    if (m == 0 || m >= kInfBits) return 1.0;
    return ldexp(1.0, -max(ilogb(from_bits(m)), -1022));
}

// Blocks [0, n): column j of H, rows 0 .. min(j+1, n-1).  Blocks [n, n+ncols): column of X.
__global__ void k_val_max(int n, const double *H, long long ldh, int ncols, const double *X, long long ldx,
                          unsigned long long *hmax, unsigned long long *xmax, int *hcol) {
    __shared__ unsigned long long red[32];
    const int j = blockIdx.x;
    unsigned long long m = 0;
    if (j < n) {
        const int rows = min(j + 2, n);
        const double *c = H + (size_t)j * ldh;
        for (int i = threadIdx.x; i < rows; i += blockDim.x) m = umax64(m, mag_bits(c[i]));
    } else {
        const double *c = X + (size_t)(j - n) * ldx;
        for (int i = threadIdx.x; i < n; i += blockDim.x) m = umax64(m, mag_bits(c[i]));
    }
    m = block_umax(m, red);
    if (threadIdx.x == 0) {
        if (j < n) {
            atomicMax(hmax, m);
            if (hcol) hcol[j] = (m == 0 || m >= kInfBits) ? 0 : max((int)(m >> 52), 1) - 1023;
        } else {
            xmax[j - n] = m;
        }
    }
}

__global__ void k_val_sums(int n, const double *H, long long ldh, int ncols, const double *X, long long ldx,
                           const unsigned long long *hmax, const unsigned long long *xmax, double *hsum,
                           double *xsum) {
    __shared__ double red[32];
    const int j = blockIdx.x;
    double s = 0.0;
    if (j < n) {
        const double sc = inv_pow2_of(*hmax);
        const int rows = min(j + 2, n);
        const double *c = H + (size_t)j * ldh;
        for (int i = threadIdx.x; i < rows; i += blockDim.x) {
            const double t = c[i] * sc;
            s = fma(t, t, s);
        }
    } else {
        const double sc = inv_pow2_of(xmax[j - n]);
        const double *c = X + (size_t)(j - n) * ldx;
        for (int i = threadIdx.x; i < n; i += blockDim.x) {
            const double t = c[i] * sc;
            s = fma(t, t, s);
        }
    }
    s = block_sum(s, red);
    if (threadIdx.x == 0) {
        if (j < n) atomicAdd(hsum, s);
        else xsum[j - n] = s;
    }
}

// CTA: rows [r0, r0+64) x columns [c0, c0+32); thread: one row, 8 columns.
__global__ void __launch_bounds__(256) k_val_gemm(int n, const double *H, long long ldh, int ncols,
                                                  const double *wr, const double *X, long long ldx,
                                                  const unsigned long long *hmax, const unsigned long long *xmax,
                                                  double *rsum) {
    __shared__ double As[kValK][kValRows];
    __shared__ double Bs[kValK][kValCols + 1];
    __shared__ double xsc[kValCols];
    const int tid = threadIdx.x;
    const int r0 = blockIdx.x * kValRows, c0 = blockIdx.y * kValCols;
    const int row = tid & (kValRows - 1), cg = tid >> 6;       // 4 groups of 8 columns
    const double sh = inv_pow2_of(*hmax);
    if (tid < kValCols) xsc[tid] = c0 + tid < ncols ? inv_pow2_of(xmax[c0 + tid]) : 1.0;
    __syncthreads();
    double acc[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c] = 0.0;
    const int kstart = (max(r0 - 1, 0) / kValK) * kValK;      // H(i, k) = 0 for k < i-1
    for (int k0 = kstart; k0 < n; k0 += kValK) {
        // H(r0 .. r0+63, k0 .. k0+31), Hessenberg part only, scaled.
        for (int e = tid; e < kValK * kValRows; e += blockDim.x) {
            const int i = e & (kValRows - 1), kk = e >> 6;
            const int gi = r0 + i, gk = k0 + kk;
            double v = 0.0;
            if (gi < n && gk < n && gk >= gi - 1) v = H[gi + (size_t)gk * ldh] * sh;
            As[kk][i] = v;
        }
        // X(k0 .. k0+31, c0 .. c0+31), each column scaled.
        for (int e = tid; e < kValK * kValCols; e += blockDim.x) {
            const int kk = e & (kValK - 1), c = e >> 5;
            const int gk = k0 + kk, gc = c0 + c;
            Bs[kk][c] = (gk < n && gc < ncols) ? X[gk + (size_t)gc * ldx] * xsc[c] : 0.0;
        }
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < kValK; ++kk) {
            const double a = As[kk][row];
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[c] = fma(a, Bs[kk][cg * 8 + c], acc[c]);
        }
        __syncthreads();
    }
    const int gi = r0 + row;
    const int lane = tid & 31;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        const int gc = c0 + cg * 8 + c;
        double r2 = 0.0;
        if (gi < n && gc < ncols) {
            const double xs = X[gi + (size_t)gc * ldx] * xsc[cg * 8 + c];
            const double r = fma(-(wr[gc] * sh), xs, acc[c]);
            r2 = r * r;
        }
        for (int o = 16; o; o >>= 1) r2 += __shfl_xor_sync(0xffffffffu, r2, o);
        if (lane == 0 && gc < ncols) atomicAdd(&rsum[gc], r2);
    }
}

__global__ void k_val_final(int ncols, const unsigned long long *hmax, const unsigned long long *xmax,
                            const double *hsum, const double *xsum, const double *rsum, double *res) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= ncols) return;
    const unsigned long long hm = *hmax, xm = xmax[k];
    double r;
    if (hm >= kInfBits || xm >= kInfBits) r = __longlong_as_double(0x7ff8000000000000LL);   // NaN
    else if (xm == 0) r = __longlong_as_double(0x7ff0000000000000LL);                      // +Inf
    else if (hm == 0) r = sqrt(rsum[k]) / sqrt(xsum[k]);                                    // H = 0: ||lambda x||/||x||
    else r = sqrt(rsum[k]) / (sqrt(*hsum) * sqrt(xsum[k]));
    res[k] = r;
}

// ------------------------------------------------------- digit product
// H x on the tensor cores (hsr_digits.cuh).  A: rows of H, its columns evened
// out by their largest entries' exponents (hcol), which go into x instead, so
// that a graded H loses nothing; B: columns of x.
struct ValH {
    const double *H;
    long long ld;
    int n, row0;
    __device__ __forceinline__ double operator()(int r, int k) const {
        const int i = row0 + r;
        return (i < n && k < n && k >= i - 1) ? H[i + (size_t)k * ld] : 0.0;
    }
    __device__ __forceinline__ int first(int r) const { return max(row0 + r - 1, 0); }
};
struct ValX {
    const double *X;
    long long ld;
    int n, cols;
    __device__ __forceinline__ double operator()(int r, int k) const {
        return (r < cols && k < n) ? X[k + (size_t)r * ld] : 0.0;
    }
    __device__ __forceinline__ int first(int) const { return 0; }
};
// Per column of a chunk, once: -lambda scaled as H, and the exponents that
// scale a column of x and a column of the product.
struct ValCol {
    double nlam;
    int ex, ep;
};
__global__ void k_val_cols(int cols, const double *wr, const unsigned long long *hmax, const unsigned long long *xmax,
                           const int *xex, ValCol *col) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cols) return;
    const double sh = inv_pow2_of(*hmax), xs = inv_pow2_of(xmax[c]);
    const int esh = (int)((ubits(sh) >> 52) & 0x7ff) - 1023, exs = (int)((ubits(xs) >> 52) & 0x7ff) - 1023;
    col[c] = ValCol{-(wr[c] * sh), exs, max(xex[c], kDgZero) + exs + esh - 2044};
}
// r = H x - lambda x of a tile (scaled by the exact powers of two of H and x),
// its sum of squares per column.  Tiles in row-block order: the longest (the
// first rows) first, and CTAs that run together share H's digits.
struct ValEpi {
    using Sum = DgTwo<16>;
    static constexpr int kWarps = 16;
    int row0, rows, cols, steps, cblocks;
    const double *X;
    long long ldx;
    const int *hex;
    const ValCol *col;
    double *rsum;
    __device__ __forceinline__ DgTile tile(int t) const {
        const int bx = t / cblocks;
        const int by = t - bx * cblocks, s0 = max(row0 + bx * kDgBM - 1, 0) / kDgBK;
        return DgTile{bx, by, 0, (long long)bx * steps + s0, (long long)by * steps + s0, steps - s0};
    }
    __device__ __forceinline__ void finish(const DgTile &, int row, int col0, const Sum &sum) const {
        const bool in = row < rows;
        const int lane = threadIdx.x & 31;
        const int er = in ? max(hex[row], kDgZero) : 0;
        constexpr int NC = Sum::kCols;
        double r2[NC];
        // Eight columns at a time, their x loaded ahead of the arithmetic (one
        // load at a time pays its latency for every column).
#pragma unroll
        for (int c0 = 0; c0 < NC; c0 += 8) {
            double x[8];
#pragma unroll
            for (int c = 0; c < 8; ++c)
                x[c] = X[row0 + min(row, rows - 1) + (size_t)min(col0 + c0 + c, cols - 1) * ldx];
#pragma unroll
            for (int c = 0; c < 8; ++c) {
                const ValCol k = col[min(col0 + c0 + c, cols - 1)];
                const double r = fma(k.nlam, dg_ldexp(x[c], k.ex), sum.value(c0 + c, er + k.ep));
                r2[c0 + c] = in ? r * r : 0.0;
            }
        }
        // Sum over the warp's rows: lanes l and l + 16 end with halves of
        // column l mod 16, added last.
        static_assert(NC == 16, "the exchange below");
#pragma unroll
        for (int o = NC / 2; o; o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int c = 0; c < NC / 2; ++c) {
                if (c >= o) break;
                const double keep = up ? r2[c + o] : r2[c], send = up ? r2[c] : r2[c + o];
                r2[c] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        r2[0] += __shfl_xor_sync(0xffffffffu, r2[0], 16);
        if (lane < NC && col0 + lane < cols) atomicAdd(&rsum[col0 + lane], r2[0]);
    }
    __device__ void poison(int thread, int threads) const {
        for (int c = thread; c < cols; c += threads) rsum[c] = __longlong_as_double(0x7ff8000000000000LL);
    }
};

}  // namespace
}  // namespace hsr

using namespace hsr;

extern "C" int hsr_residuals_device(int n, const double *dH, int lddH, int ncols, const double *dwr,
                                    const double *dX, int lddX, double *d_res, void *stream) {
    if (n <= 0 || lddH < n || ncols < 0 || lddX < n || !dH || (ncols > 0 && (!dwr || !dX || !d_res)))
        return HSR_ERR_ARG;
    if (ncols == 0) return HSR_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    static thread_local Scratch sc;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return HSR_ERR_CUDA;
    // Digits: rows of H and columns of x in chunks of at most kValHBytes and
    // kValXBytes, exponents (hcol, hex, xex) beside them; behind the sums, where
    // there is memory for it.
    const long long steps = (n + kDgBK - 1) / kDgBK;
    const size_t per_row = (size_t)steps * kDgBK * kDgDigits * 2;
    const auto chunk = [&](size_t cap, int count, int block) {
        const size_t most = std::max<size_t>(1, cap / (per_row * block)) * block;
        return (int)std::min<size_t>(most, (size_t)((count + block - 1) / block) * block);
    };
    const int rch = chunk(kValHBytes, n, kDgBM), cch = chunk(kValXBytes, ncols, kDgBN);
    const size_t hbytes = (size_t)rch * per_row, xbytes = (size_t)cch * per_row;
    const size_t sums = ((size_t)(2 + 3 * (size_t)ncols) * 8 + 255) / 256 * 256;
    const size_t dbytes = hbytes + xbytes + (size_t)cch * sizeof(ValCol) + (size_t)(n + rch + cch) * sizeof(int);
    const ScratchUse use(sc, n < kValDigitsN ? sums : sums + dbytes, sums, dev, st);
    if (!use) return HSR_ERR_NOMEM;
    const bool digits = use.bytes() > sums;
    unsigned long long *hmax = reinterpret_cast<unsigned long long *>(use.get());
    double *hsum = reinterpret_cast<double *>(hmax + 1);
    unsigned long long *xmax = hmax + 2;
    double *xsum = reinterpret_cast<double *>(xmax + ncols);
    double *rsum = xsum + ncols;
    if (cudaMemsetAsync(hmax, 0, 16, st) != cudaSuccess ||
        cudaMemsetAsync(rsum, 0, (size_t)ncols * 8, st) != cudaSuccess)
        return HSR_ERR_CUDA;
    unsigned char *hdig = use.get() + sums, *xdig = hdig + hbytes;
    ValCol *vcol = reinterpret_cast<ValCol *>(xdig + xbytes);
    int *hcol = digits ? reinterpret_cast<int *>(vcol + cch) : nullptr, *hex = hcol + n, *xex = hex + rch;
    int sms = 1;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    k_val_max<<<n + ncols, 256, 0, st>>>(n, dH, lddH, ncols, dX, lddX, hmax, xmax, hcol);
    k_val_sums<<<n + ncols, 256, 0, st>>>(n, dH, lddH, ncols, dX, lddX, hmax, xmax, hsum, xsum);
    if (digits) {
        for (int r0 = 0; r0 < n; r0 += rch) {
            const int rows = std::min(rch, n - r0), rb = (rows + kDgBM - 1) / kDgBM;
            const ValH lh{dH, lddH, n, r0};
            if (cudaMemsetAsync(hex, 0x80, (size_t)rows * sizeof(int), st) != cudaSuccess) return HSR_ERR_CUDA;
            k_dg_exp_r<<<dim3((rows + 255) / 256, (n + 127) / 128), 256, 0, st>>>(lh, rows, n, 128, hcol, -1, hex);
            k_dg_split<ValH, true><<<dim3(rb * (kDgBM / 32), (unsigned)((2 * steps + 7) / 8)), 256, 0, st>>>(
                lh, kDgBM, rb * kDgBM, steps, hex, hcol, -1, rows, n, hdig);
            for (int c0 = 0; c0 < ncols; c0 += cch) {
                const int cols = std::min(cch, ncols - c0), cb = (cols + kDgBN - 1) / kDgBN;
                const double *Xc = dX + (size_t)c0 * lddX;
                const ValX lx{Xc, lddX, n, cols};
                k_dg_exp_k<<<cols, 256, 0, st>>>(lx, n, hcol, 1, xex);
                k_dg_split<ValX, false><<<dim3(cb * (kDgBN / 8), (unsigned)((2 * steps + 31) / 32)), 256, 0, st>>>(
                    lx, kDgBN, cb * kDgBN, steps, xex, hcol, 1, cols, n, xdig);
                k_val_cols<<<(cols + 127) / 128, 128, 0, st>>>(cols, dwr + c0, hmax, xmax + c0, xex, vcol);
                const ValEpi epi{r0, rows, cols, (int)steps, cb, Xc, lddX, hex, vcol, rsum + c0};
                if (dg_gemm(rb * cb, sms, hdig, xdig, epi, nullptr, st) != cudaSuccess) return HSR_ERR_CUDA;
            }
        }
        k_val_final<<<(ncols + 127) / 128, 128, 0, st>>>(ncols, hmax, xmax, hsum, xsum, rsum, d_res);
        return cudaGetLastError() == cudaSuccess ? HSR_OK : HSR_ERR_CUDA;
    }
    dim3 g((n + kValRows - 1) / kValRows, (ncols + kValCols - 1) / kValCols);
    k_val_gemm<<<g, 256, 0, st>>>(n, dH, lddH, ncols, dwr, dX, lddX, hmax, xmax, rsum);
    k_val_final<<<(ncols + 127) / 128, 128, 0, st>>>(ncols, hmax, xmax, hsum, xsum, rsum, d_res);
    return cudaGetLastError() == cudaSuccess ? HSR_OK : HSR_ERR_CUDA;
}
