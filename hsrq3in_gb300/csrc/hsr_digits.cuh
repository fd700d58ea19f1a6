// hsr_digits.cuh -- FP64 matrix products on the bf16 tensor cores.
//
// The FP64 pipe of this part runs 2 FMAs per clock and SM, the bf16 tensor
// cores 4096.  A product C = A B is therefore split by digits (the
// error-free splitting of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59,
// 2012, with fixed-point digits):
//
//   * every row i of A has an exponent ex_i above all its entries, every
//     column j of B likewise, and an entry becomes the 63-bit fixed-point
//     number t = round(a 2^(62 - ex_i)), |t| <= 2^62;
//   * t is written in eight balanced base-256 digits, -128 .. 127 (the
//     leading one within +-64), each exact in bf16 with its weight
//     2^(-6 - 8 p), p = 0 .. 7;
//   * C is the sum of the digit products (p, q) with p + q <= 7, which the
//     tensor cores accumulate in FP32.  Products with equal p + q = d share
//     an accumulator.  In units of 2^(-12 - 8 d) every term is an integer of
//     at most 2^14 (2^13 with a leading digit), so over 192 columns the sums of
//     d = 0 .. 5 stay below 2^24 and are exact; d = 6 and 7 share one
//     accumulator, whose FP32 rounding (by truncation, some 200 times) lies
//     2^-58 below the leading product.  With d = 5 in that accumulator too
//     the same truncations came to 2^-51 a chunk, more than an FP64 chain's;
//   * every 192 columns the accumulators are added to two 64-bit integers per
//     entry, exactly, so the order of the columns does not matter and results
//     are the same for every tiling.  A sum over at most 128 columns goes into
//     one integer in units of 2^-55 (DgOne), half an ulp of an entry of size
//     1/4 where every product's bound is 1.
//
// What is lost is the rounding of t (2^-63 of the row's largest entry) and
// the products with p + q >= 8 (2^-60 of the largest product).  So the method is
// accurate relative to the largest product of a row and a column, not to the
// sum of their products' magnitudes as an FP64 fma chain is: for operands of
// entries of like size its error is below the chain's, for others it may be far
// above.  Where the columns of A (index k) differ in size a power of two per k
// evens them out (dk, taken out of A and put into B); where a result's small
// entries count the caller checks the sizes first (hsr_hessenberg.cu: k_hb_even,
// k_hq_even).  The residuals need no check: with their columns evened out the
// error in a row is at most 2^-60 sqrt(n) of the largest c_k |x_k|, c_k the
// largest entry of column k, and that of FP64 in the row where c_k lies about
// 2^-53 of it, so the norm of r is no less accurate.
//
// Digits are stored tile by tile in the order in which the tensor cores read
// shared memory (8 x 16-byte core matrices, no swizzle), so that a stage of
// 16 columns is one contiguous block per operand: 128 rows x 16 x 8 digits =
// 32 KB of A and 64 x 16 x 8 = 16 KB of B, moved by cp.async.bulk into a ring
// of four.
//
// Rates: a 128 x 64 tile takes 36 digit products per 16 columns, each
// 128 x 64 x 16, which read 6 KB of shared memory at 128 B per clock: 48
// clocks each, 1728 per stage and 75 FP64-equivalent FMAs per clock and SM,
// against 2 on the FP64 pipe.
#pragma once
#include "hsr_device.cuh"

#include <algorithm>
#include <climits>
#include <cstdint>
#include <cuda_runtime.h>

namespace hsr {

constexpr int kDgDigits = 8;
constexpr int kDgBM = 128, kDgBN = 64, kDgBK = 16;
constexpr int kDgGroups = 7;                       // accumulators: d = 0 .. 5 and d >= 6
constexpr int kDgChunk = 12;                       // stages (of 16 columns) between drains
constexpr int kDgStages = 4;
constexpr int kDgABytes = kDgBM * kDgBK * kDgDigits * 2, kDgBBytes = kDgBN * kDgBK * kDgDigits * 2;
constexpr int kDgSmem = kDgStages * (kDgABytes + kDgBBytes) + 1024;
constexpr int kDgZero = -(1 << 20);                // exponent of an all-zero row
constexpr int kDgBad = 1 << 20;                    // exponent field of a row with an Inf or NaN

// Exponent field of x as an upper bound: |x| < 2^(E - 1022); kDgZero for 0,
// kDgBad for a non-finite x.
__device__ __forceinline__ int dg_exp(double x) {
    const unsigned long long m = mag(x);
    if (m == 0) return kDgZero;
    if (m >= kInfBits) return kDgBad;
    const int e = (int)(m >> 52);
    return e ? e : 1;
}

// Biased digits of x with row exponent ex (field) and column shift dk: byte
// 7 - p of the result is digit p plus 128.  base = ex + dk - 9.
__device__ __forceinline__ unsigned long long dg_digits(double x, int base) {
    const unsigned long long b = ubits(x);
    int e = (int)((b >> 52) & 0x7ff);
    unsigned long long m = b & kSigMask;
    if (e) m |= kHidden;
    else e = 1;
    const int sh = e - base;                       // <= 9
    unsigned long long t;
    if (sh >= 0) t = m << min(sh, 9);
    else {
        const int r = min(-sh, 60);
        t = (m + (1ULL << (r - 1))) >> r;          // nearest
    }
    if (b >> 63) t = 0ULL - t;
    return t + 0x8080808080808080ULL;
}

// The bf16 values of digit p of two entries, packed (first in the low half):
// byte u becomes the float 2^(17-8p) + u 2^(-6-8p), minus 2^(17-8p) +
// 2^(1-8p), which is exact; a digit fits bf16's eight significant bits, so the
// upper half of the float is the bf16 value.
template <int P>
__device__ __forceinline__ unsigned dg_pack(unsigned long long u0, unsigned long long u1) {
    constexpr unsigned base = (unsigned)(127 + 17 - 8 * P) << 23;
    const unsigned b0 = (unsigned)(u0 >> (8 * (7 - P))) & 0xffu, b1 = (unsigned)(u1 >> (8 * (7 - P))) & 0xffu;
    const float off = __uint_as_float(base + 128u);
    const float f0 = __uint_as_float(base + b0) - off, f1 = __uint_as_float(base + b1) - off;
    return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}
template <int P>
__device__ __forceinline__ void dg_store(const unsigned long long (&u)[8], unsigned char *dst, int slice_bytes) {
    uint4 v;
    v.x = dg_pack<P>(u[0], u[1]);
    v.y = dg_pack<P>(u[2], u[3]);
    v.z = dg_pack<P>(u[4], u[5]);
    v.w = dg_pack<P>(u[6], u[7]);
    *reinterpret_cast<uint4 *>(dst + (size_t)P * slice_bytes) = v;
}
// Digits of eight consecutive columns of one row to their places.  dst: the
// 16 bytes of digit 0.
__device__ __forceinline__ void dg_store8(const unsigned long long (&u)[8], unsigned char *dst, int slice_bytes) {
    dg_store<0>(u, dst, slice_bytes);
    dg_store<1>(u, dst, slice_bytes);
    dg_store<2>(u, dst, slice_bytes);
    dg_store<3>(u, dst, slice_bytes);
    dg_store<4>(u, dst, slice_bytes);
    dg_store<5>(u, dst, slice_bytes);
    dg_store<6>(u, dst, slice_bytes);
    dg_store<7>(u, dst, slice_bytes);
}
// Place of (row r, columns 8 c8 ..) in an operand with RB rows per block and
// `steps` stages per row block.
__device__ __forceinline__ size_t dg_place(int r, int c8, int RB, long long steps) {
    const int ks = c8 >> 1, kc = c8 & 1;
    const size_t blk = (size_t)(r / RB) * (size_t)steps + (size_t)ks;
    const int rr = r % RB;
    return blk * (size_t)(RB * kDgBK * kDgDigits * 2) + (size_t)((rr >> 3) * 256 + kc * 128 + (rr & 7) * 16);
}

__device__ __forceinline__ int dg_dk(const int *dk, int k) {     // no scaling by a zero or non-finite column
    const int d = dk[k];
    return d <= -kDgBad / 2 || d >= kDgBad / 2 ? 0 : d;
}

// Digit products are for operands whose entries are of like size; a call that
// leaves the choice to the device passes a word `off` to the products, which
// store nothing where it is not 0 (the caller's other form then runs).  Only
// the warps that store read it, beside the first products: read at the start of
// every product and split it cost the back-transform of n = 5000 1.5%.
__device__ __forceinline__ bool dg_off(const int *off) { return off && *off != 0; }

// ---------------------------------------------------------- preparation
// Exponents and digits of an operand of R rows and K columns, read through a
// loader ld(r, k) (0 outside the operand).  dk (optional): exponents taken
// out of the columns (sign = -1, the A side) or put in (sign = +1, the B
// side).  The row exponents start at a value below kDgZero (bytes 0x80).

// Rows contiguous along k: a block per row.
template <class Ld>
__global__ void __launch_bounds__(256) k_dg_exp_k(Ld ld, int K, const int *dk, int sign, int *ex) {
    __shared__ int red[8];
    const int r = blockIdx.x;
    int m = kDgZero;
    for (int k = threadIdx.x; k < K; k += blockDim.x) {
        const int e = dg_exp(ld(r, k));
        m = max(m, dk && e != kDgZero ? e + sign * dk[k] : e);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) m = max(m, red[w]);
        ex[r] = m;
    }
}
// Columns contiguous along r: a thread per row, a block column per `span`
// columns.  ld.first(r0): the first column that rows r0 .. can have.
template <class Ld>
__global__ void __launch_bounds__(256) k_dg_exp_r(Ld ld, int R, int K, int span, const int *dk, int sign, int *ex) {
    const int r = blockIdx.x * 256 + threadIdx.x;
    const int ka = max((int)(blockIdx.y * span), ld.first(blockIdx.x * 256)), kb = min(K, (int)(blockIdx.y + 1) * span);
    if (r >= R) return;
    int m = kDgZero;
#pragma unroll 4
    for (int k = ka; k < kb; ++k) {
        const int e = dg_exp(ld(r, k));
        m = max(m, dk && e != kDgZero ? e + sign * dk[k] : e);
    }
    if (m > kDgZero) atomicMax(&ex[r], m);
}
// Digits.  RC: lanes along the rows (columns contiguous along r), else lanes
// as 8 rows x 4 groups of eight columns (rows contiguous along k), so that
// both the loads and the 16-byte stores of a warp cover whole sectors.
template <class Ld, bool RC>
__global__ void __launch_bounds__(256) k_dg_split(Ld ld, int RB, int Rpad, long long steps, const int *ex,
                                                  const int *dk, int sign, int R, int K, unsigned char *out) {
    const int t = threadIdx.x;
    const int r = RC ? blockIdx.x * 32 + (t & 31) : blockIdx.x * 8 + (t & 7);
    const int c8 = RC ? blockIdx.y * 8 + (t >> 5) : blockIdx.y * 32 + (t >> 3);
    if (r >= Rpad || c8 >= 2 * steps || c8 * 8 + 7 < ld.first(r / RB * RB) / kDgBK * kDgBK) return;
    double x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = ld(r, c8 * 8 + e);
    const int base = (r < R ? max(ex[r], kDgZero) : 0) - 9;
    unsigned long long u[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int k = c8 * 8 + e;
        u[e] = dg_digits(x[e], dk && k < K ? base - sign * dk[k] : base);
    }
    dg_store8(u, out + dg_place(r, c8, RB, steps), RB * kDgBK * 2);
}

// Exponents and digits in one pass for K <= 128: a thread keeps its eight
// entries between the two.  RC: a CTA takes 32 rows, else 8; its 16 thread
// groups one group of eight columns each.
template <class Ld, bool RC>
__global__ void __launch_bounds__(RC ? 512 : 128) k_dg_small(Ld ld, int RB, int R, int Rpad, int K, const int *dk,
                                                             int sign, int *ex, unsigned char *out) {
    constexpr int ROWS = RC ? 32 : 8;
    __shared__ int red[ROWS][17];
    const int t = threadIdx.x, rr = RC ? t & 31 : t & 7, c8 = RC ? t >> 5 : t >> 3;
    const int r = blockIdx.x * ROWS + rr;
    const int steps = (K + kDgBK - 1) / kDgBK;
    double x[8];
    int m = kDgZero;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int k = c8 * 8 + e;
        x[e] = r < R && k < K ? ld(r, k) : 0.0;
        const int ee = dg_exp(x[e]);
        m = max(m, dk && k < K && ee != kDgZero ? ee + sign * dg_dk(dk, k) : ee);
    }
    red[rr][c8] = m;
    __syncthreads();
    m = kDgZero;
#pragma unroll
    for (int q = 0; q < 16; ++q) m = max(m, red[rr][q]);
    if (c8 == 0 && r < R) ex[r] = m;
    if (c8 >= 2 * steps || r >= Rpad) return;
    unsigned long long u[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const int k = c8 * 8 + e;
        u[e] = dg_digits(x[e], dk && k < K ? m - 9 - sign * dg_dk(dk, k) : m - 9);
    }
    dg_store8(u, out + dg_place(r, c8, RB, steps), RB * kDgBK * 2);
}

// ------------------------------------------------------- tcgen05 wrappers
__device__ __forceinline__ uint64_t dg_desc(uint32_t addr) {
    // K-major, no swizzle: core matrices 128 B apart along K (leading offset),
    // 256 B apart along the rows (stride offset); descriptor version 1.
    return (uint64_t)((addr >> 4) & 0x3fffu) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) |
           ((uint64_t)1 << 46);
}
constexpr uint32_t kDgIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kDgBN >> 3) << 17) |
                              ((uint32_t)(kDgBM >> 4) << 24);   // D f32, A and B bf16, both K-major
__device__ __forceinline__ void dg_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
        ::"r"(d), "l"(a), "l"(b), "r"(kDgIdesc), "r"(acc)
        : "memory");
}
__device__ __forceinline__ void dg_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void dg_ld(uint32_t addr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(addr));
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void dg_ld(uint32_t addr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(addr));
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void dg_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void dg_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void dg_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void dg_bulk(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
// One tile: its row and column block, a part index, the places of its first
// stage in A and B (counted in stages) and the number of stages.
struct DgTile {
    int bx, by, bz;
    long long a, b;
    int stages;
};
// Bounded wait without a device error word: false after the poll limit.
__device__ __forceinline__ bool dg_wait(uint64_t *bar, uint32_t parity) {
    for (long it = 0; it < (1L << 22); ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// x 2^e for any e, results outside the normal range included.
static __host__ __device__ __noinline__ double dg_ldexp_rare(double x, int e) { return ldexp(x, e); }
__device__ __forceinline__ double dg_ldexp(double x, int e) {
    const int f = (int)((ubits(x) >> 52) & 0x7ff);
    if (is_zero(x)) return x;
    if (f == 0 || f + e <= 0 || f + e >= 0x7ff) return dg_ldexp_rare(x, e);
    return from_bits(ubits(x) + ((unsigned long long)(long long)e << 52));
}
// (hi 2^36 + lo) 2^e, e the scale's exponent, on the integer pipe (three
// FP64 instructions less, 64 clocks of a sub-partition each): the sum's sign
// and magnitude, its leading 64 bits, rounded to 53 (ties up; what lies below
// the 64 bits does not enter).  Results outside the normal range: ldexp.
// Both forms compile for the host too, where a test checks them.
__host__ __device__ __forceinline__ int dg_clz(unsigned long long x) {   // x != 0
#ifdef __CUDA_ARCH__
    return __clzll((long long)x);
#else
    return __builtin_clzll(x);
#endif
}
__host__ __device__ __forceinline__ double dg_value(long long hi, long long lo, int e) {
    long long H = hi + (lo >> 36);
    unsigned long long L = (unsigned long long)lo & ((1ULL << 36) - 1);
    const unsigned long long sign = (unsigned long long)H & 0x8000000000000000ULL;
    if (sign) {
        const bool z = L == 0;
        L = z ? 0 : (1ULL << 36) - L;
        H = z ? -H : ~H;
    }
    if (H == 0) {                                                // below 2^36 units
        if (L == 0) return 0.0;
        H = (long long)L;
        L = 0;
        e -= 36;
    }
    const int z = dg_clz((unsigned long long)H);                 // 1 .. 63
    unsigned long long m = ((unsigned long long)H << z) | ((L << 28) >> (64 - z));
    int f = 1023 + 63 + 36 - z + e;
    m = (m >> 11) + ((m >> 10) & 1ULL);                          // 2^52 .. 2^53
    if (f <= 0 || f >= 0x7fe) return dg_ldexp_rare(from_bits(sign | (0x3ffULL << 52)) * (double)m, f - 1075);
    return from_bits(sign | (((unsigned long long)(f - 1) << 52) + m));
}

// The same for one word, T 2^(e - 55), |T| <= 2^62.  The rounding bit is added
// after the shift: bit 63 of a << z is set, so adding it before could carry out.
__host__ __device__ __forceinline__ double dg_value(long long T, int e) {
    if (T == 0) return 0.0;
    const unsigned long long sign = (unsigned long long)T & 0x8000000000000000ULL;
    const unsigned long long a = (unsigned long long)(T < 0 ? -T : T);
    const int z = dg_clz(a);
    unsigned long long m = a << z;
    m = (m >> 11) + ((m >> 10) & 1ULL);                          // 2^52 .. 2^53
    const int f = 1023 + 63 - z - 55 + e;
    if (f <= 0 || f >= 0x7fe) return dg_ldexp_rare(from_bits(sign | (0x3ffULL << 52)) * (double)m, f - 1075);
    return from_bits(sign | (((unsigned long long)(f - 1) << 52) + m));
}

// A thread's sums: kCols columns of one row, as hi 2^-28 + lo 2^-64 ...
template <int N>
struct DgTwo {
    static constexpr int kCols = N;
    long long hi[N], lo[N];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int c = 0; c < N; ++c) hi[c] = lo[c] = 0;
    }
    __device__ __forceinline__ void add(int g, int c, float v) {  // one wide multiply-add each
        const float unit = g == 0 ? 0x1p12f : g == 1 ? 0x1p20f : g == 2 ? 0x1p28f : g == 3 ? 0x1p36f
                         : g == 4 ? 0x1p44f : g == 5 ? 0x1p52f : 0x1p64f;
        const int i = __float2int_rn(v * unit);
        if (g < 3) hi[c] += (long long)i * (1 << (16 - 8 * g));
        else lo[c] += (long long)i * (1 << (g == 6 ? 0 : 28 - 8 * (g - 3)));
    }
    __device__ __forceinline__ double value(int c, int e) const { return dg_value(hi[c], lo[c], e - 64); }
};
// ... or, for at most 128 columns, as T 2^-55.
template <int N>
struct DgOne {
    static constexpr int kCols = N;
    long long T[N];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int c = 0; c < N; ++c) T[c] = 0;
    }
    __device__ __forceinline__ void add(int g, int c, float v) {
        const float unit = g == 0 ? 0x1p12f : g == 1 ? 0x1p20f : g == 2 ? 0x1p28f : g == 3 ? 0x1p36f
                         : g == 4 ? 0x1p44f : g == 5 ? 0x1p52f : 0x1p55f;
        const int i = __float2int_rn(v * unit);
        if (g < 2) T[c] += (long long)((unsigned long long)(unsigned)(i << (11 - 8 * g)) << 32);   // the high word only
        else T[c] += (long long)i * (1 << (g == 6 ? 0 : 27 - 8 * (g - 2)));
    }
    __device__ __forceinline__ double value(int c, int e) const { return dg_value(T[c], e); }
};

// One elected lane of a converged warp.
__device__ __forceinline__ bool dg_elect() {
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(p));
    return p != 0;
}
// The digit products of group G of a stage, by the elected lane.  Unrolled,
// and called with operands that are uniform over the warp, so that they stay
// in uniform registers: issued from a loop, or from code that only one lane
// entered, a product cost 60 to 170 clocks instead of its own 48.
template <int G>
__device__ __forceinline__ void dg_products(uint32_t tmem, uint64_t da, uint64_t db, uint32_t keep) {
#pragma unroll
    for (int d = G; d <= (G == kDgGroups - 1 ? kDgDigits - 1 : G); ++d)
#pragma unroll
        for (int p = 0; p <= d; ++p)
            dg_mma(tmem + (uint32_t)(G * kDgBN), da + (uint64_t)((p * (kDgABytes / kDgDigits)) >> 4),
                   db + (uint64_t)(((d - p) * (kDgBBytes / kDgDigits)) >> 4), d == G && p == 0 ? keep : 1u);
}
// Group G of a chunk's first stage (waits until the last chunk's sum is
// drained and starts a new one) or last stage (commits it).
template <int G>
__device__ __forceinline__ bool dg_group(uint32_t tmem, uint64_t da, uint64_t db, bool begin, bool end, unsigned chunk,
                                         uint64_t *acc_empty, uint64_t *acc_full) {
    bool ok = true;
    if (begin && chunk > 0) {
        ok = dg_wait(&acc_empty[G], (chunk - 1) & 1);
        dg_fence_after();
    }
    if (dg_elect()) {
        dg_products<G>(tmem, da, db, begin ? 0u : 1u);
        if (end) dg_commit(&acc_full[G]);
    }
    __syncwarp();
    return ok;
}

// Tiles of 128 x 64 of A B.  A: digits of row blocks of 128, B: of 64.
// epi.tile(t) gives tile t's blocks and stages; epi.finish takes a thread's
// row and Epi::Sum::kCols columns of it as integers.
//
// Persistent: CTA c works through tiles c, c + gridDim.x, ...; the copy and
// MMA warps run on into the next tile while the drain warps finish the last
// one.  The accumulators of a chunk are drained group by group: group g is
// committed as soon as its last product is issued, and the next chunk's first
// products into it wait for its own drain only, so draining (4,000 clocks a
// chunk) overlaps the products of the neighbouring stages (1,800 clocks a
// chunk remain).  Bound by the tensor cores' shared-memory reads: 49.4 clocks
// per product measured, 48 by its bytes.  A wait that runs out (a copy that
// never lands) ends the CTA's work, and epi.poison marks the results.  H x at
// n = 5000 with 5000 columns: one tile per CTA with one drain barrier 5.3 ms,
// this form 3.7 ms; the fma chain on the FP64 pipe 114 ms.
template <class Epi>
__global__ void __launch_bounds__(64 + 32 * Epi::kWarps, 1)
k_dg_gemm(const unsigned char *__restrict__ A, const unsigned char *__restrict__ B, int tiles, Epi epi, const int *off) {
    extern __shared__ __align__(1024) unsigned char dg_sm[];
    __shared__ __align__(8) uint64_t full[kDgStages], empty[kDgStages], acc_full[kDgGroups], acc_empty[kDgGroups];
    __shared__ uint32_t tmem_base;
    __shared__ int failed;
    const int tid = threadIdx.x, wid = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < kDgStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int g = 0; g < kDgGroups; ++g) {
            mbar_init(&acc_full[g], 1);
            mbar_init(&acc_empty[g], Epi::kWarps);
        }
        mbar_fence_init();
        failed = 0;
    }
    if (wid == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&tmem_base))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    dg_fence_before();
    __syncthreads();
    dg_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    unsigned char *const sa = reinterpret_cast<unsigned char *>(((uintptr_t)dg_sm + 1023) & ~(uintptr_t)1023);
    unsigned char *const sb = sa + kDgStages * kDgABytes;
    const uint32_t sa0 = __shfl_sync(0xffffffffu, smem_u32(sa), 0), sb0 = sa0 + kDgStages * kDgABytes;

    if (wid == 0) {
        if (lane == 0) {
            unsigned it = 0;                                     // stages issued so far
            bool ok = true;
            for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
                const DgTile q = epi.tile(tile);
                const unsigned char *ga = A + (size_t)q.a * kDgABytes, *gb = B + (size_t)q.b * kDgBBytes;
                for (int t = 0; t < q.stages; ++t, ++it) {
                    const unsigned st = it % kDgStages;
                    if (it >= kDgStages && !dg_wait(&empty[st], (it / kDgStages - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&full[st], kDgABytes + kDgBBytes);
                    dg_bulk(sa + (size_t)st * kDgABytes, ga + (size_t)t * kDgABytes, kDgABytes, &full[st]);
                    dg_bulk(sb + (size_t)st * kDgBBytes, gb + (size_t)t * kDgBBytes, kDgBBytes, &full[st]);
                }
            }
            // The last copies have landed before the CTA's shared memory goes.
            for (unsigned t = it > kDgStages ? it - kDgStages : 0; t < it; ++t)
                ok = dg_wait(&full[t % kDgStages], (t / kDgStages) & 1) && ok;
            if (!ok) failed = 1;
        }
        __syncwarp();
    } else if (wid == 1) {
        unsigned it = 0, chunk = 0;                              // stages consumed, chunks begun
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            const DgTile q = epi.tile(tile);
            const int nst = q.stages;
            for (int t = 0; t < nst && ok; ++t, ++it) {
                const int in_chunk = t % kDgChunk;
                const unsigned st = it % kDgStages;
                ok = dg_wait(&full[st], (it / kDgStages) & 1);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                dg_fence_after();
                const uint64_t da = dg_desc(sa0 + st * kDgABytes), db = dg_desc(sb0 + st * kDgBBytes);
                const bool begin = in_chunk == 0, end = in_chunk == kDgChunk - 1 || t == nst - 1;
                if (!begin && !end) {
                    if (dg_elect()) {
                        dg_products<0>(tmem, da, db, 1u);
                        dg_products<1>(tmem, da, db, 1u);
                        dg_products<2>(tmem, da, db, 1u);
                        dg_products<3>(tmem, da, db, 1u);
                        dg_products<4>(tmem, da, db, 1u);
                        dg_products<5>(tmem, da, db, 1u);
                        dg_products<6>(tmem, da, db, 1u);
                        dg_commit(&empty[st]);
                    }
                } else {
                    ok = dg_group<0>(tmem, da, db, begin, end, chunk, acc_empty, acc_full);
                    ok = dg_group<1>(tmem, da, db, begin, end, chunk, acc_empty, acc_full) && ok;
                    ok = dg_group<2>(tmem, da, db, begin, end, chunk, acc_empty, acc_full) && ok;
                    ok = dg_group<3>(tmem, da, db, begin, end, chunk, acc_empty, acc_full) && ok;
                    ok = dg_group<4>(tmem, da, db, begin, end, chunk, acc_empty, acc_full) && ok;
                    ok = dg_group<5>(tmem, da, db, begin, end, chunk, acc_empty, acc_full) && ok;
                    ok = dg_group<6>(tmem, da, db, begin, end, chunk, acc_empty, acc_full) && ok;
                    ok = __all_sync(0xffffffffu, ok);
                    if (dg_elect()) dg_commit(&empty[st]);
                    if (end) ++chunk;
                }
                __syncwarp();
            }
        }
        // ... and the last commit has arrived.
        if (it > 0) ok = ok && dg_wait(&empty[(it - 1) % kDgStages], ((it - 1) / kDgStages) & 1);
        if (!ok) failed = 1;
    } else {
        // Warp w reads TMEM lanes 32 (w mod 4) .. and kCols of the 64 columns.
        constexpr int kCols = kDgBN * 4 / Epi::kWarps;
        const int quad = wid & 3, part = (wid - 2) >> 2;
        const int row = quad * 32 + lane;
        const uint32_t base = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(part * kCols);
        const bool skip = dg_off(off);
        unsigned chunk = 0;
        bool ok = true;
        for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
            const DgTile q = epi.tile(tile);
            typename Epi::Sum sum;
            sum.zero();
            const int nchunk = (q.stages + kDgChunk - 1) / kDgChunk;
            for (int ch = 0; ch < nchunk && ok; ++ch, ++chunk) {
#pragma unroll
                for (int g = 0; g < kDgGroups; ++g) {
                    ok = __all_sync(0xffffffffu, dg_wait(&acc_full[g], chunk & 1));
                    if (!ok) break;
                    dg_fence_after();
                    float v[kCols];
                    dg_ld(base + (uint32_t)(g * kDgBN), v);
                    dg_wait_ld();
                    dg_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acc_empty[g]);
                    // Groups 0 .. 5 are exact integers in units of 2^(-12 - 8 g).
#pragma unroll
                    for (int c = 0; c < kCols; ++c) sum.add(g, c, v[c]);
                }
            }
            if (ok && !skip) epi.finish(q, q.bx * kDgBM + row, q.by * kDgBN + part * kCols, sum);
        }
        if (!ok) failed = 1;
    }
    dg_fence_before();
    __syncthreads();
    dg_fence_after();
    if (wid == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
    if (failed && !dg_off(off)) epi.poison(threadIdx.x, blockDim.x);
}

// ------------------------------------------------------------- epilogues
__device__ __forceinline__ bool dg_bad(int ex) { return ex >= kDgBad / 2; }
__host__ __device__ __forceinline__ double dg_nan() { return from_bits(0x7ff8000000000000ULL); }

// Stages [0, steps) of every tile cut into nz parts of `per` stages; part z
// of C(i, j) goes to out[z * cz + i * si + j * sj].
template <class S, int W>
struct DgStore {
    using Sum = S;
    static constexpr int kWarps = W;
    int mblocks, nblocks, steps, per, M, N;
    const int *ea, *eb;
    double *out;
    long long si, sj, cz;
    __device__ __forceinline__ DgTile tile(int t) const {
        const int mn = mblocks * nblocks, bz = t / mn, r = t - bz * mn, by = r / mblocks;
        const int bx = r - by * mblocks, s0 = bz * per;
        return DgTile{bx, by, bz, (long long)bx * steps + s0, (long long)by * steps + s0, min(steps - s0, per)};
    }
    __device__ __forceinline__ void finish(const DgTile &q, int i, int j0, const Sum &sum) const {
        const int lane = threadIdx.x & 31;
        const int ecl = max(eb[min(j0 + lane, N - 1)], kDgZero), er = max(ea[min(i, M - 1)], kDgZero);
        double *o = out + (size_t)q.bz * cz + (size_t)i * si + (size_t)j0 * sj;
#pragma unroll
        for (int c = 0; c < S::kCols; ++c) {
            const int ec = __shfl_sync(0xffffffffu, ecl, c);
            const double v = sum.value(c, er + ec - 2044);
            if (i < M && j0 + c < N) o[(size_t)c * sj] = dg_bad(er) || dg_bad(ec) ? dg_nan() : v;
        }
    }
    // Every part: the tile that failed may be of any, and the others' owners
    // may still store theirs.
    __host__ __device__ void poison(int thread, int threads) const {
        for (int z = 0; z * per < steps; ++z)
            for (long long e = thread; e < (long long)M * N; e += threads)
                out[z * cz + (e % M) * si + (e / M) * sj] = dg_nan();
    }
};
using DgStoreLong = DgStore<DgTwo<16>, 16>;
using DgStoreShort = DgStore<DgOne<16>, 16>;
// C(i, j) -= sum over at most 128 columns; cex (optional): the columns'
// exponents are raised to the new entries' in rows cex_row ...  One FP64 instruction per entry (a
// warp's takes 64 clocks), the rest on the integer pipe.  Sixteen drain warps
// with one word per sum: with eight and two words (168 registers, two warps
// per scheduler) this end took 13,000 clocks of a tile whose products take
// 14,000, and the two did not overlap.
struct DgUpdate {
    using Sum = DgOne<16>;
    static constexpr int kWarps = 16;
    int mblocks, steps, M, N;
    const int *ea, *eb;
    double *C;
    long long ldc;
    int *cex, cex_row;
    __device__ __forceinline__ DgTile tile(int t) const {
        const int by = t / mblocks;
        const int bx = t - by * mblocks;
        return DgTile{bx, by, 0, (long long)bx * steps, (long long)by * steps, steps};
    }
    __device__ __forceinline__ void finish(const DgTile &, int i, int j0, const Sum &sum) const {
        // Lane c holds column j0 + c's exponents, loaded once.
        const int lane = threadIdx.x & 31, jl = min(j0 + lane, N - 1);
        const int ecl = max(eb[jl], kDgZero), er = max(ea[min(i, M - 1)], kDgZero);
        const bool in = i < M, any_bad = __any_sync(0xffffffffu, dg_bad(er) || dg_bad(ecl));
        const int cl = cex ? cex[jl] : 0;
        unsigned big = 0;                                        // largest high word of the lane's column
        double *Ci = C + min(i, M - 1) + (size_t)j0 * ldc;
        const int cols = min(Sum::kCols, N - j0);
        double x[Sum::kCols];
#pragma unroll
        for (int c = 0; c < Sum::kCols; ++c) x[c] = c < cols ? Ci[(size_t)c * ldc] : 0.0;
#pragma unroll
        for (int c = 0; c < Sum::kCols; ++c) {
            const int ec = __shfl_sync(0xffffffffu, ecl, c);
            x[c] = x[c] - sum.value(c, er + ec - 2044);
            if (any_bad && (dg_bad(er) || dg_bad(ec))) x[c] = dg_nan();
            if (in && c < cols) Ci[(size_t)c * ldc] = x[c];
        }
        if (!cex) return;
#pragma unroll
        for (int c = 0; c < Sum::kCols; ++c) {
            const unsigned m = __reduce_max_sync(
                0xffffffffu, in && i >= cex_row ? (unsigned)(ubits(x[c]) >> 32) & 0x7fffffffu : 0u);
            if (lane == c) big = m;
        }
        if (lane < cols) {
            const int m = big >= 0x7ff00000u ? kDgBad : max((int)(big >> 20), 1);
            if (m > cl) atomicMax(&cex[jl], m);
        }
    }
    __device__ void poison(int thread, int threads) const {
        for (long long e = thread; e < (long long)M * N; e += threads) C[(e % M) + (e / M) * ldc] = dg_nan();
    }
};

// Parts of a sum over `steps` stages for `tiles` tiles (per: stages of a
// part): as many as give the fewest stages on the busiest SM, five stages'
// time counted for the end of each part.
inline int dg_parts(int tiles, int sms, int most, int steps, int &per) {
    long long best = LLONG_MAX;
    int nz = 1;
    for (int z = 1; z <= most && (z == 1 || z * kDgChunk / 2 <= steps); ++z) {
        const long long pz = (steps + z - 1) / z, cost = (((long long)tiles * z + sms - 1) / sms) * (pz + 5);
        if (cost < best) {
            best = cost;
            nz = z;
        }
    }
    per = (steps + nz - 1) / nz;
    return (steps + per - 1) / per;
}
template <class Epi>
inline cudaError_t dg_gemm(int tiles, int sms, const unsigned char *A, const unsigned char *B, const Epi &epi,
                           const int *off, cudaStream_t st) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_dg_gemm<Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDgSmem);
    if (e != cudaSuccess) return e;
    k_dg_gemm<Epi><<<std::min(tiles, sms), 64 + 32 * Epi::kWarps, kDgSmem, st>>>(A, B, tiles, epi, off);
    return cudaGetLastError();
}

}  // namespace hsr
