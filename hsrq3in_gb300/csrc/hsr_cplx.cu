// hsr_cplx.cu -- sm_103a kernels for complex-conjugate shifts.
//
// A shift mu = wr + i wi makes H - mu I complex on its diagonal only.  The
// sweep is the real one (hsr_kernels.cu) in complex arithmetic:
//   k_init_c    start vector eps3 in the real part, crossover columns
//               H(:, n-1) - mu e_n
//   k_diag_c    lane-per-pair: complex Givens generation of the diagonal tile
//               fused with the robust back-substitution (reduce.c:27-68 +
//               solve-task.c:19-225), the complex 1x1 solves going through the
//               robust complex division of robust.c:486-773; then the stage
//               operands W and Zs
//   k_diag_cn   the same for few pairs: 4, 8 or 16 per CTA, the two chains and
//               the 1x1 systems on warps of their own
//   k_part1_c   the exact no-rescale test per (tile, pair), the full complex
//               Part 1 of update-task.c:68-226 where a decision can fire
//   k_gemm_c    the real GEMM over H (hsr_kernels.cu) with a complex epilogue:
//               the imaginary parts are just more columns of W and Zs
//   k_finalize<true>  (hsr_kernels.cu) reconciliation, complex back-transform,
//               2-norm, convergence
// Layout: pair p holds its real part in column 2p and its imaginary part in
// column 2p+1 of X, R, W, Zs, Zslow and of the per-column scalars pi, ytil,
// zlast and the shifts; the cosine of a rotation is Cr[.][2p], the complex
// sine Sr[.][2p] + i Sr[.][2p+1]; the per-pair scaling factor, norm bound,
// perturbation and protected-path flags live at column 2p.
//
// Magnitude bounds use cabs1 = |Re| + |Im| (LAPACK's CABS1).  Every complex
// operation has one fma shape (hsr_device.cuh) shared with the oracle's
// complex path, which the device reproduces bit for bit.
#include "hsr_device.cuh"
#include "hsr_kernels.h"

#include <cfloat>
#include <type_traits>

namespace hsr {

// ---------------------------------------------------------------- init
// Start vectors: mode 0 eps3 (inverse_iteration.c:19-34), mode 1 the
// dlaein-style restart vector of round `its` (:36-57), both real; crossover
// columns H(:, n-1) - mu e_n (reduce.c:276-308); unit scaling factors.
__global__ void k_init_c(DevProblem P, int mode, const double *eps3_dev, int its) {
    const int p = blockIdx.y;
    if (2 * p >= P.S) return;
    const int k = 2 * p;
    const double eps3 = *eps3_dev;
    const int n = P.n;
    const double sq = sqrt((double)n);
    const double tmp = eps3 / (sq + 1.0);
    double *xr = P.X + (size_t)k * P.ldx, *xi = xr + P.ldx;
    double *rr = P.R + (size_t)k * P.ldr, *ri = rr + P.ldr;
    const double *hl = P.H + (size_t)(n - 1) * P.ldh;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double h = hl[i], hi = 0.0;
        if (i == n - 1) {
            h = h - P.wr[k];
            hi = -P.wr[k + 1];
        }
        rr[i] = h;
        ri[i] = hi;
        double v = eps3;
        if (mode == 1) {
            v = (i == 0) ? eps3 : tmp;
            if (i == n - 1 - its) v -= eps3 * sq;
        }
        xr[i] = v;
        xi[i] = 0.0;
    }
    if (blockIdx.x == 0) {
        const double ub = mode == 1 ? fmax(fmax(eps3, tmp), absd(tmp - eps3 / sq)) : eps3;
        for (int I = threadIdx.x; I < P.T; I += blockDim.x) {
            P.beta[(size_t)I * P.Spad + k] = sc_one(P.is);
            P.beta[(size_t)I * P.Spad + k + 1] = sc_one(P.is);
            P.ynorm[(size_t)I * P.Spad + k] = ub;
            P.ynorm[(size_t)I * P.Spad + k + 1] = ub;
        }
        if (threadIdx.x == 0) P.pert[k] = P.pert[k + 1] = 0;
    }
}

cudaError_t launch_init_c(const DevProblem &P, int mode, const double *eps3_dev, int its, cudaStream_t st) {
    int bx = (P.n + 255) / 256;
    if (bx > 64) bx = 64;
    dim3 g(bx, P.S / 2);
    k_init_c<<<g, 256, 0, st>>>(P, mode, eps3_dev, its);
    return cudaGetLastError();
}

// -------------------------------------------------------------- diagonal
// 32 pairs per CTA, one per lane, on NW warps (at least one per SM
// sub-partition).  Warp 0 evaluates each step's scalar chain -- complex
// Givens, the robust complex 1x1 solve, the three overflow decisions -- and
// hands its results to the others through shared memory; warps 1 .. NW-1
// update the rows of y and of the running column v, one step behind the
// chain: in step j warp 0 first updates row j-2 itself and then evaluates
// everything of step j-1's chain that does not need the new bounds, while
// the other warps update rows 0 .. j-3; after a barrier warp 0 folds their
// maxima into step j-1's third decision.  Every row sees the same operations
// in the same order as in the unpipelined form, so the result is unchanged
// bit for bit.  v and y live in shared memory as [row][lane] (real and
// imaginary parts in separate arrays); when 4*32*b doubles do not fit, in a
// global scratch region.  The bound of y(0:j-2) is the largest cabs1 at the
// start of the step, times the step's scaling factors.
//   NW = 8 with v/y in shared memory (two warps per sub-partition hide the
//   FP64 latency), NW = 4 with v/y in global scratch, where the CTAs share
//   SMs with the concurrent GEMM.
constexpr int kDiagWarpsC = 4;       // v/y in global scratch
constexpr int kDiagWarpsCSmem = 8;   // v/y in shared memory
constexpr int kDiagBcastC = 12;

// Everything but v/y: three staged columns of H, per-warp maxima [NW][2][32]
// and the broadcast slots.
__host__ __device__ constexpr size_t diagc_small_bytes(int b, int nw) {
    return (size_t)(3 * (b + 1)) * sizeof(double) + (size_t)nw * 2 * 32 * 8 + (size_t)kDiagBcastC * 32 * 8;
}
size_t diag_c_smem_bytes(int b, bool *global_vy) {
    const size_t small = diagc_small_bytes(b, kDiagWarpsCSmem);
    const size_t full = small + (size_t)4 * 32 * b * sizeof(double);
    const bool fits = full <= 220 * 1024;
    if (global_vy) *global_vy = !fits;
    return fits ? full : small;
}

template <int NW>
__global__ void __launch_bounds__(32 * NW) k_diag_c(DevProblem P, int J, double *gscratch) {
    extern __shared__ double sm[];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    const int np = P.S / 2;
    const int p0 = blockIdx.x * 32;
    const int pidx = p0 + lane;
    const bool act = pidx < np;
    const int k = 2 * pidx;
    const int l = P.fr[J], b = P.fr[J + 1] - l;
    const bool is = P.is != 0;
    const size_t Spad = (size_t)P.Spad;
    constexpr int NR = NW - 1;                                         // row warps
    {
        // A launch given less shared memory than the layout needs records a
        // shape error and touches nothing.
        const size_t need = diagc_small_bytes(b, NW) + (gscratch ? 0 : (size_t)4 * 32 * b * sizeof(double));
        if (need > dynamic_smem_bytes()) {
            if (threadIdx.x == 0) atomicOr(P.err, kErrShape);
            return;
        }
    }

    double *hc = sm;                                                   // [3][b+1]
    unsigned long long *pmax = reinterpret_cast<unsigned long long *>(sm + 3 * (b + 1));   // [NW][2][32]
    double *bc = sm + 3 * (b + 1) + NW * 2 * 32;                       // [kDiagBcastC][32]
    double *vr_, *vi_, *yr_, *yi_;
    if (gscratch) {
        vr_ = gscratch + (size_t)blockIdx.x * 4 * 32 * b;
    } else {
        vr_ = bc + kDiagBcastC * 32;
    }
    vi_ = vr_ + (size_t)32 * b;
    yr_ = vi_ + (size_t)32 * b;
    yi_ = yr_ + (size_t)32 * b;
#define VR(i) vr_[(size_t)(i) * 32 + lane]
#define VI(i) vi_[(size_t)(i) * 32 + lane]
#define YR(i) yr_[(size_t)(i) * 32 + lane]
#define YI(i) yi_[(size_t)(i) * 32 + lane]
#define PM(w, which) pmax[((w) * 2 + (which)) * 32 + lane]
#define BC(q) bc[(q) * 32 + lane]
#define HCOL(col) (hc + (size_t)((col) % 3) * (b + 1))

    // Load the crossover column and the solution tile, transposed.
    for (int c = wid; c < 32; c += NW) {
        const int pc = p0 + c;
        if (pc < np) {
            const double *rr = P.R + l + (size_t)(2 * pc) * P.ldr, *ri = rr + P.ldr;
            const double *xr = P.X + l + (size_t)(2 * pc) * P.ldx, *xi = xr + P.ldx;
            for (int i = lane; i < b; i += 32) {
                vr_[(size_t)i * 32 + c] = rr[i];
                vi_[(size_t)i * 32 + c] = ri[i];
                yr_[(size_t)i * 32 + c] = xr[i];
                yi_[(size_t)i * 32 + c] = xi[i];
            }
        } else {
            for (int i = lane; i < b; i += 32) {
                vr_[(size_t)i * 32 + c] = 1.0;
                vi_[(size_t)i * 32 + c] = 0.0;
                yr_[(size_t)i * 32 + c] = 0.0;
                yi_[(size_t)i * 32 + c] = 0.0;
            }
        }
    }

    const dcplx mu = act ? cmk(P.wr[k], P.wr[k + 1]) : cmk(0.0, 0.0);
    const double smin = fmax(DBL_EPSILON / 2 * cabs1(mu), P.smlnum);
    const double Hnorm = P.Hn[J + (size_t)J * P.T];
    double beta = act ? P.beta[(size_t)J * Spad + k] : sc_one(is);
    int pert = 0;

    const double *Hd = P.H + l + (size_t)l * P.ldh;
    auto stage_col = [&](int col) {                                    // H(l : l+col+1, l+col), warp 0
        int rows = col + 2;
        if (rows > b) rows = b;
        const double *src = Hd + (size_t)col * P.ldh;
        double *dst = HCOL(col);
        for (int i = lane; i < rows; i += 32) cp_async8(dst + i, src + i);
        cp_async_commit();
    };
    if (wid == 0 && b >= 2) stage_col(b - 2);
    if (wid == 0 && b >= 3) stage_col(b - 3);
    if (wid == 0) cp_async_wait_all();
    __syncthreads();                                                   // tiles and columns loaded

    // Largest cabs1 of y(0:b-3) and v(0:b-3) for the first step.
    {
        unsigned long long ym = 0, vm = 0;
        if (wid > 0)
            for (int i = wid - 1; i < b - 2; i += NR) {
                ym = umax64(ym, abs_bits(cabs1(cmk(YR(i), YI(i)))));
                vm = umax64(vm, abs_bits(cabs1(cmk(VR(i), VI(i)))));
            }
        PM(wid, 0) = ym;
        PM(wid, 1) = vm;
    }

    // Chain state of warp 0.
    dcplx vcar = cmk(VR(b - 1), VI(b - 1)), ycar = cmk(YR(b - 1), YI(b - 1));
    double c = 0.0, a1 = 1.0, a2 = 1.0, a3 = 1.0;
    dcplx sg = cmk(0.0, 0.0), yc = sg, ys = sg, yj = sg, yjm1 = sg;

    // Parts 1-2 of step jj's chain: Givens, the 1x1 solve, the y(jj-1)
    // decision and update (solve-task.c:76-90), the next running column entry
    // (solve-task.c:105-108).  vjm1, yjm1_in are row jj-1.
    auto chain12 = [&](int jj, dcplx vjm1, dcplx yjm1_in) {
        const double *hcol = HCOL(jj - 1);
        const double hsub = hcol[jj];
        const dcplx hd = cmk(hcol[jj - 1] - mu.re, -mu.im);
        const dcplx vj = vcar;
        yj = ycar;
        yjm1 = yjm1_in;
        cgivens(vj, hsub, c, sg);
        if (act) {
            P.Cr[(size_t)(l + jj) * Spad + k] = c;
            P.Sr[(size_t)(l + jj) * Spad + k] = sg.re;
            P.Sr[(size_t)(l + jj) * Spad + k + 1] = sg.im;
        }
        // y(j) := y(j) / R(j,j), R(j,j) = c v(j) - conj(sigma) H(j,j-1).
        double phi = sc_one(is);
        pert |= csolve_1x1(smin, c * vj.re, c * vj.im, sg.re * hsub, (-sg.im) * hsub, yj, phi, is);
        beta = sc_combine(beta, phi, is);
        a1 = sc_value(phi, is);
        if (!is_one(a1)) yjm1 = cscal(a1, yjm1);
        phi = protect_double_update(cabs1(vjm1), cabs1(yj), cabs1(hd), cabs1(yj), cabs1(yjm1), is);
        a2 = sc_value(phi, is);
        if (!is_one(a2)) {
            yj = cscal(a2, yj);
            yjm1 = cscal(a2, yjm1);
        }
        beta = sc_combine(beta, phi, is);
        yc = cscal(c, yj);
        ys = cmulc(sg, yj);
        yjm1 = cfma(ys, hd, cfnma(yc, vjm1, yjm1));
        const dcplx sv = cmul(sg, vjm1);
        vcar = cmk(fma(c, hd.re, sv.re), fma(c, hd.im, sv.im));
    };
    // Part 3 of step jj's chain: the y(0:jj-2) decision (solve-task.c:92-100)
    // with the maxima of rows 0 .. jj-2 folded by the row warps, then the
    // step's scalars for the row warps, the solved entry y(jj) and y(jj-1).
    auto chain3 = [&](int jj) {
        unsigned long long ymb = 0, vmb = 0;
#pragma unroll
        for (int w = 1; w < NW; ++w) {
            ymb = umax64(ymb, PM(w, 0));
            vmb = umax64(vmb, PM(w, 1));
        }
        double ymax = from_bits(ymb);
        if (!is_one(a1)) ymax = a1 * ymax;
        if (!is_one(a2)) ymax = a2 * ymax;
        const double phi = protect_double_update(from_bits(vmb), cabs1(yj), Hnorm, cabs1(yj), ymax, is);
        a3 = sc_value(phi, is);
        if (!is_one(a3)) {
            yj = cscal(a3, yj);
            yjm1 = cscal(a3, yjm1);
            yc = cscal(c, yj);
            ys = cmulc(sg, yj);
        }
        beta = sc_combine(beta, phi, is);
        BC(0) = c;
        BC(1) = sg.re;
        BC(2) = sg.im;
        BC(3) = yc.re;
        BC(4) = yc.im;
        BC(5) = ys.re;
        BC(6) = ys.im;
        BC(7) = a1;
        BC(8) = a2;
        BC(9) = a3;
        YR(jj) = yj.re;
        YI(jj) = yj.im;
        ycar = yjm1;
    };

    if (wid == 0 && b >= 2) chain12(b - 1, cmk(VR(b - 2), VI(b - 2)), cmk(YR(b - 2), YI(b - 2)));
    __syncthreads();                                                   // first maxima in
    if (wid == 0 && b >= 2) chain3(b - 1);
    __syncthreads();                                                   // step b-1's scalars visible

    for (int j = b - 1; j >= 1; --j) {
        // Step j's scalars: registers on warp 0, shared memory for the rest.
        double sc_c = c, s1 = a1, s2 = a2, s3 = a3;
        dcplx sc_sg = sg, sc_yc = yc, sc_ys = ys;
        if (wid != 0) {
            sc_c = BC(0);
            sc_sg = cmk(BC(1), BC(2));
            sc_yc = cmk(BC(3), BC(4));
            sc_ys = cmk(BC(5), BC(6));
            s1 = BC(7);
            s2 = BC(8);
            s3 = BC(9);
        }
        const bool scaled = (!is_one(s1)) || (!is_one(s2)) || (!is_one(s3));
        const double *hcol = HCOL(j - 1);
        // Row i of step j (the unpipelined loop body).
        auto row = [&](int i, dcplx &yo, dcplx &vo) {
            const double h = hcol[i];
            dcplx yv = cmk(YR(i), YI(i));
            const dcplx vv = cmk(VR(i), VI(i));
            if (scaled) {
                if (!is_one(s1)) yv = cscal(s1, yv);
                if (!is_one(s2)) yv = cscal(s2, yv);
                if (!is_one(s3)) yv = cscal(s3, yv);
            }
            yo = cfmar(sc_ys, h, cfnma(sc_yc, vv, yv));
            const dcplx sv = cmul(sc_sg, vv);
            vo = cmk(fma(sc_c, h, sv.re), sv.im);
            YR(i) = yo.re;
            YI(i) = yo.im;
            VR(i) = vo.re;
            VI(i) = vo.im;
        };
        if (wid == 0) {
            if (j >= 2) {
                dcplx yn, vn;
                row(j - 2, yn, vn);                                    // enters step j-1's chain
                cp_async_wait_all();                                   // column j-2, staged last step
                __syncwarp();                                          // ... by all lanes of warp 0
                chain12(j - 1, vn, yn);
            }
            if (j >= 3) stage_col(j - 3);                              // for step j-2's chain
        } else {
            if (scaled) {
                for (int i = j + 1 + ((wid - 1 - (j + 1)) % NR + NR) % NR; i < b; i += NR) {
                    dcplx t = cmk(YR(i), YI(i));
                    if (!is_one(s1)) t = cscal(s1, t);
                    if (!is_one(s2)) t = cscal(s2, t);
                    if (!is_one(s3)) t = cscal(s3, t);
                    YR(i) = t.re;
                    YI(i) = t.im;
                }
            }
            unsigned long long ymx = 0, vmx = 0;
            for (int i = wid - 1; i < j - 2; i += NR) {                // rows 0 .. j-3
                dcplx yo, vo;
                row(i, yo, vo);
                ymx = umax64(ymx, abs_bits(cabs1(yo)));
                vmx = umax64(vmx, abs_bits(cabs1(vo)));
            }
            PM(wid, 0) = ymx;
            PM(wid, 1) = vmx;
        }
        __syncthreads();                                               // rows of step j done, maxima in
        if (wid == 0 && j >= 2) chain3(j - 1);
        __syncthreads();                                               // step j-1's scalars visible
    }

    double c0 = 1.0;
    dcplx s0 = cmk(0.0, 0.0);
    {
        dcplx y0 = cmk(0.0, 0.0);
        double a = 1.0;
        if (wid == 0) {
            dcplx v0 = b >= 2 ? vcar : cmk(VR(0), VI(0));
            y0 = b >= 2 ? ycar : cmk(YR(0), YI(0));
            if (J > 0) {
                // Final rotation with H(l, l-1) (reduce.c:53-61).
                const double hleft = P.H[l + (size_t)(l - 1) * P.ldh];
                if (hleft != 0) {
                    cgivens(v0, hleft, c0, s0);
                } else {
                    c0 = 1.0;
                    s0 = cmk(0.0, 0.0);
                }
                if (act) {
                    P.Cr[(size_t)l * Spad + k] = c0;
                    P.Sr[(size_t)l * Spad + k] = s0.re;
                    P.Sr[(size_t)l * Spad + k + 1] = s0.im;
                }
                v0 = cmk(fma(v0.re, c0, -(hleft * s0.re)), fma(v0.im, c0, hleft * s0.im));
            }
            double phi = sc_one(is);
            pert |= csolve_1x1(smin, v0.re, v0.im, 0.0, 0.0, y0, phi, is);
            beta = sc_combine(beta, phi, is);
            a = sc_value(phi, is);
            BC(0) = c0;
            BC(1) = s0.re;
            BC(2) = s0.im;
            BC(3) = a;
        }
        __syncthreads();
        if (wid != 0) {
            c0 = BC(0);
            s0 = cmk(BC(1), BC(2));
            a = BC(3);
        }
        if (!is_one(a))
            for (int i = 1 + ((wid - 1) % NW + NW) % NW; i < b; i += NW) {
                YR(i) = a * YR(i);
                YI(i) = a * YI(i);
            }
        if (wid == 0) {
            YR(0) = y0.re;
            YI(0) = y0.im;
        }
    }
    __syncthreads();

    for (int c = wid; c < 32; c += NW) {
        const int pc = p0 + c;
        if (pc < np) {
            double *xr = P.X + l + (size_t)(2 * pc) * P.ldx, *xi = xr + P.ldx;
            for (int i = lane; i < b; i += 32) {
                xr[i] = yr_[(size_t)i * 32 + c];
                xi[i] = yi_[(size_t)i * 32 + c];
            }
        }
    }
    if (act && wid == 0) {
        P.beta[(size_t)J * Spad + k] = beta;
        if (pert) P.pert[k] = P.pert[k + 1] = 1;
    }
    if (J == 0 || !act) return;

    if (wid == 0) {
        // W(q) = c_q prod_{p<q} sigma_p, pi = prod sigma (crossover propagation).
        dcplx pk = cmk(1.0, 0.0);
        for (int q = 0; q < b; ++q) {
            const double cq = P.Cr[(size_t)(l + q) * Spad + k];
            const dcplx sq = cmk(P.Sr[(size_t)(l + q) * Spad + k], P.Sr[(size_t)(l + q) * Spad + k + 1]);
            const dcplx w = cscal(cq, pk);
            P.W[(size_t)q * Spad + k] = w.re;
            P.W[(size_t)q * Spad + k + 1] = w.im;
            pk = cmul(pk, sq);
        }
        P.pi[k] = pk.re;
        P.pi[k + 1] = pk.im;
    }
    if (wid == 1) {
        // Ytilde2 (update-task.c:170-198): Zs(q) = Ytilde2(q-1), Zs(0) = 0,
        // zlast = Ytilde2(b-1); ytilde = -conj(sigma_0) x_0 for Part 1.
        unsigned long long zmx = 0;
        dcplx z = cscal(c0, cmk(YR(0), YI(0)));
        P.Zs[k] = 0.0;
        P.Zs[k + 1] = 0.0;
        for (int q = 1; q < b; ++q) {
            const double cq = P.Cr[(size_t)(l + q) * Spad + k];
            const dcplx sq = cmk(P.Sr[(size_t)(l + q) * Spad + k], P.Sr[(size_t)(l + q) * Spad + k + 1]);
            const dcplx t2 = cmk(YR(q), YI(q));
            const dcplx zo = crot_out(cq, sq, z, t2);
            z = crot_next(cq, sq, z, t2);
            P.Zs[(size_t)q * Spad + k] = zo.re;
            P.Zs[(size_t)q * Spad + k + 1] = zo.im;
            zmx = umax64(zmx, abs_bits(cabs1(zo)));
        }
        zmx = umax64(zmx, abs_bits(cabs1(z)));
        P.zlast[k] = z.re;
        P.zlast[k + 1] = z.im;
        P.z2n[k] = from_bits(zmx);
        const dcplx q0 = cmulc(s0, cmk(YR(0), YI(0)));
        P.ytil[k] = -q0.re;
        P.ytil[k + 1] = -q0.im;
    }
#undef VR
#undef VI
#undef YR
#undef YI
#undef PM
#undef HCOL
#undef BC
}

// Narrow form for few pairs: SC pairs per CTA, the step's serial chain on
// three warps, as diag_body_narrow (hsr_kernels.cu) does it for real shifts:
//   warp 0  rotation j, rows j-1 and j-2 of v;
//   warp 4  the 1x1 system: its coefficient and, for c_dladiv, the ratio r of
//           its parts and t = 1 / (c + d r); stages the columns of H;
//   warp 1  the solve, the decisions, rows j-1 and j-2 of y;
//   warps 2, 3, 5, 6, 7  rows 0 .. j-3 of v and y, 32 / SC rows x SC pairs per
//           instruction.
// In the chains even lane groups take the real part of a complex result, odd
// ones the imaginary part (or two quotients of one divisor), so that both cost
// one FP64 instruction; the partner's part is one exchange away.  Every element
// sees the operations of k_diag_c in their order: the same bits.
//
// Bound by the rows' FP64 issue (11 instructions of 64 clocks per 32 / SC rows
// on less than three sub-partitions), so SC is the smallest that still fits
// one wave of CTAs.  n = 2000, 500 pairs, tiles of 160: k_diag_c 3,026 us
// a tile, k_diag_cn<4> 513 us; the whole solve 49.3 -> 18.3 ms.
constexpr int kNarrowCWarps = 8, kNarrowCRows = 5;
constexpr size_t kNarrowCSmem = 200 * 1024;
template <int SC>
__host__ __device__ constexpr size_t diag_cn_smem_bytes(int b) {
    return (size_t)(4 * (b + 2) + 2 * (7 + 4 + 7) * SC + 2 * kNarrowCRows * SC + 4 * SC * b) * sizeof(double);
}

template <int SC>
__global__ void __launch_bounds__(32 * kNarrowCWarps) k_diag_cn(DevProblem P, int J) {
    static_assert(SC == 4 || SC == 8 || SC == 16, "pairs per CTA");
    constexpr int NW = kNarrowCWarps, NR = kNarrowCRows, RL = 32 / SC;
    extern __shared__ double sm[];
    __shared__ __align__(8) uint64_t bars[8];                          // two each: rotation, system, factors, rows
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int sh = lane % SC, rs = lane / SC;                          // pair slot; row slot, lane group
    const bool odd = (rs & 1) != 0, store_lane = lane < SC;
    const int rw = wid < 4 ? wid - 2 : wid - 3;                        // row-warp index
    const int np = P.S / 2, p0 = blockIdx.x * SC, pidx = p0 + sh;
    const bool act = pidx < np;
    const int k = 2 * pidx;
    const int l = P.fr[J], b = P.fr[J + 1] - l;
    const bool is = P.is != 0;
    const size_t Spad = (size_t)P.Spad;
    if (diag_cn_smem_bytes<SC>(b) > dynamic_smem_bytes()) {
        if (tid == 0) atomicOr(P.err, kErrShape);
        return;
    }

    double *hc = sm;                                                   // [4][b+2]
    double *sa = hc + 4 * (b + 2);                                     // [2][7][SC]: c, sigma, v(j), v(j-1)
    double *sx = sa + 2 * 7 * SC;                                      // [2][4][SC]: r, t, kind, Re(H(j-1,j-1) - mu)
    double *sb = sx + 2 * 4 * SC;                                      // [2][7][SC]: yc, ys, a1, a2, a3
    unsigned *pm = reinterpret_cast<unsigned *>(sb + 2 * 7 * SC);      // [2][NR][2][SC], high words
    double *vr_ = sb + 2 * 7 * SC + 2 * NR * SC;
    double *vi_ = vr_ + (size_t)SC * b, *yr_ = vi_ + (size_t)SC * b, *yi_ = yr_ + (size_t)SC * b;
#define VR(i) vr_[(size_t)(i) * SC + sh]
#define VI(i) vi_[(size_t)(i) * SC + sh]
#define YR(i) yr_[(size_t)(i) * SC + sh]
#define YI(i) yi_[(size_t)(i) * SC + sh]
#define SA(t, q) sa[(((t) & 1) * 7 + (q)) * SC + sh]
#define SX(t, q) sx[(((t) & 1) * 4 + (q)) * SC + sh]
#define SB(t, q) sb[(((t) & 1) * 7 + (q)) * SC + sh]
#define PM(t, w, which) pm[((((t) & 1) * NR + (w)) * 2 + (which)) * SC + sh]
#define HCOL(col) (hc + (size_t)((col) & 3) * (b + 2))

    if (tid == 0) {
        for (int q = 0; q < 8; ++q) mbar_init(&bars[q], q < 6 ? 1 : NR);
        mbar_fence_init();
    }
    for (int idx = tid; idx < SC * b; idx += 32 * NW) {
        const int c = idx / b, i = idx - c * b, pc = p0 + c;
        const size_t at = (size_t)i * SC + c;
        if (pc < np) {
            const double *rr = P.R + l + i + (size_t)(2 * pc) * P.ldr, *xr = P.X + l + i + (size_t)(2 * pc) * P.ldx;
            vr_[at] = rr[0];
            vi_[at] = rr[P.ldr];
            yr_[at] = xr[0];
            yi_[at] = xr[P.ldx];
        } else {
            vr_[at] = 1.0;
            vi_[at] = yr_[at] = yi_[at] = 0.0;
        }
    }
    const dcplx mu = act ? cmk(P.wr[k], P.wr[k + 1]) : cmk(0.0, 0.0);
    const double smin = fmax(DBL_EPSILON / 2 * cabs1(mu), P.smlnum);
    double beta = act ? P.beta[(size_t)J * Spad + k] : sc_one(is);
    int pert = 0;
    const double *Hd = P.H + l + (size_t)l * P.ldh;
    auto stage_col = [&](int col) {                                    // H(l : l+col+1, l+col), warp 4
        if (col >= 0) {
            const int rows = min(col + 2, b);
            const double *src = Hd + (size_t)col * P.ldh;
            double *dst = HCOL(col);
            for (int i = lane; i < rows; i += 32) cp_async8(dst + i, src + i);
        }
        cp_async_commit();                                             // one group per column, empty ones too
    };
    if (wid == 4) {
        stage_col(b - 2);
        stage_col(b - 3);
    }
    __syncthreads();                                                   // tile and barriers ready

    // The barriers of step t = b - 1 - j, as in diag_body_narrow.
    constexpr int kRot = 0, kSys = 2, kFac = 4, kRows = 6;
    bool ok = true;
    auto await = [&](int which, int t) { ok = ok && mbar_wait(&bars[which + (t & 1)], (uint32_t)((t >> 1) & 1), P.err); };
    auto post = [&](int which, int t) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars[which + (t & 1)]);
    };
    constexpr unsigned kAll = 0xffffffffu;
    auto even_of = [&](double x) { return __shfl_sync(kAll, x, sh); };             // the even group's value
    auto odd_of = [&](double x) { return __shfl_sync(kAll, x, sh + SC); };
    auto hi_mag = [](double x) { return (unsigned)(ubits(x) >> 32) & 0x7fffffffu; };
    auto hi_pow2 = [](int e) { return (unsigned)(pow2_bits(e) >> 32); };

    dcplx v0 = cmk(0.0, 0.0), y0 = v0;                                 // rows 0 of v (warp 0) and y (warp 1)
    if (wid == 0) {
        dcplx vj = cmk(VR(b - 1), VI(b - 1)), vw = b >= 2 ? cmk(VR(b - 2), VI(b - 2)) : vj;   // v(j), v(j-1)
        auto entry = [&](int row, int col) { return col >= 0 && row >= 0 ? Hd[row + (size_t)col * P.ldh] : 0.0; };
        double hsub = entry(b - 1, b - 2), hdiag = entry(b - 2, b - 2) - mu.re, htop = entry(b - 3, b - 2);
        double hs1 = entry(b - 2, b - 3), hd1 = entry(b - 3, b - 3), ht1 = entry(b - 4, b - 3);
        for (int j = b - 1, t = 0; j >= 1; --j, ++t) {
            double c;
            dcplx sg;
            {
                // cgivens() with the quotients of one divisor on two lane groups.
                const unsigned long long mr = mag(vj.re), mi = mag(vj.im), mg = mag(hsub);
                const unsigned long long lo = pow2_bits(-200), hi = pow2_bits(200);
                const bool in = mr > lo && mr < hi && mi > lo && mi < hi && mg > lo && mg < hi;
                const int ef = (int)(umax64(mr, mi) >> 52) - 1023, eg = (int)(mg >> 52) - 1023, e = ef > eg ? ef : eg;
                const double fsr = add_exp(vj.re, -ef), fsi = add_exp(vj.im, -ef);
                double q1, q2;
                bool okq = true;
                auto quots = [&](double ss, double a1) {               // a1 / sqrt(ss) per group; the root returned
                    unsigned long long y;
                    const unsigned long long db = ip_sqrt(in ? ubits(ss) : kOneBits + 1, y), fb = db & kSigMask, u = ubits(a1);
                    const int ea = (int)((u >> 52) & 0x7ff), eb = (int)(db >> 52);
                    okq = okq && ip_div_ok(ea, eb, fb);
                    q1 = from_bits(ip_quot((u & kSigMask) | kHidden, fb | kHidden, ip_recip_root(db, y), ea - eb + 1023,
                                           u & 0x8000000000000000ULL));
                    return from_bits(db);
                };
                const double af1 = quots(fma(fsr, fsr, fsi * fsi), odd ? fsi : fsr);
                q2 = q1;                                               // pr, pi
                const double af = add_exp(af1, ef - e), gs = add_exp(hsub, -e);
                quots(fma(af, af, gs * gs), odd ? gs : af);            // c, t
                if (__all_sync(kAll, (in && okq) || !act)) {            // pairs past the last count as in range
                    c = even_of(q1);
                    const double tt = odd_of(q1), sp = tt * q2;
                    sg = cmk(neg(even_of(sp)), odd_of(sp));
                } else {
                    cgivens(vj, hsub, c, sg);
                }
            }
            if (store_lane) {
                SA(t, 0) = c;
                SA(t, 1) = sg.re;
                SA(t, 2) = sg.im;
                SA(t, 3) = vj.re;
                SA(t, 4) = vj.im;
                SA(t, 5) = vw.re;
                SA(t, 6) = vw.im;
            }
            post(kRot, t);
            if (act && store_lane) {
                P.Cr[(size_t)(l + j) * Spad + k] = c;
                P.Sr[(size_t)(l + j) * Spad + k] = sg.re;
                P.Sr[(size_t)(l + j) * Spad + k + 1] = sg.im;
            }
            const double hdu = hdiag, htu = htop;                      // the next step's, off the chain's path
            hsub = hs1;
            hdiag = hd1 - mu.re;
            htop = ht1;
            hs1 = entry(j - 2, j - 3);
            hd1 = entry(j - 3, j - 3);
            ht1 = entry(j - 4, j - 3);
            await(kRows, t);                                           // rows of step j+1: row j-2 is in v
            const dcplx vo = !odd ? vw : (j >= 2 ? cmk(VR(j - 2), VI(j - 2)) : cmk(0.0, 0.0));
            const dcplx sv = cmul(sg, vo);
            const double nr = fma(c, !odd ? hdu : htu, sv.re), ni = !odd ? fma(c, -mu.im, sv.im) : sv.im;
            vj = cmk(even_of(nr), even_of(ni));
            vw = cmk(odd_of(nr), odd_of(ni));
        }
        v0 = vj;
    } else if (wid == 4) {
        for (int j = b - 1, t = 0; j >= 1; --j, ++t) {
            cp_async_wait_one();                                       // column j-1, for the other warps too
            await(kRot, t);
            __syncwarp();
            const double hsub = HCOL(j - 1)[j], hdg = HCOL(j - 1)[j - 1] - mu.re;
            const double x0 = (odd ? SA(t, 1) : SA(t, 0)) * (odd ? hsub : SA(t, 3));
            const double x1 = (odd ? neg(SA(t, 2)) : SA(t, 0)) * (odd ? hsub : SA(t, 4));
            const double tr = even_of(x0), lr = odd_of(x0), ti = even_of(x1), li = odd_of(x1);
            const double csr = tr - lr, csi = ti - li;
            // csolve_1x1's conditions on the coefficient, the second
            // decision's on v(j-1) and H (a |Re| + |Im| below 2^497).
            const unsigned lim = hi_pow2(200), l495 = hi_pow2(495);
            const bool swap = mag(csi) >= mag(csr);
            const double cc = swap ? csi : csr, dd = swap ? csr : csi;
            bool plain = hi_mag(tr) < lim && hi_mag(ti) < lim && hi_mag(lr) < lim && hi_mag(li) < lim &&
                         mag(dd) > pow2_bits(-200) && hi_mag(SA(t, 5)) < l495 && hi_mag(SA(t, 6)) < l495 &&
                         hi_mag(hdg) < l495 && hi_mag(mu.im) < l495;
            plain = plain && !(ubits(absd(csr) + absd(csi)) < ubits(smin));
            double r = 0.0, tq = 0.0;
            if (plain) {
                r = ddiv_rn(dd, cc);
                tq = ddiv_rn(1.0, cc + dd * r);
            }
            if (store_lane) {
                SX(t, 0) = r;
                SX(t, 1) = tq;
                SX(t, 2) = from_bits(plain ? (swap ? 1ULL : 0ULL) : 2ULL);
                SX(t, 3) = hdg;
            }
            post(kSys, t);
            if (t > 0) await(kFac, t - 1);                             // column j+1 gives way
            stage_col(j - 3);
        }
    } else if (wid == 1) {
        const double Hnorm = P.Hn[J + (size_t)J * P.T];
        const unsigned l200 = hi_pow2(200), lm400 = hi_pow2(-400), l490 = hi_pow2(490), l495 = hi_pow2(495), l497 = hi_pow2(497),
                       l990 = hi_pow2(990), l993 = hi_pow2(993);
        // fits: parts of y below 2^990 and of v below 2^490 before a step
        // without scaling whose factors' parts are below 2^497 give parts
        // below 2^991 and 2^492 after it (|c|, |sigma| <= 1, |H| < 2^490).
        const bool hfits = hi_mag(Hnorm) < l490;
        bool fits = false;
        // The lane's part (real in even groups) of y(j) and y(j-1).
        double ycar = odd ? YI(b - 1) : YR(b - 1), ynext = b >= 2 ? (odd ? YI(b - 2) : YR(b - 2)) : 0.0;
        unsigned ymh = 0, vmh = 0;
        auto bounds = [&](int t) {
            ymh = vmh = 0;
#pragma unroll
            for (int w = 0; w < NR; ++w) {
                ymh = max(ymh, PM(t, w, 0));
                vmh = max(vmh, PM(t, w, 1));
            }
        };
        auto other = [&](double x) { return __shfl_xor_sync(kAll, x, SC); };
        for (int j = b - 1, t = 0; j >= 1; --j, ++t) {
            await(kSys, t);
            const double *hcol = HCOL(j - 1);
            const double c = SA(t, 0), r = SX(t, 0), tq = SX(t, 1), hdg = SX(t, 3);
            const dcplx sg = cmk(SA(t, 1), SA(t, 2)), vjm1 = cmk(SA(t, 5), SA(t, 6)), hd = cmk(hdg, -mu.im);
            const unsigned kind = (unsigned)ubits(SX(t, 2));
            double yold = ynext, a1 = 1.0, a2 = 1.0, a3 = 1.0, yjm1 = 0.0;
            const double yo = other(ycar);
            // (a + b r) t and (b - a r) t of c_dladiv: x.re and x.im, or with
            // the parts exchanged x.re and -x.im.
            const bool swap = kind == 1;
            const double xre = odd ? yo : ycar, xim = odd ? ycar : yo;
            const double pa = swap ? xim : xre, pb = swap ? xre : xim;
            double yj = ((odd ? pb : pa) + (odd ? neg(pa) : pb) * r) * tq;
            if (odd && swap) yj = neg(yj);
            bool plain = kind < 2 && hi_mag(ycar) < l200 && hi_mag(ycar) > lm400 && hi_mag(yj) < l495 && hi_mag(yold) < l993 && fits;
            plain = __all_sync(kAll, plain || !act);
            double yc, ysc;                                            // the lane's parts of yc and ys
            if (plain) {
                const double yjo = other(yj);
                yc = c * yj;
                const double m = sg.im * yjo;
                ysc = fma(sg.re, yj, odd ? neg(m) : m);
            } else {
                dcplx x = cmk(xre, xim), yp = cmk(even_of(yold), odd_of(yold));
                double phi = sc_one(is);
                pert |= csolve_1x1(smin, mul_rare(c, SA(t, 3)), mul_rare(c, SA(t, 4)), mul_rare(sg.re, hcol[j]),
                                   mul_rare(-sg.im, hcol[j]), x, phi, is);
                beta = sc_combine(beta, phi, is);
                a1 = sc_value(phi, is);
                if (!is_one(a1)) yp = cscal(a1, yp);
                phi = protect_double_update(cabs1(vjm1), cabs1(x), cabs1(hd), cabs1(x), cabs1(yp), is);
                a2 = sc_value(phi, is);
                if (!is_one(a2)) {
                    x = cscal(a2, x);
                    yp = cscal(a2, yp);
                }
                beta = sc_combine(beta, phi, is);
                dcplx zc = cscal(c, x), zs = cmulc(sg, x);
                await(kRows, t);                                       // rows of step j+1
                unsigned long long ymb = 0, vmb = 0;                   // the maxima over rows 0 .. j-2
                bounds(t);
                if (!(ymh < l993 && vmh < l495 && hi_mag(x.re) < l495 && hi_mag(x.im) < l495 && hi_mag(Hnorm) < l497 &&
                      is_one(a1) && is_one(a2))) {
                    for (int i = 0; i <= j - 2; ++i) {
                        ymb = umax64(ymb, abs_bits(cabs1(cmk(YR(i), YI(i)))));
                        vmb = umax64(vmb, abs_bits(cabs1(cmk(VR(i), VI(i)))));
                    }
                    double ymax = from_bits(ymb);
                    if (!is_one(a1)) ymax = a1 * ymax;
                    if (!is_one(a2)) ymax = a2 * ymax;
                    phi = protect_double_update(from_bits(vmb), cabs1(x), Hnorm, cabs1(x), ymax, is);
                    a3 = sc_value(phi, is);
                    beta = sc_combine(beta, phi, is);
                }
                if (!is_one(a3)) {
                    const dcplx z = cscal(a3, cfma(zs, hd, cfnma(zc, vjm1, yp)));
                    yjm1 = odd ? z.im : z.re;
                    x = cscal(a3, x);
                    zc = cscal(c, x);
                    zs = cmulc(sg, x);
                }
                yj = odd ? x.im : x.re;
                yold = odd ? yp.im : yp.re;
                yc = odd ? zc.im : zc.re;
                ysc = odd ? zs.im : zs.re;
            }
            const bool scaled = !is_one(a1) || !is_one(a2) || !is_one(a3);
            if (lane < 2 * SC) {
                SB(t, odd ? 1 : 0) = yc;
                SB(t, odd ? 3 : 2) = ysc;
                if (odd) YI(j) = yj;
                else YR(j) = yj;
            }
            if (store_lane) {
                SB(t, 4) = a1;
                SB(t, 5) = a2;
                SB(t, 6) = a3;
            }
            post(kFac, t);
            // y - yc v: fma(-yc.re, v.re, fma(yc.im, v.im, y.re)) and
            // fma(-yc.re, v.im, fma(-yc.im, v.re, y.im)).
            const double yco = other(yc), yso = other(ysc);
            const double ycr = odd ? yco : yc, yci = odd ? yc : yco, ysr = odd ? yso : ysc, ysi = odd ? ysc : yso;
            auto minus = [&](dcplx v, double y) {
                return fma(-ycr, odd ? v.im : v.re, fma(odd ? neg(yci) : yci, odd ? v.re : v.im, y));
            };
            if (is_one(a3)) {
                const double u = minus(vjm1, yold);
                yjm1 = fma(ysr, odd ? hd.im : hd.re, fma(odd ? ysi : neg(ysi), odd ? hd.re : hd.im, u));
            }
            // Row j-2 of y, for the next step's chain, and the bounds of the
            // rows of step j+1.
            await(kRows, t);
            bounds(t);
            fits = hfits && !scaled && ymh < l990 && vmh < l490 && hi_mag(yc) < l497 && hi_mag(yco) < l497 &&
                   hi_mag(ysc) < l497 && hi_mag(yso) < l497;
            if (j >= 2) {
                double yi = odd ? YI(j - 2) : YR(j - 2);
                if (scaled) {
                    if (!is_one(a1)) yi = a1 * yi;
                    if (!is_one(a2)) yi = a2 * yi;
                    if (!is_one(a3)) yi = a3 * yi;
                }
                ynext = fma(odd ? ysi : ysr, hcol[j - 2], minus(cmk(VR(j - 2), VI(j - 2)), yi));
            }
            ycar = yjm1;
        }
        y0 = cmk(even_of(ycar), odd_of(ycar));
    } else {
        unsigned ym = 0, vm = 0;
        auto note = [&](dcplx y, dcplx v) {
            ym = max(ym, max(hi_mag(y.re), hi_mag(y.im)));
            vm = max(vm, max(hi_mag(v.re), hi_mag(v.im)));
        };
        auto fold = [&](int tm) {
#pragma unroll
            for (int o = SC; o < 32; o <<= 1) {
                ym = max(ym, __shfl_xor_sync(kAll, ym, o));
                vm = max(vm, __shfl_xor_sync(kAll, vm, o));
            }
            if (store_lane) {
                PM(tm, rw, 0) = ym;
                PM(tm, rw, 1) = vm;
            }
            post(kRows, tm);
        };
        for (int i = rw * RL + rs; i < b - 2; i += NR * RL) note(cmk(YR(i), YI(i)), cmk(VR(i), VI(i)));
        fold(0);
        for (int j = b - 1, t = 0; j >= 1; --j, ++t) {
            await(kFac, t);                                            // ... and with it the rotation and the column
            const double c = SA(t, 0), s1 = SB(t, 4), s2 = SB(t, 5), s3 = SB(t, 6);
            const dcplx sg = cmk(SA(t, 1), SA(t, 2)), yc = cmk(SB(t, 0), SB(t, 1)), ys = cmk(SB(t, 2), SB(t, 3));
            const double *hcol = HCOL(j - 1);
            const bool scaled = !is_one(s1) || !is_one(s2) || !is_one(s3);
            auto rescale = [&](dcplx y) {
                if (!is_one(s1)) y = cscal(s1, y);
                if (!is_one(s2)) y = cscal(s2, y);
                if (!is_one(s3)) y = cscal(s3, y);
                return y;
            };
            if (scaled) {
                for (int q = j + 1 + rw * RL + rs; q < b; q += NR * RL) {
                    const dcplx u = rescale(cmk(YR(q), YI(q)));
                    YR(q) = u.re;
                    YI(q) = u.im;
                }
            }
            ym = vm = 0;
            constexpr int ST = NR * RL;
            const int lim = j - 2;                                     // rows 0 .. j-3
            int i = rw * RL + rs;
            auto rows = [&](auto tag) {
                constexpr int U = decltype(tag)::value;
                double h[U];
                dcplx y[U], v[U];
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    h[q] = hcol[i + q * ST];
                    y[q] = cmk(YR(i + q * ST), YI(i + q * ST));
                    v[q] = cmk(VR(i + q * ST), VI(i + q * ST));
                    if (scaled) y[q] = rescale(y[q]);
                }
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    y[q] = cfmar(ys, h[q], cfnma(yc, v[q], y[q]));
                    const dcplx sv = cmul(sg, v[q]);
                    v[q] = cmk(fma(c, h[q], sv.re), sv.im);
                }
#pragma unroll
                for (int q = 0; q < U; ++q) {
                    YR(i + q * ST) = y[q].re;
                    YI(i + q * ST) = y[q].im;
                    VR(i + q * ST) = v[q].re;
                    VI(i + q * ST) = v[q].im;
                    note(y[q], v[q]);
                }
            };
            for (; i + ST < lim; i += 2 * ST) rows(std::integral_constant<int, 2>{});
            for (; i < lim; i += ST) rows(std::integral_constant<int, 1>{});
            fold(t + 1);
        }
    }
    __syncthreads();                                                   // the last step's rows written

    double c0 = 1.0;
    dcplx s0 = cmk(0.0, 0.0);
    if (wid == 0) {
        if (J > 0) {
            // Final rotation with H(l, l-1) (reduce.c:53-61).
            const double hleft = P.H[l + (size_t)(l - 1) * P.ldh];
            if (hleft != 0) cgivens(v0, hleft, c0, s0);
            if (act && store_lane) {
                P.Cr[(size_t)l * Spad + k] = c0;
                P.Sr[(size_t)l * Spad + k] = s0.re;
                P.Sr[(size_t)l * Spad + k + 1] = s0.im;
            }
            v0 = cmk(fma(v0.re, c0, -(hleft * s0.re)), fma(v0.im, c0, hleft * s0.im));
        }
        if (store_lane) {
            SA(0, 0) = c0;
            SA(0, 1) = s0.re;
            SA(0, 2) = s0.im;
            SA(0, 3) = v0.re;
            SA(0, 4) = v0.im;
        }
    }
    __syncthreads();
    c0 = SA(0, 0);
    s0 = cmk(SA(0, 1), SA(0, 2));
    if (wid == 1) {
        double phi = sc_one(is);
        pert |= csolve_1x1(smin, SA(0, 3), SA(0, 4), 0.0, 0.0, y0, phi, is);
        beta = sc_combine(beta, phi, is);
        if (store_lane) SB(0, 4) = sc_value(phi, is);
    }
    __syncthreads();
    {
        const double a = SB(0, 4);
        if (!is_one(a))
            for (int i = 1 + wid * RL + rs; i < b; i += NW * RL) {
                YR(i) = a * YR(i);
                YI(i) = a * YI(i);
            }
        if (wid == 1 && store_lane) {
            YR(0) = y0.re;
            YI(0) = y0.im;
        }
    }
    __syncthreads();

    for (int idx = tid; idx < SC * b; idx += 32 * NW) {
        const int c = idx / b, i = idx - c * b, pc = p0 + c;
        if (pc < np) {
            double *xr = P.X + l + i + (size_t)(2 * pc) * P.ldx;
            xr[0] = yr_[(size_t)i * SC + c];
            xr[P.ldx] = yi_[(size_t)i * SC + c];
        }
    }
    if (act && wid == 1 && store_lane) {
        P.beta[(size_t)J * Spad + k] = beta;
        if (pert) P.pert[k] = P.pert[k + 1] = 1;
    }
    if (J == 0) return;

    // The stage operands, a lane's part each (whole warps: the parts meet by
    // exchange; groups past the second repeat the first two).
    const int kk = act ? k : 0;
    const bool st = act && lane < 2 * SC;
    if (wid == 0) {
        // W(q) = c_q prod_{p<q} sigma_p, pi = prod sigma (crossover propagation).
        double pk = odd ? 0.0 : 1.0;
        for (int q = 0; q < b; ++q) {
            const double cq = P.Cr[(size_t)(l + q) * Spad + kk];
            const dcplx sq = cmk(P.Sr[(size_t)(l + q) * Spad + kk], P.Sr[(size_t)(l + q) * Spad + kk + 1]);
            if (st) P.W[(size_t)q * Spad + k + (odd ? 1 : 0)] = cq * pk;
            // cmul(pk, sq)
            const double po = __shfl_xor_sync(kAll, pk, SC), pr = odd ? po : pk, pi = odd ? pk : po;
            const double m = pi * (odd ? sq.re : sq.im);
            pk = fma(pr, odd ? sq.im : sq.re, odd ? m : neg(m));
        }
        if (st) P.pi[k + (odd ? 1 : 0)] = pk;
    }
    if (wid == 1) {
        // Ytilde2 (update-task.c:170-198): Zs(q) = Ytilde2(q-1), Zs(0) = 0,
        // zlast = Ytilde2(b-1); ytilde = -conj(sigma_0) x_0 for Part 1.
        unsigned long long zmx = 0;
        const double x0 = odd ? YI(0) : YR(0);
        double z = c0 * x0;
        if (st) P.Zs[k + (odd ? 1 : 0)] = 0.0;
        for (int q = 1; q < b; ++q) {
            const double cq = P.Cr[(size_t)(l + q) * Spad + kk];
            const dcplx sq = cmk(P.Sr[(size_t)(l + q) * Spad + kk], P.Sr[(size_t)(l + q) * Spad + kk + 1]);
            const double t2 = odd ? YI(q) : YR(q), t2o = odd ? YR(q) : YI(q), zo_ = __shfl_xor_sync(kAll, z, SC);
            // crot_out: c z - conj(s) t2; crot_next: c t2 + s z.
            const double m = sq.im * t2o;
            const double q2 = fma(sq.re, t2, odd ? neg(m) : m);
            const double zo = fma(cq, z, neg(q2));
            const double mz = sq.im * zo_;
            const double p2 = fma(sq.re, z, odd ? mz : neg(mz));
            z = fma(cq, t2, p2);
            if (st) P.Zs[(size_t)q * Spad + k + (odd ? 1 : 0)] = zo;
            zmx = umax64(zmx, abs_bits(absd(zo) + absd(__shfl_xor_sync(kAll, zo, SC))));
        }
        const double zc = __shfl_xor_sync(kAll, z, SC);
        zmx = umax64(zmx, abs_bits(absd(z) + absd(zc)));
        if (st) P.zlast[k + (odd ? 1 : 0)] = z;
        if (act && store_lane) {
            P.z2n[k] = from_bits(zmx);
            const dcplx q0 = cmulc(s0, cmk(YR(0), YI(0)));
            P.ytil[k] = -q0.re;
            P.ytil[k + 1] = -q0.im;
        }
    }
#undef VR
#undef VI
#undef YR
#undef YI
#undef SA
#undef SX
#undef SB
#undef PM
#undef HCOL
}

// Pairs per CTA of the narrow form (0: the wide one): the smallest that fits
// one wave.
int diag_c_narrow(int np) {
    const int sms = device_sms();
    for (int sc = 4; sc <= 16; sc *= 2)
        if ((np + sc - 1) / sc <= sms) return sc;
    return 0;
}
template <int SC>
cudaError_t launch_diag_cn(const DevProblem &P, int J, int b, cudaStream_t st) {
    static size_t configured = 0;
    const size_t smem = diag_cn_smem_bytes<SC>(b);
    const cudaError_t e = raise_smem_limit((const void *)k_diag_cn<SC>, &configured, smem);
    if (e != cudaSuccess) return e;
    k_diag_cn<SC><<<(P.S / 2 + SC - 1) / SC, 32 * kNarrowCWarps, smem, st>>>(P, J);
    return cudaGetLastError();
}

// The dynamic shared-memory limit of each k_diag_c form only ever grows.
template <int NW>
cudaError_t diag_c_smem_attr(size_t smem) {
    static size_t configured = 0;
    return raise_smem_limit((const void *)k_diag_c<NW>, &configured, smem);
}

cudaError_t launch_diag_c(const DevProblem &P, int J, int b, double *gscratch, cudaStream_t st) {
    // (A tile too high for the narrow form's shared memory takes the wide one.)
    const int sc = diag_c_narrow(P.S / 2);
    if (sc == 4 && diag_cn_smem_bytes<4>(b) <= kNarrowCSmem) return launch_diag_cn<4>(P, J, b, st);
    if (sc == 8 && diag_cn_smem_bytes<8>(b) <= kNarrowCSmem) return launch_diag_cn<8>(P, J, b, st);
    if (sc == 16 && diag_cn_smem_bytes<16>(b) <= kNarrowCSmem) return launch_diag_cn<16>(P, J, b, st);
    bool gvy = false;
    const size_t smem = diag_c_smem_bytes(b, &gvy);
    if (gvy && !gscratch) return cudaErrorInvalidValue;
    const int grid = (P.S / 2 + 31) / 32;
    if (gscratch) {
        const size_t small = diagc_small_bytes(b, kDiagWarpsC);
        const cudaError_t e = diag_c_smem_attr<kDiagWarpsC>(small);
        if (e != cudaSuccess) return e;
        k_diag_c<kDiagWarpsC><<<grid, 32 * kDiagWarpsC, small, st>>>(P, J, gscratch);
    } else {
        const cudaError_t e = diag_c_smem_attr<kDiagWarpsCSmem>(smem);
        if (e != cudaSuccess) return e;
        k_diag_c<kDiagWarpsCSmem><<<grid, 32 * kDiagWarpsCSmem, smem, st>>>(P, J, nullptr);
    }
    return cudaGetLastError();
}

int diag_c_ctas_per_sm(int b) {
    bool gvy = false;
    const size_t smem = diag_c_smem_bytes(b, &gvy);
    if (gvy) return 0;
    if (diag_c_smem_attr<kDiagWarpsCSmem>(smem) != cudaSuccess) return 0;
    int nb = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_diag_c<kDiagWarpsCSmem>, 32 * kDiagWarpsCSmem,
                                                      smem) != cudaSuccess)
        return 0;
    return nb;
}

// --------------------------------------------------------------- Part 1
// The real k_part1 in complex arithmetic: lane per pair for the exact
// no-rescale test, one warp per (tile, pair) for the full Part 1.  The test
// of hsr_kernels.cu (part1_fast) holds with cabs1 bounds: with hn,
// cabs1(mu), cabs1(ytilde) < 2^496 and Yn < 2^993, each updated entry has
// cabs1 <= (2^993 + 2^992 + 2^992)(1+u)^3 < 2^995, so with Hn, ||Ytilde2|| <
// 2^497 neither decision can fire.
__device__ __forceinline__ bool part1_fast_c(double Xs, double Ys, double hn, double mu1, double yt1, double Yn,
                                             double Hn, double z2) {
    return ubits(Xs) == ubits(Ys) && mag(hn) < pow2_bits(496) && mag(mu1) < pow2_bits(496) &&
           mag(yt1) < pow2_bits(496) && mag(Yn) < pow2_bits(993) && mag(Hn) < pow2_bits(497) &&
           mag(z2) < pow2_bits(497);
}

__device__ __noinline__ void part1_full_c(const DevProblem &P, int J, int I, int pidx) {
    const int lane = threadIdx.x & 31;
    const bool is = P.is != 0;
    const size_t Spad = (size_t)P.Spad;
    const int T = P.T;
    const int k = 2 * pidx;
    const int r0 = P.fr[I], m = P.fr[I + 1] - r0;
    const int l = P.fr[J], b = P.fr[J + 1] - l;
    const bool applyShift = (I == J - 1);
    double *yr = P.X + r0 + (size_t)k * P.ldx, *yi = yr + P.ldx;
    const double *h = P.H + r0 + (size_t)(l - 1) * P.ldh;
    const dcplx mu = cmk(P.wr[k], P.wr[k + 1]);
    double Ys = P.beta[(size_t)I * Spad + k];
    const double Xs = P.beta[(size_t)J * Spad + k];
    double Yn = P.ynorm[(size_t)I * Spad + k];

    // Part 0: consistent scaling.
    if (Xs < Ys) {
        const double a = sc_upscale(Xs, Ys, is);
        if (!is_one(a))
            for (int i = lane; i < m; i += 32) {
                yr[i] = a * yr[i];
                yi[i] = a * yi[i];
            }
        Yn = a * Yn;
        Ys = Xs;
    }
    // Part 1: y -= (H(I, l-1) - mu e_last) ytilde, ytilde = -conj(sigma_0) x_0.
    dcplx x0 = cmk(P.X[l + (size_t)k * P.ldx], P.X[l + (size_t)(k + 1) * P.ldx]);
    if (Ys < Xs) x0 = cscal(sc_upscale(Ys, Xs, is), x0);
    const dcplx s0 = cmk(P.Sr[(size_t)l * Spad + k], P.Sr[(size_t)l * Spad + k + 1]);
    const dcplx q0 = cmulc(s0, x0);
    const dcplx yt = cmk(-q0.re, -q0.im);
    const double hnrm = P.hn[I + (size_t)J * T];
    const double alpha = protect_update(fmax(hnrm, cabs1(mu)), cabs1(yt), Yn, is);
    const double a = sc_value(alpha, is);
    unsigned long long mx = 0;
    if (!is_one(a)) {
        const dcplx at = cscal(a, yt);
        for (int i = lane; i < m; i += 32) {
            dcplx v = cmk(fma(-h[i], at.re, a * yr[i]), fma(-h[i], at.im, a * yi[i]));
            if (applyShift && i == m - 1) v = cfma(mu, at, v);
            yr[i] = v.re;
            yi[i] = v.im;
            mx = umax64(mx, abs_bits(cabs1(v)));
        }
    } else {
        for (int i = lane; i < m; i += 32) {
            dcplx v = cmk(fma(-h[i], yt.re, yr[i]), fma(-h[i], yt.im, yi[i]));
            if (applyShift && i == m - 1) v = cfma(mu, yt, v);
            yr[i] = v.re;
            yi[i] = v.im;
            mx = umax64(mx, abs_bits(cabs1(v)));
        }
    }
    Ys = sc_combine(Ys, alpha, is);
    for (int o = 16; o; o >>= 1) mx = umax64(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    Yn = from_bits(mx);

    // Part 2 decision.
    bool slow = false;
    double z2 = P.z2n[k];
    double *zs = P.Zslow + (size_t)I * P.tlsz * Spad + k;      // re at zs[q*Spad], im at +1
    if (Ys < Xs) {
        slow = true;
        const double a2 = sc_upscale(Ys, Xs, is);
        const double *xr = P.X + l + (size_t)k * P.ldx, *xi = xr + P.ldx;
        unsigned long long zmx = 0;
        dcplx z = cscal(P.Cr[(size_t)l * Spad + k], cscal(a2, cmk(xr[0], xi[0])));
        for (int q = 1; q < b; ++q) {
            const double cq = P.Cr[(size_t)(l + q) * Spad + k];
            const dcplx sq = cmk(P.Sr[(size_t)(l + q) * Spad + k], P.Sr[(size_t)(l + q) * Spad + k + 1]);
            const dcplx t2 = cscal(a2, cmk(xr[q], xi[q]));
            const dcplx zo = crot_out(cq, sq, z, t2);
            z = crot_next(cq, sq, z, t2);
            if (lane == 0) {
                zs[(size_t)(q - 1) * Spad] = zo.re;
                zs[(size_t)(q - 1) * Spad + 1] = zo.im;
            }
            zmx = umax64(zmx, abs_bits(cabs1(zo)));
        }
        zmx = umax64(zmx, abs_bits(cabs1(z)));
        if (lane == 0) {
            zs[(size_t)(b - 1) * Spad] = z.re;
            zs[(size_t)(b - 1) * Spad + 1] = z.im;
        }
        z2 = from_bits(zmx);
    }
    const double tsc = protect_update(P.Hn[I + (size_t)J * T], z2, Yn, is);
    const double ta = sc_value(tsc, is);
    if (!is_one(ta)) {
        if (!slow) {
            for (int q = lane; q < b - 1; q += 32) {
                zs[(size_t)q * Spad] = P.Zs[(size_t)(q + 1) * Spad + k];
                zs[(size_t)q * Spad + 1] = P.Zs[(size_t)(q + 1) * Spad + k + 1];
            }
            if (lane == 0) {
                zs[(size_t)(b - 1) * Spad] = P.zlast[k];
                zs[(size_t)(b - 1) * Spad + 1] = P.zlast[k + 1];
            }
            __syncwarp();
        }
        slow = true;
        __syncwarp();
        for (int q = lane; q < b; q += 32) {
            zs[(size_t)q * Spad] = ta * zs[(size_t)q * Spad];
            zs[(size_t)q * Spad + 1] = ta * zs[(size_t)q * Spad + 1];
        }
        for (int i = lane; i < m; i += 32) {
            yr[i] = ta * yr[i];
            yi[i] = ta * yi[i];
        }
        Ys = sc_combine(Ys, tsc, is);
    }
    __syncwarp();
    if (lane == 0) {
        P.beta[(size_t)I * Spad + k] = Ys;
        P.ynorm[(size_t)I * Spad + k] = 0.0;
        P.slow[(size_t)I * Spad + k] = slow ? 1 : 0;
    }
    __syncwarp();
}

__global__ void __launch_bounds__(256) k_part1_c(DevProblem P, int J) {
    const int lane = threadIdx.x & 31;
    const int np = P.S / 2;
    const int pw = blockIdx.x * kPart1Shifts + (threadIdx.x >> 5) * 32;
    if (pw >= np) return;
    const int pidx = pw + lane;
    const bool act = pidx < np;
    const int k = 2 * pidx;
    const size_t Spad = (size_t)P.Spad;
    const size_t T = (size_t)P.T;
    double mu1 = 0.0, yt1 = 0.0, z2 = 0.0, Xs = 0.0;
    if (act) {
        mu1 = cabs1(cmk(P.wr[k], P.wr[k + 1]));
        yt1 = cabs1(cmk(P.ytil[k], P.ytil[k + 1]));
        z2 = P.z2n[k];
        Xs = P.beta[(size_t)J * Spad + k];
    }
    bool any = false;
    if (act) {
        for (int I = 0; I < J; ++I) {
            const size_t ik = (size_t)I * Spad + k;
            if (part1_fast_c(Xs, P.beta[ik], P.hn[I + J * T], mu1, yt1, P.ynorm[ik], P.Hn[I + J * T], z2)) {
                P.ynorm[ik] = 0.0;
                P.slow[ik] = 2;
            } else {
                any = true;
            }
        }
    }
    if (!__any_sync(0xffffffffu, any)) return;
    for (int I = 0; I < J; ++I) {
        bool pend = false;
        if (act) {
            const size_t ik = (size_t)I * Spad + k;
            pend = !part1_fast_c(Xs, P.beta[ik], P.hn[I + J * T], mu1, yt1, P.ynorm[ik], P.Hn[I + J * T], z2);
        }
        unsigned msk = __ballot_sync(0xffffffffu, pend);
        while (msk) {
            const int src = __ffs(msk) - 1;
            msk &= msk - 1;
            part1_full_c(P, J, I, pw + src);
        }
    }
}

cudaError_t launch_part1_c(const DevProblem &P, int J, cudaStream_t st) {
    const int np = P.S / 2;
    k_part1_c<<<(np + kPart1Shifts - 1) / kPart1Shifts, 256, 0, st>>>(P, J);
    return cudaGetLastError();
}

}  // namespace hsr
