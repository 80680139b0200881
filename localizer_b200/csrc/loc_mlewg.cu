// MLEwG fits on the GPU: maximum-likelihood Gaussian localization with a
// Nelder-Mead simplex (reference FitPositions_MLEwG::fit_positions,
// source/Localization.cpp:633-789; objective MinimizationFunction_MLEwG
// :1333-1362, position deviation CalculateMLEwGVariance :1364-1374).
//
// In FP64 and in the reference's operation order, one warp per candidate:
// this file is compiled without fused multiply-add contraction, the objective
// sums the pixels row by row as the reference does, and the simplex follows
// the same restated minimiser as the CPU oracle (GSL nmsimplex2: reflect,
// expand by 2, contract by 0.5, shrink to the best corner; centre and squared
// size updated incrementally; BLAS-style norm, dot and axpy). Start: centre at
// the candidate, width w0, background from the candidate, integral
// 2 pi w0^2 x intensity, unit steps; stop when the simplex size falls below
// 1e-2 or after 200 iterations. Rejects, in the reference's order: integral
// <= 0, centre outside the ROI, centre moved by more than 2 w0, integral
// outside [1/2, 3/2] of the start, width outside [1/2, 3/2] w0.
#include "../../include/localizer_b200.h"
#include "loc_div.h"
#include "loc_fit.cuh"

#include <cuda_runtime.h>
#include <math_constants.h>

#include <cmath>
#include <cstdint>

namespace locb {

namespace {

constexpr int N = 5, NP = 6;
constexpr double kPi = 3.1415926535897932384626433;   // the reference's PI (Defines.h:97)

struct MlCand {
    double x, y, intensity, background;
    int32_t frame, half_width;
};

// ---------------------------------------------------------------------------
// One warp per fit. The fit is a serial chain of objective evaluations (about
// 340 of them over its 200 iterations), each a sum over the ROI whose order
// the reference fixes, so a thread per fit spends its time in the latency of
// exp, log, lgamma and two divisions per pixel (16,800 fits of mixed 7 to 13 px
// ROIs: 72.3 ms that way, 13.7 ms this way). Here the 32 lanes evaluate the
// pixels' terms in parallel and every lane then adds the terms in the
// reference's order; the terms that do not change during a fit
// (lgamma(d + 1)) are evaluated once, and the divisions by the trial width
// use its reciprocal (div_by). The simplex is spread over the lanes, lane j
// holding coordinate j of every corner: a corner update is one instruction
// instead of five. The bound is now FP64 issue (about 85 FP64 operations a
// pixel and one addition of the ordered sum per term).
// ---------------------------------------------------------------------------
constexpr int kWarps = 4;      // fits per block
constexpr int kChunk = 64;     // terms summed per trip: two per lane
constexpr unsigned kAll = 0xffffffffu;

// Shared memory of one fit: lgamma(d + 1) and the pixel values, then one
// chunk of terms.
__host__ __device__ constexpr int smem_px(int r) { return ((2 * r + 1) * (2 * r + 1) + 7) / 8 * 8; }
__host__ __device__ constexpr int smem_per_fit(int r) { return kChunk * 8 + smem_px(r) * 8 + smem_px(r) * 2; }

struct RoiView {
    double *term;        // kChunk doubles
    const double *lg;    // lgamma(d + 1) per pixel
    const uint16_t *px;
    int s, npx;
    int di, dj;          // 32 pixels further: dj rows down and di to the right
    double xoff, yoff;
};

// the negative log-likelihood at (x0, y0, sd, bg, nph), the same on every lane
__device__ __forceinline__ double objective(double x0, double y0, double sd, double bg, double nph,
                                            const RoiView &roi, int lane)
{
    const double norm = nph / (2 * kPi * sd * sd);
    const double inv = 1.0 / sd;
    const bool fast = div_fast(sd);
    double sum = 0.0;
    // this lane's pixel in the frame, kept in FP64 (small integers: exact)
    const int j0 = lane / roi.s;
    int i = lane - j0 * roi.s;
    double x = roi.xoff + (double)i, y = roi.yoff + (double)j0;
    const double dx = (double)roi.di, dy = (double)roi.dj, side = (double)roi.s;
    for (int k0 = 0; k0 < roi.npx; k0 += kChunk) {
        __syncwarp();   // the previous chunk's terms have been read
        // one copy in the code: with two side by side the instruction fetches
        // cost more than the overlap gave (16 800 fits: 15.0 -> 13.7 ms)
#pragma unroll 1
        for (int u = 0; u < 2; ++u) {
            const int k = k0 + u * 32 + lane;
            double t = 0.0;
            if (k < roi.npx) {
                const double d = (double)roi.px[k];
                const double num = -((x - x0) * (x - x0) + (y - y0) * (y - y0));
                const double arg = fast && (in_range(num) || num == 0.0) ? div_by(div_by(num, sd, inv), sd, inv)
                                                                         : num / sd / sd;
                const double e = norm * exp(arg) + bg;
                t = -e + d * log(e) - roi.lg[k];
            }
            roi.term[u * 32 + lane] = t;
            i += roi.di;
            x += dx;
            y += dy;
            if (i >= roi.s) {
                i -= roi.s;
                x -= side;
                y += 1.0;
            }
        }
        __syncwarp();
        const double2 *tp = reinterpret_cast<const double2 *>(roi.term);
        const int cnt = min(kChunk, roi.npx - k0);
        if (cnt == kChunk) {
#pragma unroll 4
            for (int c = 0; c < kChunk / 2; ++c) {
                const double2 w = tp[c];
                sum += w.x;
                sum += w.y;
            }
        } else {
#pragma unroll 4
            for (int c = 0; c < cnt / 2; ++c) {
                const double2 w = tp[c];
                sum += w.x;
                sum += w.y;
            }
            if (cnt & 1) sum += roi.term[cnt - 1];
        }
    }
    return -1.0 * sum;
}

// the objective at the point whose coordinate j lane j holds
__device__ __forceinline__ double objective_at(double xj, const RoiView &roi, int lane)
{
    return objective(__shfl_sync(kAll, xj, 0), __shfl_sync(kAll, xj, 1), __shfl_sync(kAll, xj, 2),
                     __shfl_sync(kAll, xj, 3), __shfl_sync(kAll, xj, 4), roi, lane);
}

// BLAS-style norm of the vector spread over lanes 0..4, in the serial
// routine's operations: the running scale before each element is the
// largest magnitude of the earlier ones, so each lane divides for its own
// element and the five quotients are then folded in order.
__device__ __forceinline__ double dnrm2(double xj, int j)
{
    double ax[N];
#pragma unroll
    for (int k = 0; k < N; k++) ax[k] = fabs(__shfl_sync(kAll, xj, k));
    // NaN never raises the scale (the serial routine's comparison is false)
    double before = 0.0, mine = ax[0], scale = 0.0;
#pragma unroll
    for (int k = 0; k < N; k++) {
        if (k == j) {
            before = scale;
            mine = ax[k];
        }
        if (scale < ax[k]) scale = ax[k];
    }
    const bool grows = before < mine;
    const double ratio = grows ? before / mine : mine / before;
    double ssq = 1.0, run = 0.0;
#pragma unroll
    for (int k = 0; k < N; k++) {
        const double q = __shfl_sync(kAll, ratio, k);
        if (ax[k] != 0.0) {
            if (run < ax[k]) {
                ssq = 1.0 + ssq * q * q;
                run = ax[k];
            } else {
                ssq += q * q;
            }
        }
    }
    return run * sqrt(ssq);
}

// Corners by coordinate: lane j holds x1[i] = coordinate j of corner i (lanes
// past the last coordinate repeat it); the function values and the squared
// size are the same on every lane.
struct Simplex {
    double x1[NP];
    double y1[NP];
    double center;
    double S2;
};

__device__ __forceinline__ double corner_of(const double (&v)[NP], int i)
{
    double r = v[0];
#pragma unroll
    for (int k = 1; k < NP; k++) r = i == k ? v[k] : r;
    return r;
}

__device__ __forceinline__ void compute_center(Simplex &s)
{
    s.center = 0.0;
#pragma unroll
    for (int i = 0; i < NP; i++) s.center += 1.0 * s.x1[i];
    s.center *= 1.0 / NP;
}

__device__ __forceinline__ double compute_size(Simplex &s, int j)
{
    double ss = 0.0;
#pragma unroll
    for (int i = 0; i < NP; i++) {
        const double t = dnrm2(s.x1[i] + -1.0 * s.center, j);
        ss += t * t;
    }
    s.S2 = ss / NP;
    return sqrt(ss / NP);
}

__device__ __forceinline__ double trial_corner(double coeff, const Simplex &s, int corner)
{
    const double alpha = (1 - coeff) * NP / (NP - 1.0);
    const double beta = (NP * coeff - 1.0) / (NP - 1.0);
    return s.center * alpha + beta * corner_of(s.x1, corner);
}

__device__ __forceinline__ void update_point(Simplex &s, int i, double x, double val, int j)
{
    const double xo = corner_of(s.x1, i);
    const double delta = x + -1.0 * xo;
    const double xmc = xo + -1.0 * s.center;
    const double d = dnrm2(delta, j);
    const double prod = xmc * delta;
    double xmcd = 0.0;
#pragma unroll
    for (int k = 0; k < N; k++) xmcd += __shfl_sync(kAll, prod, k);
    s.S2 += (2.0 / NP) * xmcd + ((NP - 1.0) / NP) * (d * d / NP);
    const double a = 1.0 / NP;
    s.center += -a * xo;
    s.center += a * x;
#pragma unroll
    for (int k = 0; k < NP; k++) {
        if (k == i) {
            s.x1[k] = x;
            s.y1[k] = val;
        }
    }
}

// 0 ok, 5 failed contraction (non-finite values)
__device__ __forceinline__ int nm_iterate(Simplex &s, const RoiView &roi, double &x, double &size, int lane, int j)
{
    int hi = 0, lo = 0, s_hi = 1;
    double dhi = s.y1[0], dlo = s.y1[0], ds_hi = s.y1[1];
#pragma unroll
    for (int i = 1; i < NP; i++) {
        const double v = s.y1[i];
        if (v < dlo) {
            dlo = v;
            lo = i;
        } else if (v > dhi) {
            ds_hi = dhi;
            s_hi = hi;
            dhi = v;
            hi = i;
        } else if (v > ds_hi) {
            ds_hi = v;
            s_hi = i;
        }
    }
    // The trials of one iteration share one objective call site: the
    // reflection, then the expansion or the contraction, then the corners of
    // a shrink (the objective inlined once keeps the loop in the
    // instruction cache).
    const double ylo = corner_of(s.y1, lo), yhi = corner_of(s.y1, hi), yshi = corner_of(s.y1, s_hi);
    enum { REFLECT, EXPAND, CONTRACT, SHRINK };
    int step = REFLECT, corner = -1;
    double xr = trial_corner(-1.0, s, hi), xt = xr, val = 0.0;
    bool bad = false, done = false;
    while (!done) {
        const double v = objective_at(xt, roi, lane);
        if (step == REFLECT) {
            val = v;
            if (isfinite(val) && val < ylo) {
                step = EXPAND;
                xt = trial_corner(-2.0, s, hi);
            } else if (!isfinite(val) || val > yshi) {
                if (isfinite(val) && val <= yhi) update_point(s, hi, xr, val, j);
                step = CONTRACT;
                xt = trial_corner(0.5, s, hi);
            } else {
                // better than the second-worst corner: replace the worst by the reflection
                update_point(s, hi, xr, val, j);
                done = true;
            }
        } else if (step == EXPAND) {
            const bool take = isfinite(v) && v < ylo;
            update_point(s, hi, take ? xt : xr, take ? v : val, j);
            done = true;
        } else if (step == CONTRACT) {
            if (isfinite(v) && v <= corner_of(s.y1, hi)) {
                update_point(s, hi, xt, v, j);
                done = true;
            } else {
                step = SHRINK;
            }
        } else {
#pragma unroll
            for (int k = 0; k < NP; k++)
                if (k == corner) s.y1[k] = v;
            if (!isfinite(v)) bad = true;
        }
        if (step == SHRINK && !done) {
            if (++corner == lo) ++corner;
            if (corner < NP) {
                const double xl = corner_of(s.x1, lo);
#pragma unroll
                for (int k = 0; k < NP; k++)
                    if (k == corner) s.x1[k] = 0.5 * (s.x1[k] + xl);
                xt = corner_of(s.x1, corner);
            } else {
                compute_center(s);
                compute_size(s, j);
                if (bad) return 5;
                done = true;
            }
        }
    }
    lo = 0;
    double best = s.y1[0];
#pragma unroll
    for (int i = 1; i < NP; i++)
        if (s.y1[i] < best) {
            best = s.y1[i];
            lo = i;
        }
    x = corner_of(s.x1, lo);
    size = s.S2 > 0 ? sqrt(s.S2) : compute_size(s, j);
    return 0;
}

struct MlArgs {
    const uint16_t *frames;
    int n_frames, n_rows, n_cols;
    const MlCand *cands;
    int n;
    double w0;
    int r_default, r_cap;
    double *out;      // n x 10
    uint8_t *flags;
    float *params_out;
    unsigned long long *stats;
};

__global__ void __launch_bounds__(32 * kWarps, 4) k_mlewg(MlArgs a)
{
    extern __shared__ __align__(16) unsigned char sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ci = blockIdx.x * kWarps + warp;
    if (ci >= a.n) return;
    const int j = lane < N ? lane : N - 1;   // the coordinate this lane holds
    constexpr int ncol = 10;
    double *row = a.out + (size_t)ci * ncol;
    const MlCand c = a.cands[ci];
    auto reject = [&](uint8_t flag) {
        if (lane == 0) {
            row[0] = (double)c.frame;
            a.flags[ci] = flag;
        }
        if (lane >= 1 && lane < ncol - 2) row[lane] = CUDART_NAN;
    };
    if (lane >= ncol - 2 && lane < ncol) row[lane] = 0.0;
    const bool finite = isfinite(c.x) && isfinite(c.y) && isfinite(c.intensity) && isfinite(c.background);
    const int r = c.half_width > 0 ? c.half_width : a.r_default;
    if (!finite || c.frame < 0 || c.frame >= a.n_frames || c.half_width < 0 || r < 1 || r > a.r_cap) {
        reject(10);
        return;
    }
    const int s = 2 * r + 1;
    // Localization.cpp:694-704; in double, as a position far outside does not fit an int
    const double xod = floor(c.x - (double)r), yod = floor(c.y - (double)r);
    if (xod < 0 || xod + 2 * r > a.n_rows - 1 || yod < 0 || yod + 2 * r > a.n_cols - 1) {
        reject(1);
        return;
    }
    const int xo = (int)xod, yo = (int)yod, xm = xo + s - 1, ym = yo + s - 1;
    const int npx = s * s, room = smem_px(a.r_cap);
    unsigned char *mine = sm + warp * smem_per_fit(a.r_cap);
    double *term = reinterpret_cast<double *>(mine), *lg = term + kChunk;
    uint16_t *px = reinterpret_cast<uint16_t *>(lg + room);
    const uint16_t *base = a.frames + (size_t)c.frame * a.n_rows * a.n_cols + xo + (size_t)yo * a.n_rows;
    for (int k = lane; k < npx; k += 32) {
        const int jj = k / s, ii = k - jj * s;
        const uint16_t p = base[ii + (size_t)jj * a.n_rows];
        px[k] = p;
        lg[k] = lgamma((double)p + 1.0);
    }
    __syncwarp();
    const RoiView roi{term, lg, px, s, npx, 32 % s, 32 / s, (double)xo, (double)yo};
    const double integral = c.intensity * 2.0 * CUDART_PI * a.w0 * a.w0;
    double x = j == 0 ? c.x : j == 1 ? c.y : j == 2 ? a.w0 : j == 3 ? c.background : integral;
    // set: corner 0 at the start, corner i+1 one unit further along axis i
    Simplex sp;
    int status = 0;
    const double start = x;
#pragma unroll
    for (int i = 0; i < NP; i++) {
        sp.x1[i] = i == j + 1 ? start + 1.0 : start;
        sp.y1[i] = 0.0;
    }
    for (int i = 0; i < NP && status == 0; i++) {
        const double v = objective_at(corner_of(sp.x1, i), roi, lane);
        if (!isfinite(v)) status = 9;
#pragma unroll
        for (int k = 0; k < NP; k++)
            if (k == i) sp.y1[k] = v;
    }
    long iterations = 0;
    if (status == 0) {
        compute_center(sp);
        double size = compute_size(sp, j);
        int test = 1;
        do {
            iterations++;
            const int st = nm_iterate(sp, roi, x, size, lane, j);
            if (st != 0) {
                status = st;
                break;
            }
            test = size < 1e-2 ? 0 : 1;
        } while (test == 1 && iterations < 200);
        if (status == 0) status = test;   // 0 converged, 1 iteration cap
    }
    if (a.stats && lane == 0) {
        atomicAdd(&a.stats[4], 1ull);
        atomicAdd(&a.stats[5], (unsigned long long)iterations);
    }
    if (lane == 0) {
        row[ncol - 2] = (double)iterations;
        row[ncol - 1] = (double)status;
    }
    if (a.params_out && lane < N) a.params_out[(size_t)ci * N + lane] = (float)x;
    if (status == 9) {   // non-finite objective at the start: the simplex was never set up
        reject(10);
        return;
    }
    const double fx = __shfl_sync(kAll, x, 0), fy = __shfl_sync(kAll, x, 1), fw = __shfl_sync(kAll, x, 2),
                 fb = __shfl_sync(kAll, x, 3), fn = __shfl_sync(kAll, x, 4);
    // Localization.cpp:739-768
    if (fn <= 0) {
        reject(2);
        return;
    }
    if (fx < xo || fx > xm || fy < yo || fy > ym) {
        reject(3);
        return;
    }
    if (fabs(fx - c.x) > 2.0 * a.w0 || fabs(fy - c.y) > 2.0 * a.w0) {
        reject(5);
        return;
    }
    if (fn < integral / 2.0 || fn > integral * 1.5) {
        reject(11);
        return;
    }
    if (fw < a.w0 / 2.0 || fw > a.w0 * 1.5) {
        reject(4);
        return;
    }
    if (lane != 0) return;
    // CalculateMLEwGVariance (Localization.cpp:1364-1374)
    const double sigmaA = a.w0 * a.w0 + 1.0 / 12.0;
    const double var = sigmaA * sigmaA / fn * (16.0 / 9.0 + 8 * CUDART_PI * a.w0 * a.w0 * fb / fn);
    row[0] = (double)c.frame;
    row[1] = fn;
    row[2] = fw;
    row[3] = fx;
    row[4] = fy;
    row[5] = fb;
    row[6] = sqrt(var);
    row[7] = 1.0;
    a.flags[ci] = 0;
}

}  // namespace

cudaError_t enqueue_mlewg(const FitParams &p, unsigned long long *stats, cudaStream_t stream)
{
    if (p.n_cands == 0) return cudaSuccess;
    MlArgs a{p.frames, p.n_frames, p.n_rows, p.n_cols, static_cast<const MlCand *>(p.cands), p.n_cands, p.w0,
             (int)std::ceil(p.w0 * 4.0),
             p.max_half_width > 0 ? (p.max_half_width < kMaxHalfWidth ? p.max_half_width : kMaxHalfWidth)
                                  : kMaxHalfWidth,
             p.out, p.flags, p.params_out, stats};
    // a block's fits at the largest ROI the call admits: 45 KB at half-width 16
    const int smem = kWarps * smem_per_fit(a.r_cap);
    const cudaError_t e =
        cudaFuncSetAttribute(k_mlewg, cudaFuncAttributeMaxDynamicSharedMemorySize, kWarps * smem_per_fit(kMaxHalfWidth));
    if (e != cudaSuccess) return e;
    k_mlewg<<<(p.n_cands + kWarps - 1) / kWarps, 32 * kWarps, smem, stream>>>(a);
    if (p.launches) ++*p.launches;
    return cudaGetLastError();
}

}  // namespace locb
