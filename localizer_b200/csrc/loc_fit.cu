// Fit kernels of the B200 localization engine.
//
//   K0 classify / classes / scatter — validate candidates, apply the edge
//      reject of the reference (Localization.cpp:115-124), and build a work
//      queue grouped by ROI half-width (largest first).
//   K1 lm_fit — persistent solver: one thread per fit, a warp refills its
//      idle lanes from the queue with one atomic and stages their ROIs from
//      the HBM-resident uint16 frames with warp-cooperative loads into shared
//      memory; every loop trip is one model/Jacobian/normal-equation pass
//      for all active lanes (see loc_device.cuh). Level 0 solves fresh fits
//      per ROI side, level 1 (8 threads per fit) a list of suspended ones; the
//      FP64 re-run walks lists as well.
//   team (loc_team.cuh) — a warp or a block per fit, where latency counts.
//   K3 flag — which FP32 fits are re-run in FP64.
//   K2 finalize — FP64: covariance (J^T J)^-1, uncertainty scaling, the
//      reference's accept/reject rules and output columns.
#include "loc_device.cuh"
#include "loc_fit.cuh"

#include <math_constants.h>

#include <cmath>
#include <cstdio>

namespace locb {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int K = kMaxHalfWidth + 1;
// header: ROI classes present, largest half-width; length and dequeue cursor
// of the queue, of the fits past the first level's budget, and of the fits
// left to the teams. The FP64 re-run's tables (meta2, meta3) use the first
// and the last pair.
constexpr int M_NCLS = 0, M_MAXR = 1, M_TOTAL = 2, M_NEXT = 3, M_NCONT = 4, M_CONTNEXT = 5, M_NLEFT = 6, M_LEFTNEXT = 7;
// per ROI half-width r: queue start, count, dequeue cursor, histogram, fill cursor
__host__ __device__ constexpr int m_start(int r) { return 8 + 1 * K + r; }
__host__ __device__ constexpr int m_count(int r) { return 8 + 2 * K + r; }
__host__ __device__ constexpr int m_next(int r) { return 8 + 3 * K + r; }
__host__ __device__ constexpr int m_hist(int r) { return 8 + 4 * K + r; }
__host__ __device__ constexpr int m_fill(int r) { return 8 + 5 * K + r; }

__host__ __device__ constexpr int ref_cols(int method) { return method == 0 ? 12 : method == 1 ? 10 : 16; }

struct K0Args {
    const Cand *cands;
    int n;
    int n_frames, n_rows, n_cols;
    int r_default;
    int r_cap;        // candidates whose r exceeds it are rejected as bad input
    int method;
    int ncol_total;
    double *out;
    uint8_t *flags;
    int *cls;
    int *meta;
    int *cls2;   // optional: FP64 re-run marks, cleared here
    // ROI mode: a candidate that passes the edge rule must have its ROI
    // inside the packed ROI stack (else it is flagged as bad input: the
    // solver never reads outside the stack)
    const int *roi_slot;
    long long roi_px;
};

__device__ void write_reject_row(double *row, int ncol_total, int frame)
{
    row[0] = (double)frame;
    for (int k = 1; k < ncol_total - 2; ++k) row[k] = CUDART_NAN;
    row[ncol_total - 2] = 0.0;
    row[ncol_total - 1] = 0.0;
}

__global__ void k0_classify(K0Args a)
{
    __shared__ int hist[K];
    for (int r = threadIdx.x; r < K; r += blockDim.x) hist[r] = 0;
    __syncthreads();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < a.n) {
        const Cand c = a.cands[i];
        int cls = -1;
        uint8_t flag = F_PENDING;
        const bool finite = isfinite(c.x) && isfinite(c.y) && isfinite(c.intensity) && isfinite(c.background);
        const int r = c.half_width > 0 ? c.half_width : a.r_default;
        if (!finite || c.frame < 0 || c.frame >= a.n_frames || c.half_width < 0 || r < 1 || r > a.r_cap) {
            flag = F_BAD_INPUT;
        } else {
            // Localization.cpp:115-120, integer ROI origin and far corner
            const double xo = floor(c.x - (double)r), yo = floor(c.y - (double)r);
            const double xm = xo + 2 * r, ym = yo + 2 * r;
            if (xo < 0 || xm > a.n_rows - 1 || yo < 0 || ym > a.n_cols - 1) {
                flag = F_EDGE;
            } else if (a.roi_slot && (a.roi_slot[i] < 0 ||
                                      (long long)a.roi_slot[i] + (long long)(2 * r + 1) * (2 * r + 1) > a.roi_px)) {
                flag = F_BAD_INPUT;
            } else {
                cls = r;
                atomicAdd(&hist[r], 1);
            }
        }
        a.cls[i] = cls;
        if (a.cls2) a.cls2[i] = -1;
        a.flags[i] = flag;
        if (flag != F_PENDING) write_reject_row(a.out + (size_t)i * a.ncol_total, a.ncol_total, c.frame);
    }
    __syncthreads();
    for (int r = threadIdx.x; r < K; r += blockDim.x)
        if (hist[r]) atomicAdd(&a.meta[m_hist(r)], hist[r]);
}

// One block: queue layout per half-width, largest ROIs first.
__global__ void k0_classes(int *meta)
{
    if (threadIdx.x != 0) return;
    int ncls = 0, start = 0, maxr = 0;
    for (int r = K - 1; r >= 1; --r) {
        const int cnt = meta[m_hist(r)];
        if (cnt == 0) continue;
        if (r > maxr) maxr = r;
        meta[m_start(r)] = start;
        meta[m_count(r)] = cnt;
        meta[m_next(r)] = 0;
        meta[m_fill(r)] = start;
        start += cnt;
        ++ncls;
    }
    meta[M_NCLS] = ncls;
    meta[M_MAXR] = maxr;
    meta[M_TOTAL] = start;
}

__global__ void k0_scatter(const int *cls, int n, int *meta, int *order)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = i < n ? cls[i] : -1;
    const unsigned active = __ballot_sync(kFull, c >= 0);
    if (c < 0) return;
    // warp-aggregated: one atomic per distinct class in the warp
    const unsigned peers = __match_any_sync(active, c);
    const int leader = __ffs(peers) - 1;
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == leader) base = atomicAdd(&meta[m_fill(c)], __popc(peers));
    base = __shfl_sync(peers, base, leader);
    order[base + __popc(peers & ((1u << lane) - 1))] = i;
}

// Appends i of the lanes with want to a list, one atomic per warp.
__device__ __forceinline__ void push(bool want, int i, int *list, int step, int *count)
{
    const unsigned who = __ballot_sync(kFull, want);
    if (!who) return;
    const int lane = threadIdx.x & 31, first = __ffs(who) - 1;
    int at = 0;
    if (lane == first) at = atomicAdd(count, __popc(who));
    at = __shfl_sync(kFull, at, first);
    if (want) list[(long long)(at + __popc(who & ((1u << lane) - 1))) * step] = i;
}

// Fits of the FP32 solver whose result could depend on its rounding go to an
// FP64 re-run: a branch decision of the trust-region method was within
// `margin` of its threshold, the undamped normal matrix had a pivot ratio
// below `pivot` (ill-conditioned), the solver stopped for lack of progress, or
// one of the options' rules holds. Walks a list of fits (two lists, the
// second backwards, for the suspended ones) and appends the flagged ones to
// the short or, when their FP32 solve took more than long_iters iterations
// and there is one, to the long FP64 list: the long fits set the length of the
// re-run. Fits still suspended (cls2 kSuspended) are left for the pass over
// them.
constexpr int kSuspended = -2;
struct FlagArgs {
    const float *state32;
    int stride;
    const int *list, *count, *list_b, *count_b;   // list_b[-k]
    const int *cls;
    const uint8_t *flags;
    int *cls2;
    int suspended;       // the lists hold suspended fits (all finished by now)
    int *shorts, *n_short, *longs, *n_long;       // entries at [k * step]; longs NULL: one list
    int step;
    float margin, pivot, cond, skip_rej, w0;
    int warm_limit, long_iters, capped, iters_min;
};
template <int P>
__global__ void k3_flag(FlagArgs a)
{
    using SL = StateLayout<P>;
    constexpr int IX = P == 5 ? 2 : P == 4 ? 1 : 3;
    const int n_a = *a.count, count = n_a + (a.count_b ? *a.count_b : 0);
    const float margin = a.margin, pivot = a.pivot, cond = a.cond, skip_rej = a.skip_rej, w0 = a.w0;
    const int warm_limit = a.warm_limit, capped = a.capped, iters_min = a.iters_min;
    // whole warps walk together (push)
    for (int t0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); t0 < count; t0 += gridDim.x * blockDim.x) {
        const int t = t0 + (int)(threadIdx.x & 31);
        const int i = t >= count ? 0 : t < n_a ? a.list[t] : a.list_b[-(t - n_a)];
        const int r = t < count ? a.cls[i] : 0;
        bool rerun = false, is_long = false;
        if (t < count && a.flags[i] == F_PENDING && (a.suspended || a.cls2[i] != kSuspended)) {
            if (a.suspended) a.cls2[i] = -1;
            const float *s = a.state32 + (size_t)i * a.stride;
            const float status = s[SL::STATUS];
            // warm-started fits (warm_limit > 0) that needed many iterations may
            // stop elsewhere than the reference start's trajectory would
            // capped: fits the FP32 solver stopped at the iteration cap are
            // re-run too (the FP64 solve may converge where FP32 did not)
            const bool is_capped = status == (float)T_MAX_ITER;
            // cond > 0: a branch margin is also too small when it is within the
            // FP32 error the fit's conditioning allows (cond * eps32 / smallest
            // undamped pivot ratio)
            const float mthr = cond > 0.0f ? fmaxf(margin, cond * 5.96e-8f / fmaxf(s[SL::MINPIV], 1e-30f)) : margin;
            const bool risky = is_capped ? capped != 0
                                         : (s[SL::MARGIN] < mthr || s[SL::MINPIV] < pivot || status != 0.0f ||
                                            (warm_limit > 0 && s[SL::ITERS] > (float)warm_limit) ||
                                            (iters_min > 0 && s[SL::ITERS] >= (float)iters_min));
            // skip_rej > 0: a fit whose FP32 end point lies clearly inside a reject
            // rule of the finaliser (centre more than skip_rej px outside the ROI,
            // amplitude below zero by more than skip_rej of its start scale, or
            // every width more than the fraction skip_rej outside its accepted
            // range) is not re-run: only its reject code could change
            bool clear_reject = false;
            if (risky && skip_rej > 0.0f) {
                const float side = (float)(2 * r);
                const float x = s[IX], y = s[IX + 1], A = s[0];
                clear_reject = x < -skip_rej || x > side + skip_rej || y < -skip_rej || y > side + skip_rej ||
                               A < -skip_rej * fmaxf(fabsf(s[P - 1]), 1.0f);
                const float lo = 0.4f * w0 * (1.0f - skip_rej), hi = 1.5f * w0 * (1.0f + skip_rej);
                if constexpr (P == 5) {
                    const float wd = fabsf(s[1]);
                    clear_reject = clear_reject || wd < lo || wd > hi;
                } else if constexpr (P == 7) {
                    // axes of the covariance [[sx^2, rho sx sy], [rho sx sy, sy^2]]
                    const float sx = fabsf(s[1]), sy = fabsf(s[2]), rho = s[5];
                    const float a = sx * sx, c = sy * sy, b = rho * sx * sy;
                    const float ht = 0.5f * (a + c), rad = sqrtf(0.25f * (a - c) * (a - c) + b * b);
                    const float s1 = sqrtf(fmaxf(ht - rad, 0.0f)), s2 = sqrtf(ht + rad);
                    clear_reject = clear_reject || ((s1 < lo || s1 > hi) && (s2 < lo || s2 > hi));
                }
            }
            if (risky && !clear_reject) {
                a.cls2[i] = r;
                rerun = true;
                is_long = a.longs && s[SL::ITERS] > (float)a.long_iters;
            }
        }
        push(rerun && !is_long, i, a.shorts, a.step, a.n_short);
        if (a.longs) push(is_long, i, a.longs, a.step, a.n_long);
    }
}

struct K1Args {
    const uint16_t *frames;
    long long frame_px;
    int n_rows;
    const Cand *cands;
    const int *order;
    int *meta;
    void *state;
    int state_stride;   // elements of the solver's precision per candidate
    float w0;
    float inv_s2, inv_abs_s;
    double inv_s2_d, inv_abs_s_d;
    int max_iter;
    float epsabs, epsrel;
    float pivot_thr;
    const float *init_params;
    unsigned long long *stats;
    // list mode (r = 0): a list of candidates of any ROI size instead of one
    // class's part of the queue
    const int *list, *count;
    int list_step;      // entry k at list[k * list_step]
    int *next;
    const int *cls;
    int *mark;          // optional: suspended fits are marked here (cls2)
    int resume;         // the list's fits are suspended ones
    int least;          // lists of at most this many fits are left to the teams
    int budget;         // iterations a fit may use (0: all)
    int drain;          // a warp whose queue is empty hands its fits over when at most this many
                        // of its groups still have one
    int *cont, *n_cont;     // fits past the budget
    int *left, *n_left;     // fits left to the teams (entry k at left[k * left_step])
    int left_step;
    float *cont_state;  // saved solver state of both (see save_state)
    int cont_stride;
    int compensated;    // FP32 solver: sum the group's partial normal equations in FP64
    const int *roi_slot;  // ROI mode: first pixel of each candidate's packed ROI (row pitch 2r + 1)
};

template <int METHOD, int S, int TPF, typename T> struct Pass;
template <int S, int TPF, typename T> struct Pass<0, S, TPF, T> {
    __device__ __forceinline__ static void run(const float *roi, int s, int q, bool fused, T, const T (&te)[5],
                                               const T (&dt)[5],
                                               T (&acc)[14], T (&vv)[5], T &chi2, T &dchi, T &dqmax)
    {
        pass_sym<S, TPF, T>(roi, 1, s, q, fused, te, dt, acc, vv, chi2, dchi, dqmax);
    }
};
template <int S, int TPF, typename T> struct Pass<1, S, TPF, T> {
    __device__ __forceinline__ static void run(const float *roi, int s, int q, bool fused, T w0, const T (&te)[4],
                                               const T (&dt)[4], T (&acc)[9], T (&vv)[4], T &chi2, T &dchi,
                                               T &dqmax)
    {
        pass_fixed<S, TPF, T>(roi, 1, s, q, fused, w0, te, dt, acc, vv, chi2, dchi, dqmax);
    }
};
template <int S, int TPF, typename T> struct Pass<7, S, TPF, T> {
    __device__ __forceinline__ static void run(const float *roi, int s, int q, bool, T, const T (&te)[7],
                                               const T (&dt)[7],
                                               T (&acc)[27], T (&vv)[7], T &chi2, T &dchi, T &dqmax)
    {
        pass_ell<S, TPF, T>(roi, 1, s, q, te, dt, acc, vv, chi2, dchi, dqmax);
    }
};

// Shared-memory words per fit for a ROI of npx pixels and TPF threads per
// fit: the smallest stride >= npx with stride = TPF (mod 2 TPF), so that the
// 32 lanes of a warp (32/TPF fits, TPF columns each) hit 32 distinct banks.
__host__ __device__ constexpr int roi_stride(int npx, int tpf)
{
    return npx + ((tpf - npx % (2 * tpf)) + 2 * tpf) % (2 * tpf);
}

template <typename T>
__device__ __forceinline__ T group_sum(T v, int tpf, unsigned mask)
{
    for (int o = tpf >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
    return v;
}

// Group sum of FP32 partial sums carried out in FP64 and rounded once: with
// TPF threads per fit each partial covers 1/TPF of the ROI, so the total is a
// two-level (pairwise) sum whose rounding error is that of n/TPF terms
// instead of n.
__device__ __forceinline__ float group_sum_wide(float v, int tpf, unsigned mask)
{
    double d = (double)v;
    for (int o = tpf >> 1; o > 0; o >>= 1) d += __shfl_xor_sync(mask, d, o);
    return (float)d;
}

template <typename T>
__device__ __forceinline__ T group_max(T v, int tpf, unsigned mask)
{
    for (int o = tpf >> 1; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(mask, v, o));
    return v;
}

// Saved solver state of a suspended fit: parameters, J^T J, J^T f, D, last
// step, then scalars. FP32 fits keep it in cont_state (floats). An FP64 fit
// keeps parameters and J^T J where its result goes, the scalars behind them,
// and the three vectors in its cont_state record (free once its FP32 solve is
// done), as doubles.
template <int P> struct ContLayout {
    static constexpr int NT = tri(P);
    static constexpr int TH = 0, A = P, V = P + NT, D = 2 * P + NT, DX = 3 * P + NT, SC = 4 * P + NT;
    static constexpr int STRIDE = ((SC + 11) + 3) / 4 * 4;
    static_assert(P + NT + 9 <= StateLayout<P>::STRIDE && 3 * P * 2 <= STRIDE, "FP64 state of a suspended fit");
};
template <typename T> struct Scalars {
    T fnorm, delta, par, xnorm, minpiv, margin;
    int it_state, iterations, xo, yo, q_n;   // q_n: partial sums the fit runs with (FP64)
    unsigned esc;
};

// where a suspended fit's arrays are
template <typename T> struct Saved {
    T *th, *v, *D, *dx, *A, *sc;
};
template <int P, typename T>
__device__ __forceinline__ Saved<T> saved_of(float *cont_state, int cont_stride, void *state, int state_stride, int i)
{
    using CL = ContLayout<P>;
    if constexpr (sizeof(T) == 4) {
        float *o = cont_state + (size_t)i * cont_stride;
        return Saved<T>{o + CL::TH, o + CL::V, o + CL::D, o + CL::DX, o + CL::A, o + CL::SC};
    } else {
        double *s = (double *)state + (size_t)i * state_stride;
        double *o = reinterpret_cast<double *>(cont_state + (size_t)i * cont_stride);
        return Saved<T>{s, o, o + P, o + 2 * P, s + P, s + P + CL::NT};
    }
}
template <typename T> __device__ __forceinline__ void save_scalars(T *o, const Scalars<T> &c)
{
    o[0] = c.fnorm;
    o[1] = c.delta;
    o[2] = c.par;
    o[3] = c.xnorm;
    o[4] = c.minpiv;
    o[5] = c.margin;
    if constexpr (sizeof(T) == 4) {
        o[6] = __int_as_float(c.it_state);
        o[7] = __int_as_float(c.iterations);
        o[8] = __int_as_float(c.xo);
        o[9] = __int_as_float(c.yo);
        o[10] = __uint_as_float(c.esc);
    } else {   // small integers, exact
        o[6] = (double)((long long)c.iterations * 32 + (c.it_state == 1 ? 16 : 0) + c.q_n);
        o[7] = (double)c.xo;
        o[8] = (double)c.yo;
    }
}
template <typename T> __device__ __forceinline__ Scalars<T> load_scalars(const T *o)
{
    Scalars<T> c;
    c.fnorm = o[0];
    c.delta = o[1];
    c.par = o[2];
    c.xnorm = o[3];
    c.minpiv = o[4];
    c.margin = o[5];
    if constexpr (sizeof(T) == 4) {
        c.it_state = __float_as_int(o[6]);
        c.iterations = __float_as_int(o[7]);
        c.xo = __float_as_int(o[8]);
        c.yo = __float_as_int(o[9]);
        c.esc = __float_as_uint(o[10]);
        c.q_n = 0;
    } else {
        const long long w = (long long)o[6];
        c.it_state = w & 16 ? 1 : 2;   // the solver asks only whether it is the first
        c.q_n = (int)(w & 15);
        c.iterations = (int)(w >> 5);
        c.xo = (int)o[7];
        c.yo = (int)o[8];
        c.esc = 0;
    }
    return c;
}

}  // namespace
}  // namespace locb
#include "loc_team.cuh"
namespace locb {
namespace {

// Shared memory of one fit of the solver block: its ROI, then (FP64 only) its
// state and matrices.
template <typename T>
__host__ __device__ constexpr int state_smem_per_fit(int P) { return sizeof(T) == 8 ? (3 * tri(P) + 5 * P) * 8 : 0; }
template <typename T>
__host__ __device__ constexpr int slot_bytes(int P, int r, int tpf)
{
    const int roi = roi_stride((2 * r + 1) * (2 * r + 1), tpf) * 4;
    return sizeof(T) == 8 ? (roi + 15) / 16 * 16 + (state_smem_per_fit<T>(P) + 15) / 16 * 16 : roi;
}

// Process one queue: the candidates of ROI half-width r, or (r = 0) a list of
// fits of any size, fresh or suspended. TPF threads cooperate on each fit;
// S = 2r + 1 at compile time, or 0 for a runtime side.
template <int METHOD, typename T, int S, int TPF, bool ESC>
__device__ __forceinline__ void run_class(const K1Args &a, int r_class, int smem_bytes, float *smem, unsigned (&st)[ST_N])
{
    constexpr int P = Traits<METHOD>::P;
    constexpr int NT = tri(P);
    constexpr int IX = Traits<METHOD>::IX;
    using SL = StateLayout<P>;
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int q = lane % TPF;            // sub-lane within the fit's group
    const int glead = lane - q;          // lane of the group leader
    const bool leader = q == 0;
    const bool by_list = S == 0 && r_class == 0;
    // in list mode every fit brings its own ROI size, and the block has as
    // many groups as the largest one present lets into its shared memory
    int r = by_list ? a.meta[M_MAXR] : r_class;
    const int slot = slot_bytes<T>(P, r, TPF);
    const bool has_room = !by_list || (tid / TPF + 1) * slot <= smem_bytes;
    int s = S > 0 ? S : 2 * r + 1;
    int npx = s * s;
    const int stride = slot / 4;
    float *myroi = smem + (tid / TPF) * stride;
    const int *queue = by_list ? a.list : a.order + a.meta[m_start(r)];
    const int ccount = by_list ? *a.count : a.meta[m_count(r)];
    int *next = by_list ? a.next : a.meta + m_next(r);
    const T inv_s2 = sizeof(T) == 4 ? (T)a.inv_s2 : (T)a.inv_s2_d;
    const T inv_abs_s = sizeof(T) == 4 ? (T)a.inv_abs_s : (T)a.inv_abs_s_d;
    const T w0 = (T)a.w0;

    // FP64: the normal equations, parameters, scaling, last step, the scaled
    // matrix of the damped solve and its factor live in the fit's
    // shared-memory slot (in registers they push the FP64 solver into spills)
    constexpr bool kSmemState = sizeof(T) == 8;
    T *sstate = nullptr;
    if constexpr (kSmemState)
        sstate = (T *)((char *)myroi + slot - (state_smem_per_fit<T>(P) + 15) / 16 * 16);
    StateArr<T, NT, kSmemState> A(sstate);
    StateArr<T, P, kSmemState> v(sstate ? sstate + NT : nullptr);
    StateArr<T, P, kSmemState> th(sstate ? sstate + NT + P : nullptr);
    StateArr<T, P, kSmemState> D(sstate ? sstate + NT + 2 * P : nullptr);
    StateArr<T, P, kSmemState> dx(sstate ? sstate + NT + 3 * P : nullptr);
    StateArr<T, P, kSmemState> te(sstate ? sstate + 3 * NT + 4 * P : nullptr);
    T fnorm = 0, delta = 0, par = 0, xnorm = 0, jdx2 = 0, pnorm = 0;
    int phase = 0, it_state = 0, iterations = 0, trial = 0, cidx = -1, xo = 0, yo = 0;
    T minpiv_fit = T(1);
    T margin_fit = T(1e30);
    unsigned esc_fit = 0;
    bool exhausted = !has_room;
    if (!kSmemState || has_room) {
#pragma unroll
        for (int k = 0; k < P; ++k) th[k] = v[k] = D[k] = dx[k] = te[k] = T(0);
#pragma unroll
        for (int k = 0; k < NT; ++k) A[k] = T(0);
    }

    auto theta_abs = [&](int k, auto &t) -> T {
        return k == IX ? t[k] + (T)xo : (k == IX + 1 ? t[k] + (T)yo : t[k]);
    };
    auto write_finish = [&](int status) {
        if (leader) {
            T *o = (T *)a.state + (size_t)cidx * a.state_stride;
#pragma unroll
            for (int k = 0; k < P; ++k) o[k] = th[k];
#pragma unroll
            for (int k = 0; k < NT; ++k) o[P + k] = A[k];
            o[SL::FNORM] = fnorm;
            o[SL::ITERS] = (T)iterations;
            o[SL::STATUS] = (T)status;
            o[SL::XOFF] = (T)xo;
            o[SL::YOFF] = (T)yo;
            T lastr = T(0);
#pragma unroll
            for (int k = 0; k < P; ++k) {
                const T tol = (T)a.epsabs + (T)a.epsrel * fabs(theta_abs(k, th));
                const T qq = fdiv(fabs(dx[k]), tol);
                lastr = qq > lastr ? qq : lastr;
            }
            o[SL::MINPIV] = minpiv_fit;
            o[SL::LASTR] = lastr;
            o[SL::NESC] = (T)esc_fit;
            o[SL::MARGIN] = margin_fit;
            st[ST_FITS] += 1;
            st[ST_ITERS] += iterations;
        }
    };
    // park a fit that used up its iteration budget, or whose warp has run dry
    auto write_suspend = [&](bool over) {
        if (leader) {
            const Saved<T> o = saved_of<P, T>(a.cont_state, a.cont_stride, a.state, a.state_stride, cidx);
#pragma unroll
            for (int k = 0; k < P; ++k) {
                o.th[k] = th[k];
                o.v[k] = v[k];
                o.D[k] = D[k];
                o.dx[k] = dx[k];
            }
#pragma unroll
            for (int k = 0; k < NT; ++k) o.A[k] = A[k];
            save_scalars<T>(o.sc, Scalars<T>{fnorm, delta, par, xnorm, minpiv_fit, margin_fit, it_state, iterations, xo,
                                             yo, TPF, esc_fit});
            if (a.mark) a.mark[cidx] = kSuspended;
            if (over) a.cont[atomicAdd(a.n_cont, 1)] = cidx;
            else a.left[(long long)atomicAdd(a.n_left, 1) * a.left_step] = cidx;
        }
    };
    // finish() and suspend() only mark the fit; its state is written at the
    // next flush(), before the lane is refilled (one inlined copy of each
    // write-out instead of one per call site)
    int done = -1;   // -1 nothing pending, -2 over the budget, -3 left to the teams, else the termination status
    auto finish = [&](int status) {
        done = status;
        phase = 0;
    };
    auto flush = [&]() {
        if (done == -2 || done == -3) write_suspend(done == -2);
        else if (done >= 0) write_finish(done);
        done = -1;
    };
    auto test_delta = [&]() -> bool {
        bool ok = true;
        T worst = T(0);
#pragma unroll
        for (int k = 0; k < P; ++k) {
            const T tol = (T)a.epsabs + (T)a.epsrel * fabs(theta_abs(k, th));
            ok = ok && (fabs(dx[k]) < tol);
            const T qq = fdiv(fabs(dx[k]), tol);
            worst = qq > worst ? qq : worst;
        }
        margin_fit = fmin(margin_fit, fabs(worst - T(1)));
        return ok;
    };
    bool drain = false;
    auto start_iteration = [&]() {
        if (a.budget > 0 && iterations >= a.budget) {
            finish(-2);
            return;
        }
        if (drain) {
            finish(-3);
            return;
        }
        ++iterations;
        if (fnorm == T(0)) {  // iterate() returns at once; dx is unchanged
            if (test_delta()) finish(T_CONVERGED);
            else {
                iterations = a.max_iter;
                finish(T_MAX_ITER);
            }
            return;
        }
        trial = 0;
        phase = 2;
    };

    unsigned long long c_refill = 0, c_step = 0, c_pass = 0, c_decide = 0;
    long long t_mark = clock64();
    auto lap = [&](unsigned long long &acc_c) {
        const long long t = clock64();
        acc_c += (unsigned long long)(t - t_mark);
        t_mark = t;
    };
    while (true) {
        flush();
        // ---- refill idle groups from the queue: one atomic per warp ----
        const bool want = (phase == 0) && !exhausted;
        const unsigned need = __ballot_sync(kFull, want && leader);
        if (need) {
            const int first = __ffs(need) - 1;
            int base = 0;
            if (lane == first) base = atomicAdd(next, __popc(need));
            base = __shfl_sync(kFull, base, first);
            int my = -1;
            if (want) {
                const int qi = base + __popc(need & ((1u << glead) - 1));
                if (qi < ccount) my = queue[by_list ? (long long)qi * a.list_step : qi];
                else exhausted = true;
            }
            int fr = 0;
            long long rbase = 0;   // pixel offset of the ROI origin in the pixel array
            if (my >= 0) {
                const Cand cd = a.cands[my];
                const double cx = cd.x, cy = cd.y, cint = cd.intensity, cbg = cd.background;
                fr = cd.frame;
                cidx = my;
                if (by_list) {
                    r = a.cls[my];
                    s = 2 * r + 1;
                    npx = s * s;
                }
                if (by_list && a.resume) {
                    const Saved<T> o = saved_of<P, T>(a.cont_state, a.cont_stride, a.state, a.state_stride, my);
#pragma unroll
                    for (int k = 0; k < P; ++k) {
                        th[k] = o.th[k];
                        v[k] = o.v[k];
                        D[k] = o.D[k];
                        dx[k] = o.dx[k];
                    }
#pragma unroll
                    for (int k = 0; k < NT; ++k) A[k] = o.A[k];
                    const Scalars<T> c = load_scalars<T>(o.sc);
                    fnorm = c.fnorm;
                    delta = c.delta;
                    par = c.par;
                    xnorm = c.xnorm;
                    minpiv_fit = c.minpiv;
                    margin_fit = c.margin;
                    it_state = c.it_state;
                    iterations = c.iterations;
                    xo = c.xo;
                    yo = c.yo;
                    esc_fit = c.esc;
                    phase = 3;   // start the next outer iteration after staging
                } else {
                    xo = (int)floor(cx - (double)r);
                    yo = (int)floor(cy - (double)r);
                    minpiv_fit = T(1);
                    margin_fit = T(1e30);
                    esc_fit = 0;
                    if (a.init_params && !isnan(a.init_params[(size_t)my * P])) {
                        const float *ip = a.init_params + (size_t)my * P;
    #pragma unroll
                        for (int k = 0; k < P; ++k) {
                            const double off = k == IX ? (double)xo : (k == IX + 1 ? (double)yo : 0.0);
                            th[k] = (T)((double)ip[k] - off);
                        }
                    } else {
                        const T xl = (T)(cx - (double)xo), yl = (T)(cy - (double)yo);
                        if constexpr (METHOD == 0) {
                            th[0] = (T)cint; th[1] = w0; th[2] = xl; th[3] = yl; th[4] = (T)cbg;
                        } else if constexpr (METHOD == 1) {
                            th[0] = (T)cint; th[1] = xl; th[2] = yl; th[3] = (T)cbg;
                        } else {
                            th[0] = (T)cint; th[1] = w0; th[2] = w0; th[3] = xl; th[4] = yl;
                            th[5] = T(0); th[6] = (T)cbg;
                        }
                    }
                    phase = 1;
                }
                rbase = a.roi_slot ? (long long)a.roi_slot[my]
                                   : (long long)fr * a.frame_px + xo + (long long)yo * a.n_rows;
            }
            // warp-cooperative ROI staging: global uint16 -> shared float. The
            // loads of up to four fits are issued before the first is stored:
            // a trip refills about four of a warp's 32 fits, and one latency
            // per fit and round was a quarter of the first level's time
            // (520 000 dense fits: ellipsoidal 11.04 -> 10.47 ms, symmetric
            // 6.88 -> 6.36 ms; fetching further queue entries into L2 ahead of
            // time gave nothing more).
            unsigned got = __ballot_sync(kFull, my >= 0 && leader);
            if constexpr (S > 0) {
                constexpr int N = (S * S + 31) / 32, G = 4;
                while (got) {
                    uint16_t px[G][N];
                    int src[G];   // past the last fit, the last one again
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        src[g] = got ? __ffs(got) - 1 : src[g > 0 ? g - 1 : 0];
                        got &= got - 1;
                        const uint16_t *fb = a.frames + __shfl_sync(kFull, rbase, src[g]);
                        const int pitch = a.roi_slot ? S : a.n_rows;   // a packed ROI's rows are 2r + 1 pixels apart
#pragma unroll
                        for (int n = 0; n < N; ++n) {
                            const int k = min(lane + 32 * n, S * S - 1), j = k / S, i = k - j * S;
                            px[g][n] = __ldg(fb + i + (size_t)j * pitch);
                        }
                    }
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        float *dst = smem + ((tid - lane + src[g]) / TPF) * stride;
#pragma unroll
                        for (int n = 0; n < N; ++n)
                            if (lane + 32 * n < S * S) dst[lane + 32 * n] = (float)px[g][n];
                    }
                }
            } else {
                while (got) {
                    const int src = __ffs(got) - 1;
                    got &= got - 1;
                    const long long sbase = __shfl_sync(kFull, rbase, src);
                    const int side = __shfl_sync(kFull, s, src);
                    const int pitch = a.roi_slot ? side : a.n_rows;
                    const uint16_t *fb = a.frames + sbase;
                    float *dst = smem + ((tid - lane + src) / TPF) * stride;
                    for (int k = lane; k < side * side; k += 32) {
                        const int j = k / side, i = k - j * side;
                        dst[k] = (float)__ldg(fb + i + (size_t)j * pitch);
                    }
                }
            }
            __syncwarp();
        }
        // few fits left and none to refill with: hand them over
        drain = a.drain > 0 && __ballot_sync(kFull, exhausted && has_room) != 0 &&
                __popc(__ballot_sync(kFull, phase != 0 && leader)) <= a.drain;
        // fits whose last step was accepted start their next outer iteration
        // here (one inlined copy of it)
        if (phase == 3) start_iteration();
        if (__ballot_sync(kFull, phase != 0) == 0) break;
        lap(c_refill);

        // ---- choose this fit's evaluation point (identical in every sub-lane) ----
        bool do_pass = false;
        if (phase == 1) {
#pragma unroll
            for (int k = 0; k < P; ++k) te[k] = th[k];
            do_pass = true;
        } else if (phase == 2) {
            ++trial;
            T invD[P], z[P];
            StateArr<T, NT, kSmemState> Ms(sstate ? sstate + NT + 4 * P : nullptr);
#pragma unroll
            for (int k = 0; k < P; ++k) invD[k] = frcp(D[k]);
#pragma unroll
            for (int i = 0; i < P; ++i)
#pragma unroll
                for (int j = i; j < P; ++j) Ms[pku(P, i, j)] = A[pku(P, i, j)] * invD[i] * invD[j];
            unsigned nl = 0, ne = 0;
            bool sing = false;
            T npiv;
            T vr[P];
#pragma unroll
            for (int k = 0; k < P; ++k) vr[k] = v[k];
            lmpar_scaled<P, T, ESC, kSmemState>(Ms, vr, invD, sym_fuse<ESC>(s, TPF), delta, par, z, a.pivot_thr, nl, ne, sing,
                                    npiv, margin_fit, sstate ? sstate + 2 * NT + 4 * P : nullptr);
            if (leader) {
                st[ST_LAMBDA] += nl;
                st[ST_ESC] += ne;
            }
            esc_fit += ne;
            minpiv_fit = npiv < minpiv_fit ? npiv : minpiv_fit;
            if (sing) {
                finish(T_SINGULAR);
            } else {
                T pn2 = T(0), z0;
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    dx[k] = -z[k] * invD[k];
                    te[k] = th[k] + dx[k];
                    add_square<T>(z[k], k, z0, pn2);
                }
                pnorm = fsqrt(pn2);
                if (it_state == 1 && pnorm < delta) delta = pnorm;
                T qf = T(0);
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    T row = T(0);
#pragma unroll
                    for (int j = 0; j < P; ++j) row = fma(Ms[i <= j ? pku(P, i, j) : pku(P, j, i)], z[j], row);
                    qf = fma(z[i], row, qf);
                }
                jdx2 = qf;
                const bool bad = (METHOD == 0 && te[1] == T(0)) || (METHOD == 7 && (te[1] == T(0) || te[2] == T(0)));
                if (bad) finish(T_EBADFUNC);
                else do_pass = true;
            }
        }

        // ---- the pass: model, Jacobian and normal equations at te ----
        // All lanes reconverge here so that the pixel loop runs once for the
        // whole warp rather than once per divergent group.
        __syncwarp();
        lap(c_step);
        const unsigned pmask = __ballot_sync(kFull, do_pass);
        T acc[NT - 1], vv[P], chi2, dchi, dqmax;
        if (do_pass) {
            T dt[P], tev[P];
#pragma unroll
            for (int k = 0; k < P; ++k) {
                dt[k] = phase == 2 ? dx[k] : T(0);
                tev[k] = te[k];
            }
            Pass<METHOD, S, TPF, T>::run(myroi, s, q, row_fused<METHOD, T, ESC>(s, TPF), w0, tev, dt, acc, vv, chi2, dchi, dqmax);
            if constexpr (TPF > 1 && sizeof(T) == 4) {
                if (a.compensated) {
#pragma unroll
                    for (int k = 0; k < NT - 1; ++k) acc[k] = group_sum_wide(acc[k], TPF, pmask);
#pragma unroll
                    for (int k = 0; k < P; ++k) vv[k] = group_sum_wide(vv[k], TPF, pmask);
                    chi2 = group_sum_wide(chi2, TPF, pmask);
                } else {
#pragma unroll
                    for (int k = 0; k < NT - 1; ++k) acc[k] = group_sum(acc[k], TPF, pmask);
#pragma unroll
                    for (int k = 0; k < P; ++k) vv[k] = group_sum(vv[k], TPF, pmask);
                    chi2 = group_sum(chi2, TPF, pmask);
                }
                dchi = group_sum(dchi, TPF, pmask);
                dqmax = group_max(dqmax, TPF, pmask);
            } else if constexpr (TPF > 1) {
#pragma unroll
                for (int k = 0; k < NT - 1; ++k) acc[k] = group_sum(acc[k], TPF, pmask);
#pragma unroll
                for (int k = 0; k < P; ++k) vv[k] = group_sum(vv[k], TPF, pmask);
                chi2 = group_sum(chi2, TPF, pmask);
                dchi = group_sum(dchi, TPF, pmask);
                dqmax = group_max(dqmax, TPF, pmask);
            }
            if (leader) {
                if (phase == 1) {
                    st[ST_J] += 1;
                    st[ST_PIXJ] += npx;
                } else {
                    st[ST_F] += 1;
                    st[ST_PIXF] += npx;
                }
            }
        }

        __syncwarp();
        lap(c_pass);
        // ---- decide ----
        if (do_pass) {
            const T fn1 = fsqrt(chi2) * inv_abs_s;
            if (phase == 1) {
                // gsl_multifit_fdfsolver_set for lmsder
#pragma unroll
                for (int k = 0; k < NT - 1; ++k) A[k] = acc[k] * inv_s2;
                A[NT - 1] = (T)npx * inv_s2;
#pragma unroll
                for (int k = 0; k < P; ++k) v[k] = vv[k] * inv_s2;
                fnorm = fn1;
                T xn2 = T(0), t0;
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    const T cn = sqrt(A[pku(P, k, k)]);
                    D[k] = cn == T(0) ? T(1) : cn;
                    const T t = D[k] * theta_abs(k, th);
                    add_square<T>(t, k, t0, xn2);
                    dx[k] = T(0);
                }
                xnorm = sqrt(xn2);
                delta = xnorm > T(0) ? T(100) * xnorm : T(100);
                par = T(0);
                it_state = 1;
                iterations = 0;
                phase = 3;  // next outer iteration, started after the refill
            } else {
                T actred = T(-1);
                if (T(0.1) * fn1 < fnorm) {
                    if (dqmax < T(0.25)) {
                        // accurate |f|^2 change from the per-pixel model differences
                        actred = fdiv(-(dchi * inv_s2), fnorm * fnorm);
                    } else {
                        const T u = fdiv(fn1, fnorm);
                        actred = T(1) - u * u;
                    }
                }
                const T if2 = frcp(fnorm * fnorm);
                const T t2s = mul_rn(mul_rn(mul_rn(par, pnorm), pnorm), if2);
                const T prered = fma(jdx2, if2, T(2) * t2s);
                const T dirder = -fma(jdx2, if2, t2s);
                const T ratio = prered > T(0) ? fdiv(actred, prered) : T(0);
                margin_fit = fmin(margin_fit, fmin(fabs(ratio - T(0.25)), fmin(fabs(ratio - T(0.75)),
                                                                              fabs(ratio - T(1e-4)))));
                if (ratio > T(0.25)) {
                    if (par == T(0) || ratio >= T(0.75)) {
                        delta = pnorm / T(0.5);
                        par *= T(0.5);
                    }
                } else {
                    T temp = (actred >= T(0)) ? T(0.5) : fdiv(T(0.5) * dirder, dirder + T(0.5) * actred);
                    if (T(0.1) * fn1 >= fnorm || temp < T(0.1)) temp = T(0.1);
                    const T lim = pnorm / T(0.1);
                    delta = temp * (delta < lim ? delta : lim);
                    par /= temp;
                }
                if (ratio >= T(1e-4)) {
                    T xn2 = T(0), t0;
#pragma unroll
                    for (int k = 0; k < P; ++k) {
                        th[k] = te[k];
                        const T t = D[k] * theta_abs(k, th);
                        add_square<T>(t, k, t0, xn2);
                        v[k] = vv[k] * inv_s2;
                    }
#pragma unroll
                    for (int k = 0; k < NT - 1; ++k) A[k] = acc[k] * inv_s2;
                    A[NT - 1] = (T)npx * inv_s2;
                    xnorm = sqrt(xn2);
                    fnorm = fn1;
                    ++it_state;
                    if (leader) {
                        st[ST_J] += 1;  // the accepted trial's Jacobian
                        st[ST_PIXJ] += npx;
                    }
#pragma unroll
                    for (int k = 0; k < P; ++k) {
                        const T cn = sqrt(A[pku(P, k, k)]);
                        const T cnn = cn == T(0) ? T(1) : cn;
                        if (cnn > D[k]) D[k] = cnn;
                    }
                    if (test_delta()) finish(T_CONVERGED);
                    else if (iterations >= a.max_iter) finish(T_MAX_ITER);
                    else phase = 3;
                } else {
                    T gmax = T(0);
#pragma unroll
                    for (int k = 0; k < P; ++k) {
                        const T gk = fabs(fdiv(v[k], D[k]));
                        if (gk > gmax) gmax = gk;
                    }
                    const T gnorm = fdiv(gmax, fnorm);
                    if (fabs(actred) <= (T)kDblEps && prered <= (T)kDblEps && T(0.5) * ratio <= T(1))
                        finish(T_ETOLF);
                    else if (delta <= (T)kDblEps * xnorm)
                        finish(T_ETOLX);
                    else if (gnorm <= (T)kDblEps)
                        finish(T_ETOLG);
                    else if (trial >= 10)
                        finish(T_ENOPROG);
                }
            }
        }
        __syncwarp();
        lap(c_decide);
    }
    flush();
    if (lane == 0) {
        st[ST_CYC_REFILL] += (unsigned)(c_refill >> 10);
        st[ST_CYC_STEP] += (unsigned)(c_step >> 10);
        st[ST_CYC_PASS] += (unsigned)(c_pass >> 10);
        st[ST_CYC_DECIDE] += (unsigned)(c_decide >> 10);
    }
}

// blocks of 128 threads resident per SM the register budget is sized for
// (FP64: one, i.e. the full 255 registers)
__host__ __device__ constexpr int k1_min_blocks(int method, int bytes) { return bytes == 8 ? 1 : (method == 7 ? 2 : 3); }

template <int METHOD, typename T, int S, int TPF, bool ESC>
__global__ void __launch_bounds__(128, k1_min_blocks(METHOD, sizeof(T))) k1_lm_fit(K1Args a, int r, int smem_bytes)
{
    extern __shared__ float smem[];
    unsigned st[ST_N];
#pragma unroll
    for (int k = 0; k < ST_N; ++k) st[k] = 0;
    if (r > 0 ? a.meta[m_count(r)] > 0 : *a.count > a.least)
        run_class<METHOD, T, S, TPF, ESC>(a, r, smem_bytes, smem, st);
    // warp-reduce the counters, one atomic per warp and counter
#pragma unroll
    for (int k = 0; k < ST_N; ++k) {
        unsigned long long vsum = st[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) vsum += __shfl_xor_sync(kFull, vsum, o);
        if ((threadIdx.x & 31) == 0 && vsum) atomicAdd(&a.stats[k], vsum);
    }
}

struct K2Args {
    const Cand *cands;
    int n;
    int method;
    double w0;
    int r_default;
    const float *state32;   // FP32 solver state (NULL when the whole call ran in FP64)
    const double *state64;  // FP64 solver state of re-run fits (or of every fit)
    const int *rerun;       // >= 0 where the fit was re-run in FP64 (NULL: none)
    int state_stride;
    int ncol_total;
    double *out;
    uint8_t *flags;
    float *params_out;
    float *diag;
};

// Symmetric 2x2 eigen-decomposition with ascending eigenvalues (the
// reference uses Eigen::SelfAdjointEigenSolver, Localization.cpp:529-547);
// theta = atan(v00 / v10) of the eigenvector of the smaller eigenvalue.
__device__ bool eig2_theta(double a, double b, double c, double &l0, double &l1, double &theta)
{
    if (!isfinite(a) || !isfinite(b) || !isfinite(c)) return false;
    const double ht = 0.5 * (a + c), hd = 0.5 * (a - c);
    const double rad = hypot(hd, b);
    l0 = ht - rad;
    l1 = ht + rad;
    double v0, v1;
    if (b == 0.0) {
        if (a <= c) { v0 = 1.0; v1 = 0.0; } else { v0 = 0.0; v1 = 1.0; }
    } else {
        const double ua0 = b, ua1 = l0 - a, ub0 = l0 - c, ub1 = b;
        if (ua0 * ua0 + ua1 * ua1 >= ub0 * ub0 + ub1 * ub1) { v0 = ua0; v1 = ua1; }
        else { v0 = ub0; v1 = ub1; }
    }
    theta = (v1 == 0.0) ? 0.0 : atan(v0 / v1);
    return true;
}

// diag((J^T J)^-1) by Cholesky in FP64 (gsl_multifit_covar(J, 0.0, .) at
// Localization.cpp:185, 355, 556 forms the same inverse through QR).
template <int P>
__device__ bool inverse_diagonal(const double (&A)[tri(P)], double (&cd)[P])
{
    double L[tri(P)], inv[P];
#pragma unroll
    for (int j = 0; j < P; ++j) {
        double d = A[pku(P, j, j)];
#pragma unroll
        for (int k = 0; k < j; ++k) d -= L[pkl(j, k)] * L[pkl(j, k)];
        if (!(d > 0.0)) return false;
        const double l = sqrt(d);
        L[pkl(j, j)] = l;
        inv[j] = 1.0 / l;
#pragma unroll
        for (int i = j + 1; i < P; ++i) {
            double s = A[pku(P, j, i)];
#pragma unroll
            for (int k = 0; k < j; ++k) s -= L[pkl(i, k)] * L[pkl(j, k)];
            L[pkl(i, j)] = s * inv[j];
        }
    }
    // columns of L^-1; diag(A^-1)_j = sum_k (L^-1)_{kj}^2
#pragma unroll
    for (int j = 0; j < P; ++j) cd[j] = 0.0;
#pragma unroll
    for (int col = 0; col < P; ++col) {
        double y[P];
#pragma unroll
        for (int i = 0; i < P; ++i) {
            if (i < col) { y[i] = 0.0; continue; }
            double s = (i == col) ? 1.0 : 0.0;
#pragma unroll
            for (int k = 0; k < i; ++k) s -= L[pkl(i, k)] * y[k];
            y[i] = s * inv[i];
        }
#pragma unroll
        for (int i = 0; i < P; ++i) cd[col] += y[i] * y[i];
    }
    return true;
}

template <int METHOD>
__global__ void k2_finalize(K2Args a)
{
    constexpr int P = Traits<METHOD == 5 ? 7 : METHOD>::P;
    constexpr int NT = tri(P);
    using SL = StateLayout<P>;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    if (a.flags[i] != F_PENDING) return;
    const Cand cd = a.cands[i];
    const bool r64 = a.state32 == nullptr || (a.rerun && a.rerun[i] >= 0);
    const size_t base = (size_t)i * a.state_stride;
    auto sv = [&](int k) -> double { return r64 ? a.state64[base + k] : (double)a.state32[base + k]; };
    const int iterations = (int)sv(SL::ITERS);
    const int status = (int)sv(SL::STATUS);
    const int xo = (int)sv(SL::XOFF), yo = (int)sv(SL::YOFF);
    const int r = cd.half_width > 0 ? cd.half_width : a.r_default;
    const int xm = xo + 2 * r, ym = yo + 2 * r;
    const double w0 = a.w0;
    const int ncol = ref_cols(METHOD);
    double *row = a.out + (size_t)i * a.ncol_total;
    row[0] = (double)cd.frame;
    for (int k = 1; k < ncol; ++k) row[k] = CUDART_NAN;
    row[ncol] = (double)iterations;
    row[ncol + 1] = (double)status;

    double x[P];
#pragma unroll
    for (int k = 0; k < P; ++k) x[k] = sv(k);
    constexpr int IX = METHOD == 0 ? 2 : METHOD == 1 ? 1 : 3;
    x[IX] += xo;
    x[IX + 1] += yo;
    if constexpr (METHOD == 0) x[1] = fabs(x[1]);
    if constexpr (METHOD == 5 || METHOD == 7) {
        x[1] = fabs(x[1]);
        x[2] = fabs(x[2]);
    }
    if (a.params_out) {
#pragma unroll
        for (int k = 0; k < P; ++k) a.params_out[(size_t)i * P + k] = (float)x[k];
    }
    if (a.diag) {
        float *dg = a.diag + (size_t)i * 8;
        const size_t b32 = (size_t)i * a.state_stride;
        dg[0] = (float)sv(SL::MINPIV);
        dg[1] = (float)sv(SL::LASTR);
        dg[2] = (float)sv(SL::NESC);
        dg[3] = (float)sv(SL::MARGIN);
        dg[4] = r64 && a.state32 != nullptr ? 1.0f : 0.0f;
        dg[5] = a.state32 ? a.state32[b32 + SL::ITERS] : (float)iterations;
        dg[6] = a.state32 ? a.state32[b32 + SL::STATUS] : (float)status;
        dg[7] = 0.0f;
    }
    uint8_t flag = F_KEPT;
    if (x[0] <= 0) flag = F_AMPLITUDE;
    else if (x[IX] < xo || x[IX] > xm || x[IX + 1] < yo || x[IX + 1] > ym) flag = F_WINDOW;
    if (flag != F_KEPT) {
        a.flags[i] = flag;
        return;
    }
    double A[NT];
#pragma unroll
    for (int k = 0; k < NT; ++k) A[k] = sv(P + k);
    const double chi = sv(SL::FNORM);
    double cv[P];

    if constexpr (METHOD == 0) {
        if (x[1] < 0.4 * w0 || x[1] > w0 * 1.5) flag = F_WIDTH;
        else {
            const bool ok = inverse_diagonal<P>(A, cv);
            if (!ok)
                for (int k = 0; k < P; ++k) cv[k] = CUDART_NAN;
            const double dof = (double)((2 * r - 1) * (2 * r - 1) - 5);  // Localization.cpp:187 as written
            const double c = fmax(1.0, chi / sqrt(dof));
            const double pi = 3.1415926535897932384626433;
            const double width = x[1];
            const double widthDev = c * sqrt(cv[1]);
            const double integral = 2 * pi * width * width * x[0];
            const double relA = c * sqrt(cv[0]) / x[0];
            const double relW = widthDev / width;
            row[1] = integral;
            row[2] = width;
            row[3] = x[2];
            row[4] = x[3];
            row[5] = x[4];
            row[6] = 2 * pi * integral * sqrt(relA * relA + 2 * relW * relW);
            row[7] = widthDev;
            row[8] = c * sqrt(cv[2]);
            row[9] = c * sqrt(cv[3]);
            row[10] = c * sqrt(cv[4]);
            row[11] = 1.0;
        }
    } else if constexpr (METHOD == 1) {
        if (fabs(x[1] - cd.x) > 2.0 * w0 || fabs(x[2] - cd.y) > 2.0 * w0) flag = F_DRIFT;
        else {
            const bool ok = inverse_diagonal<P>(A, cv);
            if (!ok)
                for (int k = 0; k < P; ++k) cv[k] = CUDART_NAN;
            const double dof = (double)((2 * r - 1) * (2 * r - 1) - 4);
            const double c = fmax(1.0, chi / sqrt(dof));
            const double pi = 3.1415926535897932384626433;
            const double integral = 2 * pi * w0 * w0 * x[0];
            const double relA = c * sqrt(cv[0]) / x[0];
            row[1] = integral;
            row[2] = x[1];
            row[3] = x[2];
            row[4] = x[3];
            row[5] = 2 * pi * integral * w0 * w0 * sqrt(relA * relA);
            row[6] = c * sqrt(cv[1]);
            row[7] = c * sqrt(cv[2]);
            row[8] = c * sqrt(cv[3]);
            row[9] = 1.0;
        }
    } else {
        const double sx = x[1], sy = x[2], rho = x[5];
        double l0, l1, theta;
        if (!eig2_theta(sx * sx, rho * sx * sy, sy * sy, l0, l1, theta)) flag = F_EIGEN;
        else {
            const double s1 = sqrt(l0), s2 = sqrt(l1);
            if (!(((s1 >= 0.4 * w0) && (s1 <= 1.5 * w0)) || ((s2 >= 0.4 * w0) && (s2 <= 1.5 * w0)))) flag = F_NO_AXIS;
            else {
                const bool ok = inverse_diagonal<P>(A, cv);
                if (!ok)
                    for (int k = 0; k < P; ++k) cv[k] = CUDART_NAN;
                const double dof = (double)((2 * r - 1) * (2 * r - 1) - 7);
                const double c = fmax(1.0, chi / sqrt(dof));
                const double pi = 3.1415926535897932384626433;
                const double corrDev = c * sqrt(cv[5]);
                const double sxDev = c * sqrt(cv[1]), syDev = c * sqrt(cv[2]);
                double sn, cs;
                sincos(theta, &sn, &cs);
                const double s1Dev = sxDev * cs + syDev * sn;
                const double s2Dev = sxDev * sn + syDev * cs;
                const double ampDev = c * sqrt(cv[0]);
                const double omr = 1 - rho * rho;
                const double integral = 2.0 * pi * x[0] * sqrt(omr) * s1 * s2;
                row[1] = integral;
                row[2] = s1;
                row[3] = s2;
                row[4] = x[3];
                row[5] = x[4];
                row[6] = theta;
                row[7] = x[6];
                row[8] = integral * sqrt(ampDev * ampDev / x[0] / x[0] + rho * rho * corrDev * corrDev / omr / omr +
                                         s1Dev * s1Dev / s1 / s1 + s2Dev * s2Dev / s2 / s2);
                row[9] = s1Dev;
                row[10] = s2Dev;
                row[11] = c * sqrt(cv[3]);
                row[12] = c * sqrt(cv[4]);
                row[13] = 0.0;
                row[14] = c * sqrt(cv[6]);
                row[15] = 1.0;
                if constexpr (METHOD == 5) {
                    if ((0.75 * s1 > s2) || (1.25 * s1 < s2)) flag = F_SYM_RATIO;
                    else if (((s1 < w0 * 0.7) || (s1 > w0 * 1.3)) && ((s2 < w0 * 0.7) || (s2 > w0 * 1.3)))
                        flag = F_SYM_WIDTH;
                }
            }
        }
    }
    if (flag != F_KEPT) {
        for (int k = 1; k < ncol; ++k) row[k] = CUDART_NAN;
    }
    a.flags[i] = flag;
}

int solver_method(int method) { return method == 5 ? 7 : method; }

// Blocks of a persistent kernel: every SM filled to its occupancy. The limit
// on its shared memory is set to the device's, whatever this launch needs: host
// threads with other ROI sizes launch the same kernels.
template <typename F>
cudaError_t persistent_grid(F *kern, int tpb, int smem, int bps_req, int *grid)
{
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 0, bps = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, tpb, smem);
    if (e != cudaSuccess) return e;
    if (bps < 1) return cudaErrorInvalidConfiguration;
    if (bps_req > 0 && bps_req < bps) bps = bps_req;
    *grid = nsm * bps;
    return cudaSuccess;
}

// r > 0: the class's queue; r = 0: a list, ROIs up to r_cap.
template <int METHOD, typename T, int S, int TPF, bool ESC = false>
cudaError_t launch_k1_s(const K1Args &ka, int r, int r_cap, int tpb, int bps_req, cudaStream_t stream)
{
    auto kern = k1_lm_fit<METHOD, T, S, TPF, ESC>;
    const int slot = slot_bytes<T>(Traits<METHOD>::P, r > 0 ? r : r_cap, TPF);
    int smem = (tpb / TPF) * slot;
    if (r > 0) {
        // fewer threads per block when the block's shared memory would exceed 227 KB
        while (tpb > 32 && smem > 227 * 1024) {
            tpb -= 32;
            smem = (tpb / TPF) * slot;
        }
        if (smem > 227 * 1024) return cudaErrorInvalidValue;
    } else {
        // two blocks per SM; larger ROIs leave groups of a block without room
        const int most = 113 * 1024;
        if (slot > most) return cudaErrorInvalidValue;
        if (smem > most) smem = most;
    }
    int grid = 0;
    const cudaError_t e = persistent_grid(kern, tpb, smem, bps_req, &grid);
    if (e != cudaSuccess) return e;
    kern<<<grid, tpb, smem, stream>>>(ka, r, smem);
    return cudaGetLastError();
}

template <int METHOD, int TPF>
cudaError_t launch_k1_tpf(const K1Args &ka, int r, int tpb, int bps_req, cudaStream_t stream)
{
    // FP64 pivot escalation: one runtime-side instantiation per method
    // and threads per fit
    if (ka.pivot_thr > 0.0f) return launch_k1_s<METHOD, float, 0, TPF, true>(ka, r, r, tpb, bps_req, stream);
    switch (2 * r + 1) {
    case 5: return launch_k1_s<METHOD, float, 5, TPF>(ka, r, r, tpb, bps_req, stream);
    case 7: return launch_k1_s<METHOD, float, 7, TPF>(ka, r, r, tpb, bps_req, stream);
    case 9: return launch_k1_s<METHOD, float, 9, TPF>(ka, r, r, tpb, bps_req, stream);
    case 11: return launch_k1_s<METHOD, float, 11, TPF>(ka, r, r, tpb, bps_req, stream);
    case 13: return launch_k1_s<METHOD, float, 13, TPF>(ka, r, r, tpb, bps_req, stream);
    case 15: return launch_k1_s<METHOD, float, 15, TPF>(ka, r, r, tpb, bps_req, stream);
    case 17: return launch_k1_s<METHOD, float, 17, TPF>(ka, r, r, tpb, bps_req, stream);
    default: return launch_k1_s<METHOD, float, 0, TPF>(ka, r, r, tpb, bps_req, stream);
    }
}

// One persistent first-level launch for the queue of half-width r with tpf
// threads per fit (1, 4, 8 or 16).
template <int METHOD>
cudaError_t launch_first(const K1Args &ka, int r, int tpb, int bps_req, int tpf, cudaStream_t stream)
{
    switch (tpf) {
    case 4: return launch_k1_tpf<METHOD, 4>(ka, r, tpb, bps_req, stream);
    case 8: return launch_k1_tpf<METHOD, 8>(ka, r, tpb, bps_req, stream);
    // a half warp per fit (runtime ROI side only)
    case 16: return launch_k1_s<METHOD, float, 0, 16>(ka, r, r, tpb, bps_req, stream);
    default: return launch_k1_tpf<METHOD, 1>(ka, r, tpb, bps_req, stream);
    }
}

// One launch over a list with tpf threads per fit (FP32: 1, 4 or 8; FP64: 1,
// 2, 4 or 8).
template <int METHOD, typename T>
cudaError_t launch_list(const K1Args &ka, int r_cap, int tpb, int bps_req, int tpf, cudaStream_t stream)
{
    if constexpr (sizeof(T) == 4) {
        if (ka.pivot_thr > 0.0f)
            return tpf == 4 ? launch_k1_s<METHOD, T, 0, 4, true>(ka, 0, r_cap, tpb, bps_req, stream)
                 : tpf == 8 ? launch_k1_s<METHOD, T, 0, 8, true>(ka, 0, r_cap, tpb, bps_req, stream)
                            : launch_k1_s<METHOD, T, 0, 1, true>(ka, 0, r_cap, tpb, bps_req, stream);
    } else {
        if (tpf == 2) return launch_k1_s<METHOD, T, 0, 2>(ka, 0, r_cap, tpb, bps_req, stream);
    }
    return tpf == 4 ? launch_k1_s<METHOD, T, 0, 4>(ka, 0, r_cap, tpb, bps_req, stream)
         : tpf == 8 ? launch_k1_s<METHOD, T, 0, 8>(ka, 0, r_cap, tpb, bps_req, stream)
                    : launch_k1_s<METHOD, T, 0, 1>(ka, 0, r_cap, tpb, bps_req, stream);
}
template <typename T>
cudaError_t launch_list_m(int m, const K1Args &ka, int r_cap, int tpb, int bps_req, int tpf, cudaStream_t stream)
{
    return m == 0 ? launch_list<0, T>(ka, r_cap, tpb, bps_req, tpf, stream)
         : m == 1 ? launch_list<1, T>(ka, r_cap, tpb, bps_req, tpf, stream)
                  : launch_list<7, T>(ka, r_cap, tpb, bps_req, tpf, stream);
}

// Calls of at most this many candidates run on the team solver alone: that is
// two fits for every warp of a full device (148 SMs x 12 warps). With one
// thread per fit such a call leaves most of the device idle for as long as its
// longest fit takes (a call of 160 symmetric fits, FP64 re-run included, both
// timed in turn: 437 us with a thread per fit, 235 us by teams). Like the lines
// below it is written for the 148 SMs of a B200.
constexpr int kTeamOnlyFits = 3552;
// Lists of at most this many fits go to the teams at once (FP32, FP64). FP64:
// 3552 is the best of 1 to 3552 at 20 000 to 520 000 fits a call. For FP32 the
// line is not sensitive: 300 to 3552 measure the same, and it is the same one.
constexpr int kTeamFits32 = 3552, kTeamFits64 = 3552;
// A warp that has run dry hands its last fits over at this many groups or
// fewer: FP32 with one thread per fit (the ellipsoidal models, whose fits
// differ most in length, keep them: measured 11.9 against 12.6 ms at 520 000
// fits, while the symmetric ones lose 7.5 -> 7.8 ms without), the re-run with
// two threads per fit, and FP64-precision calls.
constexpr int kDrain1 = 4, kDrain2 = 3, kDrain64 = 8;
// Calls whose ROIs are all 3 x 3: a thread is through with nine pixels sooner
// than a team with its sums and barriers, so the groups keep their fits and
// only lists of a length that leaves the device idle go to the teams. 20 000
// fits, with the lines above -> these: FP64 ellipsoidal 6.8 -> 4.1 ms,
// symmetric 3.0 -> 2.5 ms; FP32 ellipsoidal 4.7 -> 4.1 ms, symmetric 4.3 -> 3.4
// ms. From 5 x 5 ROIs on the lines above win (FP64 ellipsoidal 1.9 against
// 3.1 ms).
constexpr int kTeamFitsTiny = 300;
// Lists of up to this many fits are solved by teams of four warps, longer ones
// by teams of one. Four warps take 0.6 of the time per fit and the instructions
// of nearly four, so they win while the longest fit sets the time: two (FP32)
// and three (FP64) fits per resident block. Measured, one warp -> four: the
// solver's part of a frame of 80 ellipsoidal fits 298 -> 248 us, the FP64 re-run
// of 262 of 520 000 symmetric fits 6.30 -> 5.70 ms for the call; with 2 400
// ellipsoidal re-runs 10.6 -> 11.8 ms, so they keep one warp.
constexpr int kBlockFits32 = 1184, kBlockFits64 = 1332;

template <int METHOD, typename T, bool ESC>
cudaError_t launch_team_m(const TeamArgs &ta, int r_cap, int n_most, int bps_req, cudaStream_t stream)
{
    auto kern = k_team<METHOD, T, ESC>;
    constexpr int tpb = 128, line = sizeof(T) == 8 ? kBlockFits64 : kBlockFits32;
    const int one = team_smem<METHOD, T, 4>(r_cap), four = 4 * team_smem<METHOD, T, 1>(r_cap);
    const int smem = one > four ? one : four;
    int grid = 0;
    const cudaError_t e = persistent_grid(kern, tpb, smem, bps_req, &grid);
    if (e != cudaSuccess) return e;
    kern<<<n_most < grid ? n_most : grid, tpb, smem, stream>>>(ta, r_cap, line);
    return cudaGetLastError();
}

// One team launch (method m of the solver) over at most n_most fits.
template <typename T>
cudaError_t launch_team(int m, const TeamArgs &ta, int r_cap, int n_most, int bps_req, cudaStream_t stream)
{
    if constexpr (sizeof(T) == 4) {
        if (ta.k.pivot_thr > 0.0f)
            return m == 0 ? launch_team_m<0, T, true>(ta, r_cap, n_most, bps_req, stream)
                 : m == 1 ? launch_team_m<1, T, true>(ta, r_cap, n_most, bps_req, stream)
                          : launch_team_m<7, T, true>(ta, r_cap, n_most, bps_req, stream);
    }
    return m == 0 ? launch_team_m<0, T, false>(ta, r_cap, n_most, bps_req, stream)
         : m == 1 ? launch_team_m<1, T, false>(ta, r_cap, n_most, bps_req, stream)
                  : launch_team_m<7, T, false>(ta, r_cap, n_most, bps_req, stream);
}

int cont_stride_of(int m) { return m == 0 ? ContLayout<5>::STRIDE : m == 1 ? ContLayout<4>::STRIDE : ContLayout<7>::STRIDE; }

}  // namespace

int state_stride(int method)
{
    const int m = solver_method(method);
    return m == 0 ? StateLayout<5>::STRIDE : m == 1 ? StateLayout<4>::STRIDE : StateLayout<7>::STRIDE;
}

// Scratch layout (256-byte aligned pieces): cls, order, meta, stats, cont,
// cont_state, state (FP32 state, or FP64 state when the call runs in FP64),
// then for the FP64 re-run of flagged fits: cls2, order2, meta2, state64.
namespace {
size_t al256(size_t b) { return (b + 255) / 256 * 256; }
}

static_assert(kStatWords >= 2 * ST_N + 1, "statistics words");

size_t scratch_bytes(int method, int n, int precision, int rerun, int warm)
{
    const size_t el = precision == 1 ? sizeof(double) : sizeof(float);
    const int m = solver_method(method);
    size_t b = al256(sizeof(int) * (size_t)n) * 2 + al256(sizeof(int) * kMetaInts) +
               al256(sizeof(unsigned long long) * kStatWords) + al256(sizeof(int) * (size_t)n) +
               al256(sizeof(float) * (size_t)n * cont_stride_of(m)) + al256(el * (size_t)n * state_stride(method));
    if (precision != 1 && rerun)
        b += al256(sizeof(int) * (size_t)n) * 3 + al256(sizeof(int) * kMetaInts) * 2 +
             al256(sizeof(double) * (size_t)n * state_stride(method));
    if (warm) b += al256(sizeof(float) * (size_t)n * 8);
    return b;
}

void carve_scratch(void *base, int method, int n, int precision, int rerun, Scratch *s, int warm)
{
    const size_t el = precision == 1 ? sizeof(double) : sizeof(float);
    char *p = (char *)base;
    s->cls = (int *)p;
    p += al256(sizeof(int) * (size_t)n);
    s->order = (int *)p;
    p += al256(sizeof(int) * (size_t)n);
    s->meta = (int *)p;
    p += al256(sizeof(int) * kMetaInts);
    s->stats = (unsigned long long *)p;
    p += al256(sizeof(unsigned long long) * kStatWords);
    s->cont = (int *)p;
    p += al256(sizeof(int) * (size_t)n);
    s->cont_state = (float *)p;
    p += al256(sizeof(float) * (size_t)n * cont_stride_of(solver_method(method)));
    s->state = (void *)p;
    p += al256(el * (size_t)n * state_stride(method));
    if (precision != 1 && rerun) {
        s->cls2 = (int *)p;
        p += al256(sizeof(int) * (size_t)n);
        s->order2 = (int *)p;
        p += al256(sizeof(int) * (size_t)n);
        s->meta2 = (int *)p;
        p += al256(sizeof(int) * kMetaInts);
        s->order3 = (int *)p;
        p += al256(sizeof(int) * (size_t)n);
        s->meta3 = (int *)p;
        p += al256(sizeof(int) * kMetaInts);
        s->state64 = (double *)p;
        p += al256(sizeof(double) * (size_t)n * state_stride(method));
    } else {
        s->cls2 = s->order2 = s->meta2 = s->order3 = s->meta3 = nullptr;
        s->state64 = nullptr;
    }
    s->init = warm ? (float *)p : nullptr;
}

cudaError_t enqueue_fit(const FitParams &p, const Scratch &s, cudaStream_t stream, int *err_detail)
{
    *err_detail = 0;
    const int n = p.n_cands;
    const int ncol_total = ref_cols(p.method) + 2;
    const int r_default = (int)std::ceil(p.w0 * 4.0);
    const bool rerun = p.precision != 1 && p.fp64_rerun && s.state64 != nullptr;
    cudaError_t e;
    e = cudaMemsetAsync(s.meta, 0, sizeof(int) * kMetaInts, stream);
    if (e != cudaSuccess) return e;
    if (rerun && (e = cudaMemsetAsync(s.meta2, 0, sizeof(int) * kMetaInts, stream)) != cudaSuccess) return e;
    const bool long_q = rerun && p.long_rerun_iters > 0;
    if (rerun && (e = cudaMemsetAsync(s.meta3, 0, sizeof(int) * kMetaInts, stream)) != cudaSuccess) return e;
    e = cudaMemsetAsync(s.stats, 0, sizeof(unsigned long long) * kStatWords, stream);
    if (e != cudaSuccess) return e;
    if (p.method == 6) {
        for (int k = 0; k < 4; ++k)
            if (p.ev[k]) cudaEventRecord(p.ev[k], stream);
        return enqueue_mlewg(p, s.stats, stream);
    }
    if (n == 0) {
        for (int k = 0; k < 4; ++k)
            if (p.ev[k]) cudaEventRecord(p.ev[k], stream);
        return cudaSuccess;
    }

    const int r_cap = p.max_half_width > 0 ? (p.max_half_width < kMaxHalfWidth ? p.max_half_width : kMaxHalfWidth)
                                           : kMaxHalfWidth;
    auto mark = [&](int k) {
        if (p.ev[k]) cudaEventRecord(p.ev[k], stream);
    };
    auto bump = [&]() {
        if (p.launches) ++*p.launches;
    };
    mark(0);
    // the pixel array the solver reads: the frames, or (ROI mode) the slots
    const bool roi_mode = p.roi_slot != nullptr;
    // the start proposal cuts its windows from whole frames
    if (roi_mode && p.warm) return cudaErrorInvalidValue;
    const uint16_t *px = roi_mode ? p.roi_stack : p.frames;
    const long long px_frame = roi_mode ? 0 : (long long)p.n_rows * p.n_cols;
    const int px_pitch = roi_mode ? 0 : p.n_rows;   // ROI mode: each ROI's own side
    K0Args k0{(const Cand *)p.cands, n, p.n_frames, p.n_rows, p.n_cols, r_default, r_cap, p.method, ncol_total,
              p.out, p.flags, s.cls, s.meta, rerun ? s.cls2 : nullptr, p.roi_slot, p.roi_px};
    const int nb = (n + 255) / 256;
    k0_classify<<<nb, 256, 0, stream>>>(k0);
    k0_classes<<<1, 32, 0, stream>>>(s.meta);
    k0_scatter<<<nb, 256, 0, stream>>>(s.cls, n, s.meta, s.order);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    bump();
    bump();
    bump();

    // Calls of few fits run on the team solver alone: one launch over all ROI
    // classes. Otherwise the first level runs a thread per fit, one launch
    // per class that exists: known bound from the caller, or the histogram
    // read back (one small synchronous copy).
    const bool team_only = n <= kTeamOnlyFits && p.threads_per_fit == 1;
    int counts[K];
    for (int r = 0; r < K; ++r) counts[r] = r <= r_cap ? 1 : 0;
    if (!team_only && p.max_half_width <= 0) {
        e = cudaMemcpyAsync(counts, s.meta + m_count(0), sizeof(int) * K, cudaMemcpyDeviceToHost, stream);
        if (e != cudaSuccess) return e;
        e = cudaStreamSynchronize(stream);
        if (e != cudaSuccess) return e;
    }
    int r_most = 1;
    for (int r = 1; r < K; ++r)
        if (counts[r] > 0) r_most = r;
    mark(1);
    // learned start proposal and start check, before the solver chains fork
    if (p.warm) {
        e = enqueue_proposal(p.prop, p.frames, (long long)p.n_rows * p.n_cols, p.n_rows, p.n_cols, p.cands, s.cls, n,
                             p.method, (float)p.w0, s.init, s.stats + 2 * ST_N, p.prop.err, stream, p.launches);
        if (e != cudaSuccess) return e;
        if (p.ev_prop) cudaEventRecord(p.ev_prop, stream);
    }
    int tpb = p.threads_per_block > 0 ? p.threads_per_block : 128;
    tpb = (tpb + 31) / 32 * 32;
    if (tpb > 128) tpb = 128;
    const double s_abs = std::fabs(p.sigma);
    const int m = solver_method(p.method);
    K1Args k1{};
    k1.frames = px;
    k1.frame_px = px_frame;
    k1.n_rows = px_pitch;
    k1.cands = (const Cand *)p.cands;
    k1.order = s.order;
    k1.meta = s.meta;
    k1.state = s.state;
    k1.state_stride = state_stride(p.method);
    k1.w0 = (float)p.w0;
    k1.inv_s2 = (float)(1.0 / (p.sigma * p.sigma));
    k1.inv_abs_s = (float)(1.0 / s_abs);
    k1.inv_s2_d = 1.0 / (p.sigma * p.sigma);
    k1.inv_abs_s_d = 1.0 / s_abs;
    k1.max_iter = p.max_iter;
    k1.epsabs = (float)p.epsabs;
    k1.epsrel = (float)p.epsrel;
    k1.pivot_thr = p.precision == 1 ? 0.0f : p.pivot_thr;
    k1.init_params = p.warm ? s.init : p.init_params;
    k1.stats = s.stats;
    k1.cls = s.cls;
    k1.list_step = 1;
    k1.cont = s.cont;
    k1.n_cont = s.meta + M_NCONT;
    k1.left = s.cont + n - 1;   // from the other end of the list: a fit is in one of the two
    k1.n_left = s.meta + M_NLEFT;
    k1.left_step = -1;
    k1.cont_state = s.cont_state;
    k1.cont_stride = cont_stride_of(m);
    k1.compensated = p.compensated;
    k1.roi_slot = p.roi_slot;
    // Auxiliary streams: independent launches run side by side so that their
    // ends overlap; the caller's stream joins them.
    int naux = 0;
    while (naux < kMaxAux && p.aux[naux]) ++naux;
    bool used[kMaxAux] = {false};
    auto fork = [&]() -> cudaError_t { return naux > 0 ? cudaEventRecord(p.fork, stream) : cudaSuccess; };
    auto side = [&](int j, cudaStream_t *cs) -> cudaError_t {
        *cs = stream;
        if (naux == 0) return cudaSuccess;
        j %= naux;
        *cs = p.aux[j];
        const cudaError_t x = used[j] ? cudaSuccess : cudaStreamWaitEvent(*cs, p.fork, 0);
        used[j] = true;
        return x;
    };
    auto join = [&]() -> cudaError_t {
        for (int j = 0; j < naux; ++j) {
            if (!used[j]) continue;
            used[j] = false;
            cudaError_t x = cudaEventRecord(p.join[j], p.aux[j]);
            if (x == cudaSuccess) x = cudaStreamWaitEvent(stream, p.join[j], 0);
            if (x != cudaSuccess) return x;
        }
        return cudaSuccess;
    };
#define LOC_TRY(call) do { if ((e = (call)) != cudaSuccess) { if (e == cudaErrorInvalidValue) *err_detail = 1; return e; } bump(); } while (0)
    cudaStream_t cs;
    const bool tiny = r_most == 1;   // 3 x 3 ROIs only
    const int fits32 = tiny ? kTeamFitsTiny : kTeamFits32, fits64 = tiny ? kTeamFitsTiny : kTeamFits64;
    const bool fp64 = p.precision == 1;
    const bool two_level = !fp64 && p.level0_budget > 0 && p.level0_budget < p.max_iter;
    TeamArgs ta{};
    ta.k = k1;
    ta.switch_it = two_level ? p.level0_budget : p.max_iter;
    ta.q0 = 1;
    ta.q1 = p.tail_threads_per_fit;
    ta.next = s.meta + M_LEFTNEXT;
    const TeamList whole{s.order, s.meta + M_TOTAL, 1, 1, 0, n};
    const TeamList left{s.cont + n - 1, s.meta + M_NLEFT, -1, 0, 0, n};
    if (team_only) {
        ta.list[0] = whole;
        LOC_TRY(fp64 ? launch_team<double>(m, ta, r_most, n, p.blocks_per_sm, stream)
                     : launch_team<float>(m, ta, r_most, n, p.blocks_per_sm, stream));
    } else if (fp64) {
        K1Args kf = k1;
        kf.list = s.order;
        kf.count = s.meta + M_TOTAL;
        kf.next = s.meta + M_NEXT;
        kf.drain = tiny ? 0 : kDrain64;
        LOC_TRY(launch_list_m<double>(m, kf, r_most, tpb, p.blocks_per_sm, 1, stream));
        ta.list[0] = left;
        LOC_TRY(launch_team<double>(m, ta, r_most, n, p.blocks_per_sm, stream));
    } else {
        // first level: the fresh candidates, one launch per ROI class
        K1Args kf = k1;
        kf.budget = two_level ? p.level0_budget : 0;
        // (fixed-width fits of 5 x 5 ROIs are over too soon for a hand-over:
        // 12 000 fits 137 -> 123 us without)
        kf.drain = p.threads_per_fit == 1 && m != 7 && r_most > (m == 1 ? 2 : 1) ? kDrain1 : 0;
        kf.mark = rerun ? s.cls2 : nullptr;
        if ((e = fork()) != cudaSuccess) return e;
        int chain = 0;
        for (int r = r_most; r >= 1; --r) {
            if (counts[r] <= 0) continue;
            if ((e = side(chain++, &cs)) != cudaSuccess) return e;
            LOC_TRY(m == 0 ? launch_first<0>(kf, r, tpb, p.blocks_per_sm, p.threads_per_fit, cs)
                  : m == 1 ? launch_first<1>(kf, r, tpb, p.blocks_per_sm, p.threads_per_fit, cs)
                           : launch_first<7>(kf, r, tpb, p.blocks_per_sm, p.threads_per_fit, cs));
        }
        if ((e = join()) != cudaSuccess || (e = fork()) != cudaSuccess) return e;
        // second level: the fits past the budget; beside it the teams finish
        // the fits that the first level's warps were left with (and the
        // second level's, if they are few)
        if (two_level) {
            K1Args kl = k1;
            kl.list = s.cont;
            kl.count = s.meta + M_NCONT;
            kl.next = s.meta + M_CONTNEXT;
            kl.resume = 1;
            kl.least = fits32;
            if ((e = side(1, &cs)) != cudaSuccess) return e;
            LOC_TRY(launch_list_m<float>(m, kl, r_most, tpb, p.blocks_per_sm, p.tail_threads_per_fit, cs));
            ta.list[1] = TeamList{s.cont, s.meta + M_NCONT, 1, 0, 0, fits32};
        }
        ta.list[0] = left;
        if ((e = side(0, &cs)) != cudaSuccess) return e;
        LOC_TRY(launch_team<float>(m, ta, r_most, n, p.blocks_per_sm, cs));
    }
    if (rerun) {
        FlagArgs fa{};
        fa.state32 = (const float *)s.state;
        fa.stride = state_stride(p.method);
        fa.cls = s.cls;
        fa.flags = p.flags;
        fa.cls2 = s.cls2;
        fa.margin = p.rerun_margin;
        fa.pivot = p.rerun_pivot;
        fa.cond = p.rerun_cond;
        // a warm fit's reject says nothing about where the reference start's
        // path ends: with a proposal every flagged fit is re-run
        fa.skip_rej = p.warm ? 0.0f : p.rerun_skip_rejected;
        fa.w0 = (float)p.w0;
        fa.warm_limit = p.warm ? p.warm_iter_limit : 0;
        fa.long_iters = p.long_rerun_iters;
        fa.capped = p.rerun_capped;
        fa.iters_min = p.rerun_iters;
        // One re-run: flag a set of fits and solve them again in FP64, on
        // stream fs. Re-run 0 takes the fits that the first level finished (or
        // all, in a team-only call) and runs beside the second level; re-run 1
        // takes the fits that were suspended. Their lists share arrays from
        // both ends and use different counters.
        auto flag = [&](int set, cudaStream_t fs) -> cudaError_t {
            FlagArgs f = fa;
            f.list = set ? s.cont : s.order;
            f.count = s.meta + (set ? M_NCONT : M_TOTAL);
            f.list_b = set ? s.cont + n - 1 : nullptr;
            f.count_b = set ? s.meta + M_NLEFT : nullptr;
            f.suspended = set;
            f.shorts = s.order2 + (set ? n - 1 : 0);
            f.n_short = s.meta2 + (set ? M_NCONT : M_TOTAL);
            f.longs = long_q ? s.order3 + (set ? n - 1 : 0) : nullptr;
            f.n_long = s.meta3 + (set ? M_NCONT : M_TOTAL);
            f.step = set ? -1 : 1;
            const int fb = n < 2 * 148 * 256 ? (n + 255) / 256 : 2 * 148;
            if (m == 0) k3_flag<5><<<fb, 256, 0, fs>>>(f);
            else if (m == 1) k3_flag<4><<<fb, 256, 0, fs>>>(f);
            else k3_flag<7><<<fb, 256, 0, fs>>>(f);
            return cudaGetLastError();
        };
        auto rerun_fits = [&](int set, cudaStream_t fs) -> cudaError_t {
            const int step = set ? -1 : 1, c_total = set ? M_NCONT : M_TOTAL, c_next = set ? M_CONTNEXT : M_NEXT;
            int *shorts = s.order2 + (set ? n - 1 : 0), *longs = long_q ? s.order3 + (set ? n - 1 : 0) : nullptr;
            // the class order is used up: the fits left to the teams go there
            int *left64 = s.order + (set ? n - 1 : 0);
            int *meta_left = set ? s.meta3 : s.meta2;
            K1Args kd = k1;
            kd.state = s.state64;
            kd.stats = s.stats + ST_N;   // counters of the re-run kept apart
            kd.pivot_thr = 0.0f;
            if (p.warm) kd.init_params = nullptr;   // warm-started fits fall back to the reference start
            kd.left = left64;
            kd.left_step = step;
            kd.n_left = meta_left + M_NLEFT;
            kd.least = fits64;
            kd.list_step = step;
            TeamArgs td{};
            td.k = kd;
            td.switch_it = p.max_iter;
            td.q0 = td.q1 = 1;
            td.next = meta_left + M_LEFTNEXT;
            const int most = team_only ? n : fits64;
            // No thread groups for the long re-runs of set 0: what the first
            // level finished took at most its budget, but for fits whose residual
            // became exactly zero (they end at the iteration cap at once, see
            // start_iteration). Those go to the teams, however many they are.
            const bool no_long = !long_q || (set == 0 && two_level && p.level0_budget <= p.long_rerun_iters);
            // the long re-runs first: they set the length of the launch
            if (long_q)
                td.list[0] = TeamList{longs, s.meta3 + c_total, step, 1, p.long_rerun_threads_per_fit, no_long ? n : most};
            td.list[1] = TeamList{shorts, s.meta2 + c_total, step, 1, p.rerun_threads_per_fit, most};
            if (!team_only) {
                // more flagged fits than the teams take: groups of threads first
                for (int k = no_long ? 1 : 0; k < 2; ++k) {
                    const int tpf = k == 0 ? p.long_rerun_threads_per_fit : p.rerun_threads_per_fit;
                    kd.list = k == 0 ? longs : shorts;
                    kd.count = (k == 0 ? s.meta3 : s.meta2) + c_total;
                    kd.next = (k == 0 ? s.meta3 : s.meta2) + c_next;
                    kd.drain = tiny ? 0 : tpf <= 2 ? kDrain2 : 1;
                    LOC_TRY(launch_list_m<double>(m, kd, r_most, tpb, p.blocks_per_sm, tpf, fs));
                }
                td.list[2] = TeamList{left64, meta_left + M_NLEFT, step, 0, 0, n};
            }
            LOC_TRY(launch_team<double>(m, td, r_most, n, p.blocks_per_sm, fs));
            return cudaSuccess;
        };
        // flagged before the suspended ones: that pass gives their marks up
        LOC_TRY(flag(0, stream));
        if (!team_only) {
            // the suspended fits' re-run follows both launches of the second level
            if (naux > 0 && (e = cudaEventRecord(p.fork, stream)) != cudaSuccess) return e;
            if ((e = side(0, &cs)) != cudaSuccess) return e;
            if (naux > 0 && (e = cudaStreamWaitEvent(cs, p.fork, 0)) != cudaSuccess) return e;
            if (naux > 1 && used[1]) {
                if ((e = cudaEventRecord(p.join[1], p.aux[1])) != cudaSuccess) return e;
                if ((e = cudaStreamWaitEvent(cs, p.join[1], 0)) != cudaSuccess) return e;
            }
            LOC_TRY(flag(1, cs));
            if ((e = rerun_fits(1, cs)) != cudaSuccess) return e;
        }
        if ((e = rerun_fits(0, stream)) != cudaSuccess) return e;
    }
    if ((e = join()) != cudaSuccess) return e;
#undef LOC_TRY
    mark(2);
    K2Args k2{(const Cand *)p.cands, n, p.method, p.w0, r_default,
              p.precision == 1 ? nullptr : (const float *)s.state,
              p.precision == 1 ? (const double *)s.state : s.state64, rerun ? s.cls2 : nullptr,
              state_stride(p.method), ncol_total, p.out, p.flags, p.params_out, p.diag};
    bump();
    switch (p.method) {
    case 0: k2_finalize<0><<<nb, 256, 0, stream>>>(k2); break;
    case 1: k2_finalize<1><<<nb, 256, 0, stream>>>(k2); break;
    case 5: k2_finalize<5><<<nb, 256, 0, stream>>>(k2); break;
    default: k2_finalize<7><<<nb, 256, 0, stream>>>(k2); break;
    }
    mark(3);
    return cudaGetLastError();
}

}  // namespace locb
