// Team solver: a warp, or a block of four warps, works on one fit.
//
// The thread-per-fit solver (run_class in loc_fit.cu) has the better
// throughput while every lane has a fit, but a single fit takes as long as
// one thread needs for all its pixels. The team solver takes the work where
// that latency, not throughput, sets the time: the fits that outlive the
// first level or are left when its queue runs dry, the FP64 re-runs, the
// all-FP64 solve, and whole calls too small to give every lane a fit.
//
// It computes bit for bit what a group of Q cooperating threads computes in
// run_class (Q partial sums over the columns q, q + Q, ... of every row, added
// pairwise), so a fit may move between the two at any iteration:
//   1. the lanes evaluate the pixels of a few rows in parallel and leave each
//      pixel's Jacobian columns, 1, the residual and the two factors of the
//      |r|^2 change in shared memory;
//   2. the sums of products of these columns are dealt out to the lanes in
//      2 x 2 blocks per partial sum, and each lane runs its chains over the
//      pixels in the serial order (four independent chains hide the FMA
//      latency; a block's operands are two vector loads per pixel);
//   3. one lane per matrix entry adds the Q partial sums in the order of the
//      threads' butterfly.
// The damped solve runs on every lane (its chain of pivots is serial); the
// per-parameter work of the accept/reject logic is spread over the lanes.
//
// In a team of four warps the pass is spread over 128 threads, and every warp
// does the rest of the iteration for itself: all of them read the same sums and
// arrive at the same step, so nothing has to be handed round.
#pragma once

#include "loc_device.cuh"

namespace locb {
namespace {

template <typename T> struct Vec2;
template <> struct Vec2<float> { using type = float2; };
template <> struct Vec2<double> { using type = double2; };

// One pair from shared memory, kept where it stands in the program: the chains
// below read their operands ahead, and left to itself the compiler moves the
// loads back to their use (20 000 all-FP64 fits 2.36 ms, with this 2.19 ms;
// the FP32 calls stay within 3 %). The memory clobber orders the loads after
// the plain stores that filled the records.
__device__ __forceinline__ void lds_pair(float2 &v, uint32_t at)
{
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(at) : "memory");
}
__device__ __forceinline__ void lds_pair(double2 &v, uint32_t at)
{
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(at) : "memory");
}

constexpr int kTeamChunk = 64;   // pixels per warp of the team whose columns are in shared memory at a time
constexpr int kTeamAhead = 4;    // records that a chain reads ahead, past the chunk's last one too
// records of a team's chunk: what is read ahead of a full chunk lies in memory
// that nobody writes
__host__ __device__ constexpr int team_records(int warps) { return warps * kTeamChunk + kTeamAhead; }

// a team is a warp (W == 1) or a block of W warps
template <int W> __device__ __forceinline__ void team_sync()
{
    if constexpr (W == 1) __syncwarp();
    else __syncthreads();
}

// Columns of one pixel, in pairs: the Jacobian columns, 1, r (and a zero to
// fill the pair), then del and 2 r - del.
template <int METHOD> struct TeamDims {
    static constexpr int P = Traits<METHOD>::P;
    static constexpr int NT = tri(P);
    static constexpr int PAIRS = (P + 2) / 2;                       // of columns, 1 and r
    static constexpr int NB = PAIRS * (PAIRS + 1) / 2 + 1;          // 2 x 2 blocks; the last is del x (2 r - del)
    static constexpr int VS = 10;                                   // values per pixel (odd multiple of a 16-byte
                                                                    // or 8-byte word: conflict-free)
    static constexpr int NE = NT + P + 2;                           // entries: A, v, |r|^2, |r|^2 change
    static_assert(2 * (PAIRS + 1) <= VS, "columns of a pixel");
    static_assert(NT <= 32 && NB * 8 <= 96 && PAIRS < 15, "one matrix entry and at most three units per lane");
};

// where entry e of (A packed, v, chi2, dchi) is in a partial sum's blocks
template <int METHOD> __device__ __forceinline__ int team_entry(int e)
{
    using D = TeamDims<METHOD>;
    int m = 0, n = 0;
    if (e < D::NT) {
        int left = e;
        while (left >= D::P - m) {
            left -= D::P - m;
            ++m;
        }
        n = m + left;
    } else if (e < D::NT + D::P) {
        m = e - D::NT;
        n = D::P;
    } else if (e == D::NT + D::P) {
        m = n = D::P;
    } else {
        return (D::NB - 1) * 4 + 1;
    }
    const int pm = m / 2, pn = n / 2;
    return (pm * D::PAIRS - pm * (pm - 1) / 2 + pn - pm) * 4 + (m & 1) * 2 + (n & 1);
}

// unit u: the two pairs of its block and its partial sum, a | b << 4 | q << 8
template <int METHOD> __device__ __forceinline__ int team_unit(int u)
{
    using D = TeamDims<METHOD>;
    int b = u % D::NB, pa = 0;
    const int q = (u / D::NB) & 7;
    if (b == D::NB - 1) return D::PAIRS * 17 | q << 8;
    while (b >= D::PAIRS - pa) {
        b -= D::PAIRS - pa;
        ++pa;
    }
    return pa | (pa + b) << 4 | q << 8;
}

// One pixel's columns at the evaluation point; the expressions are those of
// pass_sym, pass_fixed and pass_ell, statement for statement.
template <int METHOD, typename T> struct PixelEval;

template <typename T> struct PixelEval<0, T> {
    T A, x0, y0, b, dA, dxs, dys, db, A0, c1, ka_x, ka_r, cc, dc, m2dx;
    bool fused;
    __device__ __forceinline__ void prep(const T (&th)[5], const T (&dth)[5], T, int, bool row_fused)
    {
        fused = row_fused;
        const T w = th[1], dw = dth[1];
        A = th[0];
        x0 = th[2];
        y0 = th[3];
        b = th[4];
        dA = dth[0];
        dxs = dth[2];
        dys = dth[3];
        db = dth[4];
        A0 = A - dA;
        const T w0c = w - dw;
        const T w2i = T(1) / (w * w);
        c1 = -T(0.5) * w2i * (T)Expo<T>::scale;
        ka_x = A * w2i;
        ka_r = ka_x / (w * T(1.4142135623730950488));
        cc = T(0.5) / (w0c * w0c);
        const T cpr = T(0.5) * w2i;
        dc = -T(2) * dw * (T(2) * w0c + dw) * cc * cpr;
        m2dx = -T(2) * dxs;
    }
    __device__ __forceinline__ T eval(int i, int j, T dat, T (&o)[8]) const
    {
        const T wy = (T)j - y0;
        const T wy2 = wy * wy;
        const T krow = row_term<T>(fused, dxs, dys, wy);
        const T u = (T)i - x0;
        const T d2 = fma(u, u, wy2);
        const T e = Expo<T>::ex(d2 * c1);
        const T r = fma(A, e, b - dat);
        const T dd = fma(m2dx, u, krow);
        const T ydq = fma(d2, dc, cc * dd);
        const T del = fma(e, fma(-A0, expm1_series(ydq), dA), db);
        const T jr = d2 * (e * ka_r);
        const T ex = e * ka_x;
        const T jx = u * ex, jy = wy * ex;
        o[0] = e;
        o[1] = jr;
        o[2] = jx;
        o[3] = jy;
        o[4] = T(1);
        o[5] = r;
        o[6] = del;
        o[7] = fma(T(2), r, -del);
        return fabs(ydq);
    }
};

template <typename T> struct PixelEval<1, T> {
    T A, x0, y0, b, dA, dxs, dys, db, A0, c1, ka_x, cc, m2dx;
    bool fused;
    __device__ __forceinline__ void prep(const T (&th)[4], const T (&dth)[4], T w0, int, bool row_fused)
    {
        fused = row_fused;
        A = th[0];
        x0 = th[1];
        y0 = th[2];
        b = th[3];
        dA = dth[0];
        dxs = dth[1];
        dys = dth[2];
        db = dth[3];
        A0 = A - dA;
        const T w2i = T(1) / (w0 * w0);
        c1 = -T(0.5) * w2i * (T)Expo<T>::scale;
        ka_x = A * w2i;
        cc = T(0.5) * w2i;
        m2dx = -T(2) * dxs;
    }
    __device__ __forceinline__ T eval(int i, int j, T dat, T (&o)[8]) const
    {
        const T wy = (T)j - y0;
        const T wy2 = wy * wy;
        const T krow = row_term<T>(fused, dxs, dys, wy);
        const T u = (T)i - x0;
        const T d2 = fma(u, u, wy2);
        const T e = Expo<T>::ex(d2 * c1);
        const T r = fma(A, e, b - dat);
        const T ydq = cc * fma(m2dx, u, krow);
        const T del = fma(e, fma(-A0, expm1_series(ydq), dA), db);
        const T ex = e * ka_x;
        const T jx = u * ex, jy = wy * ex;
        o[0] = e;
        o[1] = jx;
        o[2] = jy;
        o[3] = T(1);
        o[4] = r;
        o[5] = T(0);
        o[6] = del;
        o[7] = fma(T(2), r, -del);
        return fabs(ydq);
    }
};

template <typename T> struct PixelEval<7, T> {
    T A, x0, y0, b, dA, dxs, dys, db, A0, isx, isy, a, c, rb, cexp, AK, ABK, rk, tr, da, dcq, drb, rb0, hk, hdk, dx2;
    __device__ __forceinline__ void prep(const T (&th)[7], const T (&dth)[7], T, int lane, bool)
    {
        const T sx = th[1], sy = th[2], rho = th[5];
        const T dsx = dth[1], dsy = dth[2], drho = dth[5];
        A = th[0];
        x0 = th[3];
        y0 = th[4];
        b = th[6];
        dA = dth[0];
        dxs = dth[3];
        dys = dth[4];
        db = dth[6];
        A0 = A - dA;
        const T sx0 = sx - dsx, sy0 = sy - dsy, rho0 = rho - drho;
        // six reciprocals, one per lane
        const int k6 = lane % 6;
        const T rr = k6 == 2 ? rho : rho0;
        T den = T(1) - rr * rr;
        if (k6 == 0) den = sx;
        if (k6 == 1) den = sy;
        if (k6 == 3) den = sx0;
        if (k6 == 4) den = sy0;
        const T inv = T(1) / den;
        isx = __shfl_sync(kFull, inv, 0);
        isy = __shfl_sync(kFull, inv, 1);
        const T k = __shfl_sync(kFull, inv, 2);
        const T isx0 = __shfl_sync(kFull, inv, 3), isy0 = __shfl_sync(kFull, inv, 4);
        const T k0 = __shfl_sync(kFull, inv, 5);
        a = isx * isx;
        c = isy * isy;
        const T bb = isx * isy;
        rb = rho * bb;
        cexp = -T(0.5) * k * (T)Expo<T>::scale;
        AK = A * k;
        ABK = AK * bb;
        rk = rho * k;
        tr = T(2) * rho;
        const T a0 = isx0 * isx0, c0 = isy0 * isy0, bb0 = isx0 * isy0;
        da = -dsx * (T(2) * sx0 + dsx) * a0 * a;
        dcq = -dsy * (T(2) * sy0 + dsy) * c0 * c;
        const T dbb = -(dsx * sy0 + sx * dsy) * bb0 * bb;
        drb = drho * bb + rho0 * dbb;
        const T dk = drho * (T(2) * rho0 + drho) * k0 * k;
        rb0 = rho0 * bb0;
        hk = -T(0.5) * k;
        hdk = -T(0.5) * dk;
        dx2 = dxs * dxs;
    }
    __device__ __forceinline__ T eval(int i, int j, T dat, T (&o)[10]) const
    {
        const T wy = (T)j - y0;
        const T wy2 = wy * wy;
        const T wc = wy * c;
        const T wrb = wy * rb;
        const T wcur = wy + dys;
        const T brow = T(2) * (dxs * (da - a) - drb * wy + rb0 * dys);
        const T crow = (da - a) * dx2 - c * dys * (T(2) * wy + dys) + dcq * wcur * wcur +
                       T(2) * rb0 * dxs * wcur;
        const T u = (T)i - x0;
        const T P1 = fma(u, a, -wrb);
        const T P2 = fma(-rb, u, wc);
        const T q = fma(u, P1, wy * P2);
        const T e = Expo<T>::ex(q * cexp);
        const T r = fma(A, e, b - dat);
        const T dQ = fma(fma(da, u, brow), u, crow);
        const T ydq = -fma(hk, dQ, hdk * (q - dQ));
        const T del = fma(e, fma(-A0, expm1_series(ydq), dA), db);
        const T ek = e * AK;
        const T jx = ek * P1, jy = ek * P2;
        const T jsx = (jx * u) * isx;
        const T jsy = (jy * wy) * isy;
        const T uw = u * wy;
        const T d2 = fma(u, u, wy2);
        const T inner = fma(-tr, uw, d2);
        const T t = fma(-rk, inner, uw);
        const T jrho = (e * ABK) * t;
        o[0] = e;
        o[1] = jsx;
        o[2] = jsy;
        o[3] = jx;
        o[4] = jy;
        o[5] = jrho;
        o[6] = T(1);
        o[7] = r;
        o[8] = del;
        o[9] = fma(T(2), r, -del);
        return fabs(ydq);
    }
};

// Shared memory of one team: ROI pixels, a chunk of columns, the partial sums,
// then the state: A and v of the current and of the trial point, the scaled
// matrix, and per-parameter vectors.
__host__ __device__ constexpr int team_roi_bytes(int r) { return ((2 * r + 1) * (2 * r + 1) * 4 + 15) / 16 * 16; }
template <int METHOD, typename T, int W> __host__ __device__ constexpr int team_smem(int r_cap)
{
    using D = TeamDims<METHOD>;
    return team_roi_bytes(r_cap) + (team_records(W) * D::VS + 8 * D::NB * 4) * (int)sizeof(T) +
           ((2 * D::NE + W * (D::NT + 3 * 8)) * (int)sizeof(T) + 4 + 15) / 16 * 16;
}

// largest of the (non-negative) values of lanes 0 to 7
__device__ __forceinline__ float max_of_8(float v)
{
    v = (threadIdx.x & 31) < 8 ? v : 0.0f;
    return __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(v)));
}
__device__ __forceinline__ double max_of_8(double v)
{
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(kFull, v, o));
    return __shfl_sync(kFull, v, 0);
}

// One pass over the ROI: the partial sums of q_n threads (1, 2, 4 or 8),
// combined into res (A and v times inv_s2, then |r|^2 and its change);
// returns whether every |q - q'| is below 0.25 (see expm1_series).
//
// A chunk is a few whole rows. A partial sum's pixels (columns q, q + q_n, ...
// of each row) lie next to each other in it, in order, so a lane's chains run
// over consecutive records whatever q_n is. Units (a 2 x 2 block of one
// partial sum) are dealt to the lanes in rounds; their sums rest in shared
// memory between chunks.
template <int METHOD, typename T, int W>
__device__ __forceinline__ bool team_pass(const float *roi, int s, T *chunk, T *sums, T *res,
                                       const T (&te)[Traits<METHOD>::P], const T (&dt)[Traits<METHOD>::P],
                                       const int (&entry)[TeamDims<METHOD>::NE / (32 * W) + 1], long long unit, T w0, T inv_s2,
                                       int q_n, bool fused, int wide, int tl)
{
    using D = TeamDims<METHOD>;
    using V2 = typename Vec2<T>::type;
    constexpr int NV = 2 * (D::PAIRS + 1);
    PixelEval<METHOD, T> px;
    px.prep(te, dt, w0, threadIdx.x & 31, fused);
    // columns per partial sum; the first `more` have one more
    const int qmask = q_n - 1, qshift = q_n == 8 ? 3 : q_n >> 1;
    const int units = D::NB * q_n, per = s >> qshift, more = s & qmask;
    constexpr int TN = 32 * W;
    const int rows = W * kTeamChunk / s;
    const uint32_t chunk_at = (uint32_t)__cvta_generic_to_shared(chunk);
    // this thread's pixels of a chunk: tl and tl + TN
    const int ja = tl / s, ia = tl - ja * s, jb = (tl + TN) / s, ib = tl + TN - jb * s;
    T dqmax = T(0);
    for (int j0 = 0; j0 < s; j0 += rows) {
        const int nr = min(rows, s - j0), n = nr * s;
        auto place = [&](int i, int j) {   // record of column i, row j of the chunk
            const int q = i & qmask;
            return chunk + (nr * (q * per + min(q, more)) + j * (per + (q < more ? 1 : 0)) + (i >> qshift)) * D::VS;
        };
        auto put = [&](T *to, const T (&o)[NV]) {
            V2 *dst = reinterpret_cast<V2 *>(to);
#pragma unroll
            for (int v = 0; v < NV / 2; ++v) {
                V2 w;
                w.x = o[2 * v];
                w.y = o[2 * v + 1];
                dst[v] = w;
            }
        };
        if (tl < n) {
            // both evaluations side by side: the second hides the first's latency
            const bool two = tl + TN < n;
            T oa[NV], ob[NV];
            const T da = px.eval(ia, j0 + ja, (T)roi[j0 * s + tl], oa);
            const T db = px.eval(ib, j0 + jb, (T)roi[j0 * s + (two ? tl + TN : tl)], ob);
            dqmax = fmax(dqmax, da);
            put(place(ia, ja), oa);
            if (two) {
                dqmax = fmax(dqmax, db);
                put(place(ib, jb), ob);
            }
        }
        team_sync<W>();
#pragma unroll 1
        for (int k = 0; k * TN + tl < units; ++k) {
            const int w = (int)(unit >> (k * 11)), q = (w >> 8) & 7;   // k < 3 only: NB * 8 <= 96
            constexpr uint32_t kRec = D::VS * sizeof(T), kPair = sizeof(V2);
            const uint32_t p = chunk_at + nr * (q * per + min(q, more)) * kRec;
            uint32_t pa = p + (w & 15) * kPair, pb = p + ((w >> 4) & 15) * kPair;
            const int cnt = nr * (per + (q < more ? 1 : 0));
            V2 *sum = reinterpret_cast<V2 *>(sums + (k * TN + tl) * 4);
            V2 lo = sum[0], hi = sum[1];
            if (j0 == 0) lo.x = lo.y = hi.x = hi.y = T(0);
            // operands are read kTeamAhead records ahead (past the last record
            // they come from another partial sum's, or from the room behind
            // the chunk, and are not used)
            V2 x[kTeamAhead], y[kTeamAhead];
#pragma unroll
            for (int d = 0; d < kTeamAhead; ++d) {
                lds_pair(x[d], pa + d * kRec);
                lds_pair(y[d], pb + d * kRec);
            }
            auto step = [&](int d) {
                lo.x = fma(x[d].x, y[d].x, lo.x);
                lo.y = fma(x[d].x, y[d].y, lo.y);
                hi.x = fma(x[d].y, y[d].x, hi.x);
                hi.y = fma(x[d].y, y[d].y, hi.y);
            };
            int at = kTeamAhead;
            for (; at <= cnt; at += kTeamAhead) {
                pa += kTeamAhead * kRec;
                pb += kTeamAhead * kRec;
#pragma unroll
                for (int d = 0; d < kTeamAhead; ++d) {
                    step(d);
                    lds_pair(x[d], pa + d * kRec);
                    lds_pair(y[d], pb + d * kRec);
                }
            }
            const int rest = cnt - at + kTeamAhead;
            if (rest > 0) step(0);
            if (rest > 1) step(1);
            if (rest > 2) step(2);
            sum[0] = lo;
            sum[1] = hi;
        }
        team_sync<W>();   // the sums are complete; the next chunk may overwrite this one
    }
    // the partial sums in the order of the threads' butterfly
#pragma unroll
    for (int k = 0; k < D::NE / TN + 1; ++k) {
        const int e = tl + k * TN;
        if (e >= D::NE) break;
        const T *p = sums + entry[k];
        auto at = [&](int q) { return p[q * D::NB * 4]; };
        T v;
        if (sizeof(T) == 4 && wide && e < D::NE - 1 && q_n > 1) {   // partial sums added in FP64
            auto d = [&](int q) { return (double)p[q * D::NB * 4]; };
            v = (T)(q_n == 8 ? ((d(0) + d(4)) + (d(2) + d(6))) + ((d(1) + d(5)) + (d(3) + d(7)))
                  : q_n == 4 ? (d(0) + d(2)) + (d(1) + d(3)) : d(0) + d(1));
        } else {
            v = q_n == 8 ? ((at(0) + at(4)) + (at(2) + at(6))) + ((at(1) + at(5)) + (at(3) + at(7)))
              : q_n == 4 ? (at(0) + at(2)) + (at(1) + at(3)) : q_n == 2 ? at(0) + at(1) : at(0);
        }
        res[e] = e < D::NT + D::P ? v * inv_s2 : v;
    }
    if constexpr (W > 1) return __syncthreads_and(dqmax < T(0.25)) != 0;
    __syncwarp();
    return __ballot_sync(kFull, !(dqmax < T(0.25))) == 0;
}

// What the team kernel works on: up to three lists of candidates, each fit
// with its own ROI half-width (k.cls).
struct TeamList {
    const int *list;    // entry i at list[i * step]
    const int *count;
    int step;
    int fresh;          // 1: start each candidate; 0: resume its suspended state
    int q_n;            // partial sums; 0: q0 and q1, or (FP64) what the suspended state says
    int most;           // longer lists are not taken (the thread groups have worked on them)
};
struct TeamArgs {
    K1Args k;               // frames, candidates, state, options, counters
    TeamList list[3];
    int *next;              // dequeue cursor over the lists
    int q0, q1, switch_it;  // partial sums up to and from iteration switch_it
};

// The fits of the lists (n_all of them, list k up to ends[k]), by teams of W
// warps.
template <int METHOD, typename T, bool ESC, int W>
__device__ __forceinline__ void team_fits(const TeamArgs &a, int r_cap, int n_all, const int (&ends)[3],
                                          unsigned char *sm_team)
{
    using D = TeamDims<METHOD>;
    constexpr int P = D::P, NT = D::NT, IX = Traits<METHOD>::IX;
    using SL = StateLayout<P>;
    const K1Args &ka = a.k;
    constexpr int TN = 32 * W;
    const int lane = threadIdx.x & 31, warp = threadIdx.x / 32;
    const int tl = W == 1 ? lane : threadIdx.x;      // thread of the team
    unsigned char *base = sm_team + (W == 1 ? warp : 0) * team_smem<METHOD, T, W>(r_cap);
    float *roi = reinterpret_cast<float *>(base);
    T *chunk = reinterpret_cast<T *>(base + team_roi_bytes(r_cap));
    T *sums = chunk + team_records(W) * D::VS;
    T *buf0 = sums + 8 * D::NB * 4;            // A, v, |r|^2 and its change, for two points
    T *msv = buf0 + 2 * D::NE + (W == 1 ? 0 : warp) * (NT + 3 * 8);   // each warp's own
    T *s_inv = msv + NT, *s_te = s_inv + 8, *s_dt = s_te + 8;
    int *s_next = reinterpret_cast<int *>(buf0 + 2 * D::NE + W * (NT + 3 * 8));
    const T inv_s2 = sizeof(T) == 4 ? (T)ka.inv_s2 : (T)ka.inv_s2_d;
    const T inv_abs_s = sizeof(T) == 4 ? (T)ka.inv_abs_s : (T)ka.inv_abs_s_d;
    const T w0 = (T)ka.w0;
    unsigned st[ST_N];
#pragma unroll
    for (int k = 0; k < ST_N; ++k) st[k] = 0;
    // lane k < P: parameter k; everything else is the same on every lane
    const bool mine = lane < P;
    const int own = mine ? lane : 0;
    int entry[D::NE / TN + 1];
#pragma unroll
    for (int k = 0; k < D::NE / TN + 1; ++k) entry[k] = tl + k * TN < D::NE ? team_entry<METHOD>(tl + k * TN) : 0;
    // this thread's units of a pass, 11 bits each, and its lane's entry of the scaled matrix
    const long long unit = (long long)team_unit<METHOD>(tl) | (long long)team_unit<METHOD>(tl + TN) << 11 |
                           (long long)team_unit<METHOD>(tl + 2 * TN) << 22;
    int mi = 0, mj = lane;
    while (mj >= P - mi && mi < P) {
        mj -= P - mi;
        ++mi;
    }
    mj += mi;
    const long long t_begin = clock64();
    unsigned long long c_pass = 0;

    while (true) {
        // ---- next fit ----
        int qi = 0;
        if (tl == 0) qi = atomicAdd(a.next, 1);
        if constexpr (W == 1) {
            qi = __shfl_sync(kFull, qi, 0);
        } else {
            if (tl == 0) *s_next = qi;
            __syncthreads();
            qi = *s_next;
        }
        if (qi >= n_all) break;
        int li = 0;
        while (qi >= ends[li]) ++li;
        const TeamList &L = li == 0 ? a.list[0] : li == 1 ? a.list[1] : a.list[2];
        const int cidx = L.list[(long long)(qi - (li == 0 ? 0 : li == 1 ? ends[0] : ends[1])) * L.step];
        const int r = ka.cls[cidx], s = 2 * r + 1, npx = s * s;
        const Cand cd = ka.cands[cidx];
        const int xo = (int)floor(cd.x - (double)r), yo = (int)floor(cd.y - (double)r);
        {
            const long long org = ka.roi_slot ? (long long)ka.roi_slot[cidx]
                                              : (long long)cd.frame * ka.frame_px + xo + (long long)yo * ka.n_rows;
            const int pitch = ka.roi_slot ? s : ka.n_rows;   // a packed ROI's rows are 2r + 1 pixels apart
            const uint16_t *fb = ka.frames + org;
            int j = tl / s, i = tl - j * s;
#pragma unroll 4
            for (int k = tl; k < npx; k += TN) {
                roi[k] = (float)__ldg(fb + i + (size_t)j * pitch);
                i += TN;
                while (i >= s) {
                    i -= s;
                    ++j;
                }
            }
        }
        // the current point (th), the trial point (te), the last step (dx) and
        // the scaling (sc) of this lane's parameter
        T th = T(0), te = T(0), dx = T(0), sc = T(1);
        T *cur = buf0, *alt = buf0 + D::NE;   // sums of the current point; of the trial point
        T fnorm = 0, delta = 0, par = 0, xnorm = 0, minpiv_fit = T(1), margin_fit = T(1e30);
        int it_state = 0, iterations = 0, done = -1, q_fix = L.q_n;
        unsigned esc_fit = 0;
        bool first = L.fresh != 0;
        if (first) {
            if (ka.init_params && !isnan(ka.init_params[(size_t)cidx * P])) {
                const double off = lane == IX ? (double)xo : (lane == IX + 1 ? (double)yo : 0.0);
                if (mine) th = (T)((double)ka.init_params[(size_t)cidx * P + lane] - off);
            } else {
                th = lane == 0 ? (T)cd.intensity : lane == P - 1 ? (T)cd.background : w0;
                if (lane == IX) th = (T)(cd.x - (double)xo);
                if (lane == IX + 1) th = (T)(cd.y - (double)yo);
                if (METHOD == 7 && lane == 5) th = T(0);
            }
        } else {
            const Saved<T> o = saved_of<P, T>(ka.cont_state, ka.cont_stride, ka.state, ka.state_stride, cidx);
            if (mine) {
                th = o.th[lane];
                sc = o.D[lane];
                dx = o.dx[lane];
                if (W == 1 || warp == 0) cur[NT + lane] = o.v[lane];
            }
            for (int k = tl; k < NT; k += TN) cur[k] = o.A[k];
            const Scalars<T> c = load_scalars<T>(o.sc);
            fnorm = c.fnorm;
            delta = c.delta;
            par = c.par;
            xnorm = c.xnorm;
            minpiv_fit = c.minpiv;
            margin_fit = c.margin;
            it_state = c.it_state;
            iterations = c.iterations;
            esc_fit = c.esc;
            if (sizeof(T) == 8) q_fix = c.q_n;
        }
        team_sync<W>();
        auto theta_abs = [&](T t) -> T { return lane == IX ? t + (T)xo : (lane == IX + 1 ? t + (T)yo : t); };
        // largest step / test_delta tolerance over the parameters (at t), and
        // whether every step is below its tolerance
        auto step_test = [&](T t, bool &small) -> T {
            const T tol = (T)ka.epsabs + (T)ka.epsrel * fabs(theta_abs(t));
            small = __ballot_sync(kFull, mine && !(fabs(dx) < tol)) == 0;
            const T qq = fdiv(fabs(dx), tol);
            return max_of_8(mine && qq > T(0) ? qq : T(0));
        };
        int trial = 0;
        while (true) {
            // ---- evaluation point ----
            T pnorm = T(0), jdx2 = T(0);
            const int q_n = q_fix > 0 ? q_fix : iterations + (trial == 0 && !first ? 1 : 0) > a.switch_it ? a.q1 : a.q0;
            if (first) {
                te = th;
            } else {
                if (trial == 0) {   // next outer iteration
                    ++iterations;
                    if (fnorm == T(0)) {   // iterate() returns at once; dx is unchanged
                        bool small;
                        margin_fit = fmin(margin_fit, fabs(step_test(th, small) - T(1)));
                        if (!small) iterations = ka.max_iter;
                        done = small ? T_CONVERGED : T_MAX_ITER;
                        break;
                    }
                }
                ++trial;
                const T inv_d = frcp(sc);
                if (mine) s_inv[lane] = inv_d;
                __syncwarp();
                if (lane < NT) msv[lane] = cur[lane] * s_inv[mi] * s_inv[mj];
                T gv[P], inv_dv[P], z[P];
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    inv_dv[k] = s_inv[k];
                    gv[k] = cur[NT + k];
                }
                __syncwarp();
                const T *Ms = msv;
                bool sing = false;
                unsigned nl = 0, ne = 0;
                T npiv;
                lmpar_scaled<P, T, ESC, false>(Ms, gv, inv_dv, sym_fuse<ESC>(s, q_n), delta, par, z, ka.pivot_thr, nl, ne, sing,
                                               npiv, margin_fit);
                if (tl == 0) {
                    st[ST_LAMBDA] += nl;
                    st[ST_ESC] += ne;
                }
                esc_fit += ne;
                minpiv_fit = npiv < minpiv_fit ? npiv : minpiv_fit;
                if (sing) {
                    done = T_SINGULAR;
                    break;
                }
                T zk = z[0], pn2 = T(0), row = T(0), z0;
#pragma unroll
                for (int k = 0; k < P; ++k) {
                    if (k == lane) zk = z[k];
                    add_square<T>(z[k], k, z0, pn2);
                }
#pragma unroll
                for (int j = 0; j < P; ++j) {
                    const int lo = min(own, j), hi = max(own, j);
                    row = fma(Ms[pku(P, lo, hi)], z[j], row);
                }
#pragma unroll
                for (int i = 0; i < P; ++i) jdx2 = fma(z[i], __shfl_sync(kFull, row, i), jdx2);
                if (mine) {
                    dx = -zk * inv_d;
                    te = th + dx;
                }
                pnorm = fsqrt(pn2);
                if (it_state == 1 && pnorm < delta) delta = pnorm;
                if (__ballot_sync(kFull, te == T(0) && ((METHOD == 0 && lane == 1) ||
                                                        (METHOD == 7 && (lane == 1 || lane == 2))))) {
                    done = T_EBADFUNC;
                    break;
                }
            }

            // ---- the pass ----
            const long long t_pass = clock64();
            if (mine) {
                s_te[lane] = te;
                s_dt[lane] = first ? T(0) : dx;
            }
            __syncwarp();
            T tev[P], dtv[P];
#pragma unroll
            for (int k = 0; k < P; ++k) {
                tev[k] = s_te[k];
                dtv[k] = s_dt[k];
            }
            const bool near = team_pass<METHOD, T, W>(roi, s, chunk, sums, alt, tev, dtv, entry, unit, w0, inv_s2, q_n,
                                                      row_fused<METHOD, T, ESC>(s, q_n), ka.compensated, tl);
            if (tl == 0) {
                if (first) {
                    st[ST_J] += 1;
                    st[ST_PIXJ] += npx;
                } else {
                    st[ST_F] += 1;
                    st[ST_PIXF] += npx;
                }
            }
            c_pass += (unsigned long long)(clock64() - t_pass);

            // ---- decide ----
            const T chi2 = alt[NT + P], dchi = alt[NT + P + 1];
            const T fn1 = fsqrt(chi2) * inv_abs_s;
            T actred = T(-1), prered = T(0), ratio = T(0);
            bool accept = true;
            if (!first) {
                if (T(0.1) * fn1 < fnorm) {
                    if (near) {
                        // accurate |f|^2 change from the per-pixel model differences
                        actred = fdiv(-(dchi * inv_s2), fnorm * fnorm);
                    } else {
                        const T u = fdiv(fn1, fnorm);
                        actred = T(1) - u * u;
                    }
                }
                const T if2 = frcp(fnorm * fnorm);
                const T t2s = mul_rn(mul_rn(mul_rn(par, pnorm), pnorm), if2);
                prered = fma(jdx2, if2, T(2) * t2s);
                const T dirder = -fma(jdx2, if2, t2s);
                ratio = prered > T(0) ? fdiv(actred, prered) : T(0);
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
                accept = ratio >= T(1e-4);
            }
            if (accept) {
                const T cn = sqrt(alt[pku(P, own, own)]);
                const T cn1 = cn == T(0) ? T(1) : cn;
                if (first) sc = cn1;   // gsl_multifit_fdfsolver_set for lmsder
                th = te;
                // |D x|, summed over the parameters in order
                const T tx = sc * theta_abs(th);
                T xn2 = T(0), t0;
#pragma unroll
                for (int k = 0; k < P; ++k) add_square<T>(__shfl_sync(kFull, tx, k), k, t0, xn2);
                xnorm = sqrt(xn2);
                fnorm = fn1;
                T *x = cur;            // the trial point's sums become the current ones
                cur = alt;
                alt = x;
                trial = 0;
                if (first) {
                    dx = T(0);
                    delta = xnorm > T(0) ? T(100) * xnorm : T(100);
                    par = T(0);
                    it_state = 1;
                    iterations = 0;
                    first = false;
                } else {
                    ++it_state;
                    if (tl == 0) {
                        st[ST_J] += 1;   // the accepted trial's Jacobian
                        st[ST_PIXJ] += npx;
                    }
                    if (cn1 > sc) sc = cn1;
                    bool small;
                    margin_fit = fmin(margin_fit, fabs(step_test(th, small) - T(1)));
                    if (small || iterations >= ka.max_iter) {
                        done = small ? T_CONVERGED : T_MAX_ITER;
                        break;
                    }
                }
            } else {
                const T gk = fabs(fdiv(cur[NT + own], sc));
                const T gnorm = fdiv(max_of_8(mine && gk > T(0) ? gk : T(0)), fnorm);
                if (fabs(actred) <= (T)kDblEps && prered <= (T)kDblEps && T(0.5) * ratio <= T(1)) done = T_ETOLF;
                else if (delta <= (T)kDblEps * xnorm) done = T_ETOLX;
                else if (gnorm <= (T)kDblEps) done = T_ETOLG;
                else if (trial >= 10) done = T_ENOPROG;
                if (done >= 0) break;
            }
        }

        // ---- write out ----
        bool small;
        const T lastr = step_test(th, small);
        T *o = (T *)ka.state + (size_t)cidx * ka.state_stride;
        if (tl < P) o[lane] = th;
        for (int k = tl; k < NT; k += TN) o[P + k] = cur[k];
        if (tl == 0) {
            o[SL::FNORM] = fnorm;
            o[SL::ITERS] = (T)iterations;
            o[SL::STATUS] = (T)done;
            o[SL::XOFF] = (T)xo;
            o[SL::YOFF] = (T)yo;
            o[SL::MINPIV] = minpiv_fit;
            o[SL::LASTR] = lastr;
            o[SL::NESC] = (T)esc_fit;
            o[SL::MARGIN] = margin_fit;
            st[ST_FITS] += 1;
            st[ST_ITERS] += iterations;
        }
        team_sync<W>();   // the next fit's ROI and sums take this one's place
    }
    if (tl == 0) {
        const unsigned long long all = (unsigned long long)(clock64() - t_begin);
        st[ST_CYC_STEP] += (unsigned)((all - c_pass) >> 10);
        st[ST_CYC_PASS] += (unsigned)(c_pass >> 10);
#pragma unroll
        for (int k = 0; k < ST_N; ++k)
            if (st[k]) atomicAdd(&ka.stats[k], (unsigned long long)st[k]);
    }
}

// Lists of up to `line` fits are solved by teams of four warps, longer ones by
// teams of one (kBlockFits32, kBlockFits64): the length is known on the device
// only. One launch that holds both takes 5 to 8 us less than two of which one
// returns at once, in the chain of every call beyond the warps alone (12 000
// fixed-width fits of 5 x 5 ROIs: 144 -> 137 us).
template <int METHOD, typename T, bool ESC>
__global__ void __launch_bounds__(128, sizeof(T) == 8 || ESC ? 3 : 4) k_team(TeamArgs a, int r_cap, int line)
{
    extern __shared__ __align__(16) unsigned char sm_team[];
    int ends[3], n_all = 0;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int n = a.list[k].count ? *a.list[k].count : 0;
        if (n <= a.list[k].most) n_all += n;
        ends[k] = n_all;
    }
    if (n_all == 0) return;
    if (n_all <= line) team_fits<METHOD, T, ESC, 4>(a, r_cap, n_all, ends, sm_team);
    else team_fits<METHOD, T, ESC, 1>(a, r_cap, n_all, ends, sm_team);
}

}  // namespace
}  // namespace locb
