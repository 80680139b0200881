// GPU candidate finder: GLRT detection + adjacent-8 particle grouping,
// restating ThresholdImage_GLRT_FFT (reference source/Segmentation.cpp:241-430)
// and ParticleFinder_adjacent8 (source/ParticleFinding.cpp:283-427) with the
// same results, bit for bit, as the host finder in loc_finder.cpp:
//
// * The GLRT decision of every interior pixel is the one of the reference's
//   floating-point operation sequence (zero-mean Gaussian window computed on
//   the host in double; exact integer window sums; the correlation
//   accumulated row by row in double with separate multiply and add; the test
//   value in the host's order). That sequence runs only where the decision is
//   close: an FP32 estimate of the same statistic with a proven error bound
//   decides the other pixels (k_glrt).
// * Connected components (8-neighbourhood) over runs of mask pixels by
//   union-find with links always pointing to the smaller run index; runs are
//   numbered in raster order, so a component's root is the run of its first
//   pixel in raster order. Particles are numbered in that order, which is the
//   order in which the reference's raster scan discovers them.
// * Particle position = unweighted mean of the component's pixel coordinates,
//   intensity = brightest pixel minus the frame background, background =
//   mean of the frame's pixels outside the mask: integer sums, exact in
//   double, divided once, as on the host.
//
// The mask is one bit per pixel. Frames are processed in chunks so that the
// working arrays stay within a bounded scratch.
#include "../../include/localizer_b200.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

namespace locb {
int record_error_fixed(int code, const char *msg);
}

namespace {

constexpr int kMaxWin = 33;    // window side up to ceil(4 w) = 33 (w <= 8)
constexpr unsigned kFull = 0xffffffffu;
constexpr int kLinkLimit = 1 << 24;

// What the decision needs, and the window.
struct Glrt {
    int n_rows, n_cols, words;      // words: 32-pixel mask words per row
    double npix, sumsq, thr;
    const double *g;                // ws x ws zero-mean window, row-major (b, a)
    // FP32 estimate (k_glrt_fast): the window is g1(a) g1(b) - mean
    float g1[13];
    float mean, inv_n, hi, lo, sat, fsumsq;
};

// The reference's operation sequence for one pixel; value(a, b) is the pixel
// at window column a, row b, as an exact integer in double.
template <typename F>
__device__ __forceinline__ bool glrt_exact(const Glrt &p, int ws, F value)
{
    long long s1 = 0, s2 = 0;
    double conv = 0.0;
    for (int b = 0; b < ws; ++b) {
        const double *gr = p.g + b * ws;
        for (int a = 0; a < ws; ++a) {
            const int iv = value(a, b);
            s1 += iv;
            s2 += (long long)iv * iv;
            conv = __dadd_rn(conv, __dmul_rn((double)iv, gr[a]));
        }
    }
    const double avg = __ddiv_rn((double)s1, p.npix);
    const double null_h = __dsub_rn((double)s2, __dmul_rn(__dmul_rn(avg, avg), p.npix));
    const double alpha = __ddiv_rn(conv, p.sumsq);
    const double test = __dmul_rn(__ddiv_rn(__dmul_rn(alpha, alpha), null_h), p.sumsq);
    return test < 1.0 && test > p.thr;
}

__device__ __forceinline__ void add_total(unsigned s, unsigned long long *total)
{
    unsigned long long t = s;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(kFull, t, o);
    if ((threadIdx.x & 31) == 0 && t) atomicAdd(total, t);
}

// ---------------------------------------------------------------------------
// GLRT mask of a chunk of frames, one bit per pixel, and the pixel total of
// each frame (the background sum is that total minus the mask's pixels).
//
// Evaluating the reference's FP64 sequence everywhere is bound by instruction
// issue (about 1000 thread instructions a pixel at ws = 7: 4.5 ms for 500
// frames of 512 x 512, 7.6 ms with the grouping). Here a block stages a tile as
// FP32 offsets from a pixel value c of the tile (exact integers), each lane
// owns PX neighbouring columns and marches down the rows: the separable part
// of the window is a 7-tap row sum and a 7-tap column sum over a register
// ring, the sums of v and v^2 likewise, with the tile's load and halo about
// 105 instructions a pixel (counted; the whole search of those frames: 15.2 ->
// 0.80 ms).
//
// With S = sum (v - c)^2, null = S - (sum (v - c))^2 / n and u = 2^-24, the
// FP32 errors are |d conv| <= (2 ws + 2) u |gg| sqrt(S) + 2 u mean sqrt(n S)
// and |d null| <= (2 ws + 4) u S, so where S <= 256 null the estimate T of
// conv^2 / (sumsq null) is off by less than the margin that the host folds
// into lo and hi (four times the bound). Outside [lo, hi] the estimate
// decides; between them, where the conditions fail (nearly constant windows,
// T near 1) the reference sequence runs. A window of pixels all equal to c
// has S = 0 and no signal: the reference's test value is then 0/0 or x/0,
// never inside (thr, 1).
// ---------------------------------------------------------------------------
constexpr int kWarps = 4;
template <int WS> struct FastTile {
    static constexpr int PX = WS <= 7 ? 4 : 2;          // columns per lane (register ring: 3 WS PX floats)
    static constexpr int HALF = WS / 2;
    static constexpr int TW = 32 * PX;                  // tile width
    static constexpr int R = 3 * WS + 1;                // output rows per warp: R + WS - 1 is 4 full rings
    static constexpr int TH = kWarps * R;
    static constexpr int ROWS = TH + 2 * HALF;
    static constexpr int NV = (PX + 2 * HALF + 3) / 4 * 4;   // floats a lane reads per row
    static constexpr int PITCH = TW - PX + NV;
    static constexpr int WORDS = TW / 32;
    static constexpr int LIST = 1024;
    static constexpr int SMEM = ROWS * PITCH * 4 + TH * WORDS * 4 + LIST * 2 + 16;
};

template <int WS>
__global__ void __launch_bounds__(32 * kWarps) k_glrt_fast(const uint16_t *frames, Glrt p, int tiles_x, int tiles,
                                                           uint32_t *mask, unsigned long long *total)
{
    using FT = FastTile<WS>;
    constexpr int PX = FT::PX, HALF = FT::HALF;
    extern __shared__ __align__(16) float tile[];
    uint32_t *open_bits = reinterpret_cast<uint32_t *>(tile + FT::ROWS * FT::PITCH);   // undecided pixels
    uint16_t *list = reinterpret_cast<uint16_t *>(open_bits + FT::TH * FT::WORDS);
    int *n_list = reinterpret_cast<int *>(list + FT::LIST);
    const int f = blockIdx.x / tiles, t = blockIdx.x - f * tiles;
    const int tx0 = (t % tiles_x) * FT::TW, ty0 = (t / tiles_x) * FT::TH;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint16_t *fr = frames + (size_t)f * p.n_rows * p.n_cols;
    // c: a low pixel value of the tile (background is what most windows hold)
    __shared__ unsigned c_min;
    if (tid == 0) {
        c_min = 65535u;
        *n_list = 0;
    }
    for (int k = tid; k < FT::TH * FT::WORDS; k += 32 * kWarps) open_bits[k] = 0;
    __syncthreads();
    {
        const int xx = min(tx0 + (int)(((unsigned)tid * 37u) % FT::TW), p.n_rows - 1);
        const int yy = min(ty0 + (int)(((unsigned)tid * 53u) % FT::TH), p.n_cols - 1);
        const unsigned v = __reduce_min_sync(kFull, (unsigned)fr[xx + (size_t)yy * p.n_rows]);
        if (lane == 0) atomicMin(&c_min, v);
    }
    __syncthreads();
    const int c = (int)c_min;
    unsigned sum = 0;
    // all loads of two rows before the first store: with one load at a time the
    // tile's memory latencies were a third of the kernel (500 frames of 512 x 512:
    // search 1.26 -> 0.81 ms; four rows at a time measure the same)
    constexpr int NX = (FT::PITCH + 31) / 32, NR = 2;
    for (int tr = warp * NR; tr < FT::ROWS; tr += kWarps * NR) {
        uint16_t px[NR][NX];
#pragma unroll
        for (int u = 0; u < NR; ++u) {
            const uint16_t *rp = fr + (size_t)min(max(ty0 - HALF + tr + u, 0), p.n_cols - 1) * p.n_rows;
#pragma unroll
            for (int n = 0; n < NX; ++n) px[u][n] = rp[min(max(tx0 - HALF + lane + 32 * n, 0), p.n_rows - 1)];
        }
#pragma unroll
        for (int u = 0; u < NR; ++u) {
            const int ty = tr + u, yy = ty0 - HALF + ty;
            if (ty >= FT::ROWS) break;
            const bool row_ok = yy >= 0 && yy < p.n_cols;
            const bool inner = ty >= HALF && ty < HALF + FT::TH;
#pragma unroll
            for (int n = 0; n < NX; ++n) {
                const int tx = lane + 32 * n, xx = tx0 - HALF + tx;
                const bool ok = row_ok && xx >= 0 && xx < p.n_rows;
                if (tx < FT::PITCH) tile[ty * FT::PITCH + tx] = ok ? (float)((int)px[u][n] - c) : 0.f;
                if (ok && inner && tx >= HALF && tx < HALF + FT::TW) sum += px[u][n];
            }
        }
    }
    add_total(sum, &total[f]);
    __syncthreads();

    // the pixels that the reference tests
    const int xs = p.n_rows - (p.n_rows % 2), ys = p.n_cols - (p.n_cols % 2);
    const bool frame_ok = xs >= WS + 2 && ys >= WS + 2;
    const int x0 = tx0 + PX * lane;
    unsigned xmask = 0;
#pragma unroll
    for (int q = 0; q < PX; ++q)
        if (x0 + q >= HALF + 1 && x0 + q < xs - HALF) xmask |= 1u << q;
    float rc[WS][PX], r1[WS][PX], r2[WS][PX];
    const int yb = warp * FT::R;
#pragma unroll 1
    for (int base = 0; base < FT::R + WS - 1; base += WS) {
        if (ty0 + yb + base >= p.n_cols + WS) break;
#pragma unroll
        for (int k = 0; k < WS; ++k) {
            // row sums of tile row yb + base + k into ring slot k
            float v[FT::NV];
            const float *src = tile + (yb + base + k) * FT::PITCH + PX * lane;
            if constexpr (PX == 4) {
#pragma unroll
                for (int q = 0; q < FT::NV / 4; ++q) {
                    const float4 w = reinterpret_cast<const float4 *>(src)[q];
                    v[4 * q] = w.x;
                    v[4 * q + 1] = w.y;
                    v[4 * q + 2] = w.z;
                    v[4 * q + 3] = w.w;
                }
            } else {
#pragma unroll
                for (int q = 0; q < FT::NV / 2; ++q) {
                    const float2 w = reinterpret_cast<const float2 *>(src)[q];
                    v[2 * q] = w.x;
                    v[2 * q + 1] = w.y;
                }
            }
            // the taps that all PX windows share are summed once
            float m1 = 0.f, m2 = 0.f;
            float sq[PX + 2 * HALF];
#pragma unroll
            for (int q = 0; q < PX + 2 * HALF; ++q) sq[q] = v[q] * v[q];
            constexpr int A = PX - 1, B = WS;   // shared taps: [A, B)
#pragma unroll
            for (int q = 0; q < WS + PX; ++q)
                if (q >= A && q < B) {
                    m1 += v[q];
                    m2 += sq[q];
                }
#pragma unroll
            for (int o = 0; o < PX; ++o) {
                float s1 = m1, s2 = m2, cv = 0.f;
#pragma unroll
                for (int a = 0; a < WS; ++a) {
                    cv = fmaf(p.g1[a], v[o + a], cv);
                    if (A < B ? (o + a < A || o + a >= B) : true) {
                        s1 += v[o + a];
                        s2 += sq[o + a];
                    }
                }
                rc[k][o] = cv;
                r1[k][o] = s1;
                r2[k][o] = s2;
            }
            // ring slots k + 1 .. k + WS (mod WS) are the window's rows in order
            const int yo = base + k - (WS - 1);
            if (yo < 0) continue;
            const int y = ty0 + yb + yo;
            unsigned in_bits = 0, un_bits = 0;
            if (y < p.n_cols) {
                const bool y_ok = frame_ok && y >= HALF + 1 && y < ys - HALF;
#pragma unroll
                for (int o = 0; o < PX; ++o) {
                    float s1 = 0.f, s2 = 0.f, cv = 0.f;
#pragma unroll
                    for (int b = 0; b < WS; ++b) {
                        const int slot = (k + 1 + b) % WS;
                        cv = fmaf(p.g1[b], rc[slot][o], cv);
                        s1 += r1[slot][o];
                        s2 += r2[slot][o];
                    }
                    const float cz = fmaf(-p.mean, s1, cv);
                    const float null_h = fmaf(-s1 * p.inv_n, s1, s2);
                    const float den = null_h * p.fsumsq, num = cz * cz;
                    const bool sound = null_h >= 16.f && s2 <= 256.f * null_h && num <= p.sat * den;
                    const bool out = s2 == 0.f || (sound && num < p.lo * den);
                    const bool in = sound && num > p.hi * den;
                    if (in) in_bits |= 1u << o;
                    if (!in && !out) un_bits |= 1u << o;
                }
                in_bits = y_ok ? in_bits & xmask : 0u;
                un_bits = y_ok ? un_bits & xmask : 0u;
            }
            // pack: 32 / PX lanes make one mask word
            constexpr int G = 32 / PX;
            unsigned word = in_bits << (PX * (lane % G));
#pragma unroll
            for (int o = 1; o < G; o <<= 1) word |= __shfl_xor_sync(kFull, word, o);
            if (lane % G == 0 && y < p.n_cols && x0 < p.n_rows)
                mask[((size_t)f * p.n_cols + y) * p.words + x0 / 32] = word;
            if (un_bits) atomicOr(&open_bits[(yb + yo) * FT::WORDS + lane / G], un_bits << (PX * (lane % G)));
        }
    }
    __syncthreads();
    // undecided pixels: the reference sequence, one pixel per thread
    for (int w = tid; w < FT::TH * FT::WORDS; w += 32 * kWarps) {
        uint32_t bits = open_bits[w];
        while (bits) {
            const int b = __ffs(bits) - 1;
            bits &= bits - 1;
            const int at = atomicAdd(n_list, 1);
            if (at < FT::LIST) list[at] = (uint16_t)((w / FT::WORDS) * FT::TW + (w % FT::WORDS) * 32 + b);
        }
    }
    __syncthreads();
    const int n_open = *n_list;
    const bool listed = n_open <= FT::LIST;   // else walk the tile
    const int n_walk = listed ? n_open : FT::TH * FT::TW;
    for (int k = tid; k < n_walk; k += 32 * kWarps) {
        const int at = listed ? list[k] : k;
        const int ly = at / FT::TW, lx = at - ly * FT::TW;
        if (!listed && !((open_bits[ly * FT::WORDS + lx / 32] >> (lx % 32)) & 1u)) continue;
        const float *src = tile + ly * FT::PITCH + lx;
        if (glrt_exact(p, WS, [&](int a, int b) { return (int)src[b * FT::PITCH + a] + c; }))
            atomicOr(&mask[((size_t)f * p.n_cols + ty0 + ly) * p.words + (tx0 + lx) / 32], 1u << ((tx0 + lx) % 32));
    }
}

// Any other window side: the reference sequence on every pixel.
constexpr int kTX = 32, kTY = 8;
__global__ void k_glrt_any(const uint16_t *frames, Glrt p, int ws, int tiles_x, int tiles, uint32_t *mask,
                           unsigned long long *total)
{
    extern __shared__ uint16_t stage[];
    const int half = ws / 2;
    const int f = blockIdx.x / tiles, t = blockIdx.x - f * tiles;
    const int tx0 = (t % tiles_x) * kTX, ty0 = (t / tiles_x) * kTY;
    const int tw = kTX + 2 * half, th = kTY + 2 * half;
    const uint16_t *fr = frames + (size_t)f * p.n_rows * p.n_cols;
    const int tid = threadIdx.y * kTX + threadIdx.x;
    for (int k = tid; k < tw * th; k += kTX * kTY) {
        const int yy = ty0 - half + k / tw, xx = tx0 - half + k % tw;
        stage[k] = (xx >= 0 && xx < p.n_rows && yy >= 0 && yy < p.n_cols) ? fr[xx + (size_t)yy * p.n_rows] : 0;
    }
    __syncthreads();
    const int x = tx0 + threadIdx.x, y = ty0 + threadIdx.y;
    bool in = false;
    unsigned v = 0;
    if (x < p.n_rows && y < p.n_cols) {
        v = stage[(threadIdx.y + half) * tw + threadIdx.x + half];
        const int xs = p.n_rows - (p.n_rows % 2), ys = p.n_cols - (p.n_cols % 2);
        if (xs >= ws + 2 && ys >= ws + 2 && y >= half + 1 && y < ys - half && x >= half + 1 && x < xs - half)
            in = glrt_exact(p, ws, [&](int a, int b) { return (int)stage[(threadIdx.y + b) * tw + threadIdx.x + a]; });
    }
    const unsigned word = __ballot_sync(kFull, in);
    if (threadIdx.x == 0 && y < p.n_cols) mask[((size_t)f * p.n_cols + y) * p.words + tx0 / 32] = word;
    add_total(v, &total[f]);
}

// (labels change under other threads' atomics: read past the first-level cache)
__device__ __forceinline__ int find_root(const volatile int *L, int x)
{
    int n = 0;
    int y = L[x];
    while (y != x && n < kLinkLimit) {
        x = y;
        y = L[x];
        ++n;
    }
    return x;
}

// link two runs' components; roots always keep the smaller index
__device__ void unite(int *L, int a, int b, unsigned long long *err)
{
    for (int n = 0; n < kLinkLimit; ++n) {
        a = find_root(L, a);
        b = find_root(L, b);
        if (a == b) return;
        if (a < b) {
            const int old = atomicMin(&L[b], a);
            if (old == b) return;
            b = old;
        } else {
            const int old = atomicMin(&L[a], b);
            if (old == a) return;
            a = old;
        }
    }
    atomicExch(err, 1ull);
}

// counters of one chunk
enum { C_RUNS = 0, C_PARTS = 1, C_ERR = 2, C_TOTAL = 3, C_N = 4 };

struct Group {
    const uint16_t *frames;
    const uint32_t *mask;
    int n_rows, n_cols, words, frame0;
    const unsigned long long *total;   // pixel total per frame
    int *runs;                         // global run table (start, end, label, rank), 4 x run_cap
    long long run_cap, part_cap;
    unsigned long long *sums;          // 4 x part_cap: x, y, pixels, brightest
    loc_candidate *cands;              // particles in order of the frames' arrival
    int *fbase, *fcount;               // first particle and number of particles of each frame
    unsigned long long *ctr;
};

// inclusive block scan of one value per thread; *sum: the block's total
__device__ __forceinline__ unsigned block_scan(unsigned v, unsigned *warp_tot, unsigned *sum)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();   // the previous scan's totals have been read
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    unsigned before = 0, all = 0;
    for (int w = 0; w < nw; ++w) {
        const unsigned t = warp_tot[w];
        before += w < wid ? t : 0;
        all += t;
    }
    *sum = all;
    return x + before;
}

// One block per frame: runs of mask pixels in raster order, their components,
// and one record per component. The run table lives in shared memory while
// the frame has at most kRunsSm runs (a 512 x 512 frame of 1000 emitters has
// about 6000), else in global memory. This replaces four passes over a label
// and a mask array of 5 to 9 bytes a pixel and a per-frame scan of all pixels.
constexpr int kRunsSm = 6144;
__global__ void __launch_bounds__(512, 2) k_group(Group a)
{
    extern __shared__ int sm_runs[];
    __shared__ unsigned warp_tot[32];
    __shared__ long long run_base, part_base;
    __shared__ unsigned long long m_sum, m_cnt;
    const int f = blockIdx.x, tid = threadIdx.x, T = blockDim.x;
    const int nw = a.n_cols * a.words;
    const uint32_t *mask = a.mask + (size_t)f * nw;
    const uint16_t *fr = a.frames + (size_t)f * a.n_rows * a.n_cols;
    if (tid == 0) m_sum = m_cnt = 0;
    auto edges = [&](int w, uint32_t &starts, uint32_t &ends) {
        const uint32_t m = mask[w];
        starts = ends = 0;
        if (m) {
            const int col = w % a.words;
            const uint32_t prev = col > 0 ? mask[w - 1] >> 31 : 0u;
            const uint32_t next = col + 1 < a.words ? mask[w + 1] & 1u : 0u;
            starts = m & ~((m << 1) | prev);
            ends = m & ~((m >> 1) | (next << 31));
        }
    };
    // how many runs, and where they go
    unsigned cnt = 0;
    for (int w = tid; w < nw; w += T) {
        uint32_t st, en;
        edges(w, st, en);
        cnt += __popc(st);
    }
    unsigned n_runs_u;
    block_scan(cnt, warp_tot, &n_runs_u);
    const int n_runs = (int)n_runs_u;
    const bool in_sm = n_runs <= kRunsSm;
    if (tid == 0) run_base = in_sm ? 0 : (long long)atomicAdd(&a.ctr[C_RUNS], (unsigned long long)n_runs);
    __syncthreads();
    if (!in_sm && run_base + n_runs > a.run_cap) {   // the host grows the table and runs the chunk again
        if (tid == 0) {
            a.fbase[f] = 0;
            a.fcount[f] = 0;
        }
        return;
    }
    int *rs = in_sm ? sm_runs : a.runs + run_base;
    const long long pitch = in_sm ? kRunsSm : a.run_cap;
    int *re = rs + pitch, *lab = re + pitch, *rank = lab + pitch;
    const volatile int *vlab = lab;
    unsigned sdone = 0, edone = 0;
    for (int w0 = 0; w0 < nw; w0 += T) {
        const int w = w0 + tid;
        uint32_t st = 0, en = 0;
        if (w < nw) edges(w, st, en);
        // at most 16 starts and ends a word: both counts in one scan
        unsigned all;
        const unsigned mine = (unsigned)__popc(st) | ((unsigned)__popc(en) << 16);
        const unsigned inc = block_scan(mine, warp_tot, &all) - mine;
        if (st | en) {
            const int px0 = (w / a.words) * a.n_rows + (w % a.words) * 32;
            unsigned si = sdone + (inc & 0xffffu), ei = edone + (inc >> 16);
            while (st) {
                rs[si++] = px0 + __ffs(st) - 1;
                st &= st - 1;
            }
            while (en) {
                re[ei++] = px0 + __ffs(en) - 1;
                en &= en - 1;
            }
        }
        sdone += all & 0xffffu;
        edone += all >> 16;
    }
    for (int i = tid; i < n_runs; i += T) lab[i] = i;
    __syncthreads();
    // link every run to the runs of the row above that touch it (8-neighbourhood)
    for (int i = tid; i < n_runs; i += T) {
        const int s = rs[i], e = re[i], row0 = s / a.n_rows * a.n_rows;
        if (row0 == 0) continue;
        const int lo = max(s - a.n_rows - 1, row0 - a.n_rows), hi = min(e - a.n_rows + 1, row0 - 1);
        int l = 0, h = i;   // first run whose end is at or after lo
        while (l < h) {
            const int m = (l + h) >> 1;
            if (re[m] < lo) l = m + 1;
            else h = m;
        }
        for (; l < i && rs[l] <= hi; ++l) unite(lab, i, l, &a.ctr[C_ERR]);
    }
    __syncthreads();
    // a run's root is final now; roots in raster order are the particles
    unsigned np = 0;
    for (int i0 = 0; i0 < n_runs; i0 += T) {
        const int i = i0 + tid;
        const bool root = i < n_runs && vlab[i] == i;
        unsigned all;
        const unsigned inc = block_scan(root ? 1u : 0u, warp_tot, &all);
        if (root) rank[i] = (int)(np + inc - 1);
        np += all;
    }
    if (tid == 0) {
        part_base = (long long)atomicAdd(&a.ctr[C_PARTS], (unsigned long long)np);
        const bool fits = part_base + np <= a.part_cap;
        a.fbase[f] = fits ? (int)part_base : 0;
        a.fcount[f] = fits ? (int)np : 0;
    }
    __syncthreads();
    if (part_base + np > a.part_cap) return;
    unsigned long long *sx = a.sums + part_base, *sy = sx + a.part_cap, *sc = sy + a.part_cap, *mx = sc + a.part_cap;
    for (unsigned i = tid; i < np; i += T) sx[i] = sy[i] = sc[i] = mx[i] = 0;
    __threadfence();
    __syncthreads();
    unsigned long long msum = 0, mcnt = 0;
    for (int i = tid; i < n_runs; i += T) {
        const int s = rs[i], e = re[i], id = rank[find_root(lab, i)];
        const int y = s / a.n_rows, xa = s - y * a.n_rows, len = e - s + 1;
        unsigned peak = 0;
        for (int q = s; q <= e; ++q) {
            const unsigned v = fr[q];
            msum += v;
            peak = max(peak, v);
        }
        mcnt += len;
        atomicAdd(&sx[id], (unsigned long long)len * (2 * (unsigned long long)xa + len - 1) / 2);
        atomicAdd(&sy[id], (unsigned long long)len * y);
        atomicAdd(&sc[id], (unsigned long long)len);
        atomicMax(&mx[id], (unsigned long long)peak);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        msum += __shfl_xor_sync(kFull, msum, o);
        mcnt += __shfl_xor_sync(kFull, mcnt, o);
    }
    if ((tid & 31) == 0 && mcnt) {
        atomicAdd(&m_sum, msum);
        atomicAdd(&m_cnt, mcnt);
    }
    __threadfence();
    __syncthreads();
    const double bg = __ddiv_rn((double)(a.total[f] - m_sum),
                                (double)((unsigned long long)a.n_rows * a.n_cols - m_cnt));
    for (unsigned i = tid; i < np; i += T) {
        loc_candidate c;
        const double n = (double)__ldcg(&sc[i]);
        c.x = __ddiv_rn((double)__ldcg(&sx[i]), n);
        c.y = __ddiv_rn((double)__ldcg(&sy[i]), n);
        c.intensity = __dsub_rn((double)__ldcg(&mx[i]), bg);
        c.background = bg;
        c.frame = a.frame0 + f;
        c.half_width = 0;
        a.cands[part_base + i] = c;
    }
}

// output offset of each frame's particles (one block), and their total
__global__ void __launch_bounds__(1024) k_offsets(const int *fcount, int nf, long long *foff, unsigned long long *ctr)
{
    __shared__ unsigned warp_tot[32];
    long long run = 0;
    for (int f0 = 0; f0 < nf; f0 += blockDim.x) {
        const int f = f0 + threadIdx.x;
        const unsigned v = f < nf ? (unsigned)fcount[f] : 0u;
        unsigned all;
        const unsigned inc = block_scan(v, warp_tot, &all);
        if (f < nf) foff[f] = run + inc - v;
        run += all;
    }
    if (threadIdx.x == 0) ctr[C_TOTAL] = (unsigned long long)run;
}

// particles into frame order, 8 bytes per thread
__global__ void k_place(const loc_candidate *cands, const int *fbase, const int *fcount, const long long *foff,
                        loc_candidate *out, long long out_base, long long max_out)
{
    constexpr int W = sizeof(loc_candidate) / 8;
    static_assert(sizeof(loc_candidate) % 8 == 0, "moved in 8-byte words");
    const int f = blockIdx.x;
    const long long to = out_base + foff[f];
    const long long n = min((long long)fcount[f], max_out - to);
    const unsigned long long *src = reinterpret_cast<const unsigned long long *>(cands + fbase[f]);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(out + to);
    for (long long k = threadIdx.x; k < n * W; k += blockDim.x) dst[k] = src[k];
}

struct Buf {
    void *p = nullptr;
    size_t cap = 0;
    cudaError_t ensure(size_t n)
    {
        if (n <= cap) return cudaSuccess;
        release();
        cudaError_t e = cudaMalloc(&p, n);
        if (e == cudaSuccess) cap = n;
        return e;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    }
    ~Buf() { release(); }
};

// Working arrays, one set per host thread, kept between calls (a call blocks
// until its kernels are done, so no stream still uses them afterwards).
struct Scratch {
    int dev = -1;
    Buf mask, win, head, runs, sums, cands, all;
    long long run_cap = 0, part_cap = 0;
    void release()
    {
        for (Buf *b : {&mask, &win, &head, &runs, &sums, &cands, &all}) b->release();
        run_cap = part_cap = 0;
    }
    // the arrays whose size depends on what is found
    cudaError_t grow(long long n_runs, long long n_parts)
    {
        cudaError_t e = cudaSuccess;
        if (n_runs > run_cap) {
            run_cap = 0;
            if ((e = runs.ensure((size_t)n_runs * 16)) != cudaSuccess) return e;
            run_cap = n_runs;
        }
        if (n_parts > part_cap) {
            part_cap = 0;
            if ((e = sums.ensure((size_t)n_parts * 32)) != cudaSuccess) return e;
            if ((e = cands.ensure((size_t)n_parts * sizeof(loc_candidate))) != cudaSuccess) return e;
            part_cap = n_parts;
        }
        return e;
    }
};
// what a thread keeps between calls
constexpr size_t kKeepBytes = 512ull << 20;

long fail(int code, const std::string &m) { return locb::record_error_fixed(code, m.c_str()); }

size_t al256(size_t b) { return (b + 255) / 256 * 256; }

template <int WS>
cudaError_t launch_fast(const uint16_t *fr, const Glrt &p, int nf, uint32_t *mask, unsigned long long *total,
                        cudaStream_t st)
{
    using FT = FastTile<WS>;
    const int tx = (p.n_rows + FT::TW - 1) / FT::TW, ty = (p.n_cols + FT::TH - 1) / FT::TH;
    const cudaError_t e =
        cudaFuncSetAttribute(k_glrt_fast<WS>, cudaFuncAttributeMaxDynamicSharedMemorySize, FT::SMEM);
    if (e != cudaSuccess) return e;
    k_glrt_fast<WS><<<(unsigned)nf * tx * ty, 32 * kWarps, FT::SMEM, st>>>(fr, p, tx, tx * ty, mask, total);
    return cudaGetLastError();
}

// Window sides 3 to 13 (PSF widths up to 3.25 px) have the filtered kernel;
// wider windows would need a register ring of more than 78 floats a lane.
cudaError_t launch_glrt(const uint16_t *fr, const Glrt &p, int ws, int nf, uint32_t *mask, unsigned long long *total,
                        cudaStream_t st)
{
    switch (ws) {
    case 3: return launch_fast<3>(fr, p, nf, mask, total, st);
    case 5: return launch_fast<5>(fr, p, nf, mask, total, st);
    case 7: return launch_fast<7>(fr, p, nf, mask, total, st);
    case 9: return launch_fast<9>(fr, p, nf, mask, total, st);
    case 11: return launch_fast<11>(fr, p, nf, mask, total, st);
    case 13: return launch_fast<13>(fr, p, nf, mask, total, st);
    default: break;
    }
    const int half = ws / 2;
    const int tx = (p.n_rows + kTX - 1) / kTX, ty = (p.n_cols + kTY - 1) / kTY;
    const size_t smem = (size_t)(kTX + 2 * half) * (kTY + 2 * half) * sizeof(uint16_t);
    k_glrt_any<<<(unsigned)nf * tx * ty, dim3(kTX, kTY), smem, st>>>(fr, p, ws, tx, tx * ty, mask, total);
    return cudaGetLastError();
}

// loc_find_candidates (alloc NULL: at most max_cands candidates into d_cands)
// and loc_find_candidates_alloc (one buffer of the exact size from alloc).
long find(const uint16_t *d_frames, int n_frames, int n_rows, int n_cols, double pfa, double psf_width,
          loc_candidate *d_cands, long max_cands, loc_alloc_fn alloc, void *user, cudaStream_t st)
{
    if (!d_frames || n_frames < 0 || n_rows <= 0 || n_cols <= 0 || !(psf_width > 0) || max_cands < 0 ||
        (max_cands > 0 && !d_cands))
        return fail(LOC_E_INVALID, "bad argument");
    int ws = (int)std::ceil(4 * psf_width);
    if (ws % 2 == 0) ws += 1;
    if (ws > kMaxWin) return fail(LOC_E_UNSUPPORTED, "PSF width too large for the GPU finder (window > 33)");
    if (n_frames == 0) return 0;
    // window as the host finder computes it (Segmentation.cpp:241-430)
    const int half = ws / 2;
    const double npix = (double)ws * (double)ws;
    std::vector<double> g((size_t)ws * ws);
    double sum = 0.0, gg = 0.0;
    for (int j = -half; j <= half; ++j)
        for (int i = -half; i <= half; ++i) {
            const double v = 1.0 / (1.77245385 * psf_width) *
                             std::exp(-1.0 / (2.0 * psf_width * psf_width) * ((double)i * i + (double)j * j));
            g[(i + half) + (j + half) * ws] = v;
            sum += v;
            gg += v * v;
        }
    sum /= npix;
    double sumsq = 0.0;
    for (auto &v : g) {
        v -= sum;
        sumsq += v * v;
    }
    const double thr = 1.0 - std::exp(-pfa / npix);
    const long long frame_px = (long long)n_rows * n_cols;
    if (frame_px > (1ll << 30)) return fail(LOC_E_UNSUPPORTED, "frame too large");

    Glrt p{};
    p.n_rows = n_rows;
    p.n_cols = n_cols;
    p.words = (n_rows + 31) / 32;
    p.npix = npix;
    p.sumsq = sumsq;
    p.thr = thr;
    if (ws <= 13) {
        for (int i = -half; i <= half; ++i)
            p.g1[i + half] = (float)(std::sqrt(1.0 / (1.77245385 * psf_width)) *
                                     std::exp(-1.0 / (2.0 * psf_width * psf_width) * ((double)i * i)));
        p.mean = (float)sum;
        p.inv_n = (float)(1.0 / npix);
        p.fsumsq = (float)sumsq;
        // margin of the FP32 estimate (see k_glrt_fast): four times the bound
        // on the correlation, relative to sqrt(sumsq null), where S <= 256 null;
        // 1e-3 relative covers null_h (2^-24 x 256 x (2 ws + 4): 4.6e-4 at ws
        // = 13) and the reference sequence's own FP64 rounding where null >= 16
        const double u = std::ldexp(1.0, -24);
        const double eps = 4.0 * 16.0 * u * ((2 * ws + 2) * std::sqrt(gg / sumsq) + 2.0 * sum * ws / std::sqrt(sumsq));
        const double margin = 2.0 * std::sqrt(std::max(thr, 0.0)) * eps + eps * eps + 1e-3 * std::max(thr, 0.0);
        p.hi = (float)(thr + margin);
        p.lo = (float)(thr - margin);
        p.sat = 0.99f;
    }

    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return fail(LOC_E_CUDA, "finder device");
    static thread_local Scratch s;
    if (s.dev != dev) {
        s.release();
        s.dev = dev;
    }
    // chunk of frames with at most 2^27 pixels (16 MB of mask)
    const int chunk = (int)std::max(1ll, std::min<long long>(n_frames, (1ll << 27) / frame_px));
    const size_t mask_bytes = (size_t)chunk * n_cols * p.words * 4;
    // head: counters, then pixel total, output offset, first particle and particle count of each frame
    const size_t h_total = al256(C_N * 8), h_off = h_total + al256((size_t)chunk * 8),
                 h_base = h_off + al256((size_t)chunk * 8), h_count = h_base + al256((size_t)chunk * 4),
                 h_bytes = h_count + al256((size_t)chunk * 4);
    if ((e = s.mask.ensure(mask_bytes)) != cudaSuccess || (e = s.win.ensure(kMaxWin * kMaxWin * 8)) != cudaSuccess ||
        (e = s.head.ensure(h_bytes)) != cudaSuccess ||
        (e = s.grow(1, std::max(1024ll, (long long)chunk * frame_px / 128))) != cudaSuccess)
        return fail(LOC_E_NOMEM, std::string("finder scratch: ") + cudaGetErrorString(e));
    if ((e = cudaMemcpyAsync(s.win.p, g.data(), g.size() * 8, cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return fail(LOC_E_CUDA, std::string("window upload: ") + cudaGetErrorString(e));
    p.g = (const double *)s.win.p;
    char *head = (char *)s.head.p;
    unsigned long long *ctr = (unsigned long long *)head, *ftotal = (unsigned long long *)(head + h_total);
    long long *foff = (long long *)(head + h_off);
    int *fbase = (int *)(head + h_base), *fcount = (int *)(head + h_count);
    uint32_t *mask = (uint32_t *)s.mask.p;
    const int words = n_cols * p.words;
    const int threads = words >= 1024 ? 512 : 128;
    const int run_smem = kRunsSm * 16;
    if ((e = cudaFuncSetAttribute(k_group, cudaFuncAttributeMaxDynamicSharedMemorySize, run_smem)) != cudaSuccess)
        return fail(LOC_E_CUDA, std::string("finder: ") + cudaGetErrorString(e));
    const bool one_chunk = chunk >= n_frames;
    long long total = 0;
    for (int f0 = 0; f0 < n_frames; f0 += chunk) {
        const int nf = std::min(chunk, n_frames - f0);
        const uint16_t *fr = d_frames + (size_t)f0 * frame_px;
        cudaMemsetAsync(head, 0, h_off, st);   // counters and pixel totals
        if ((e = launch_glrt(fr, p, ws, nf, mask, ftotal, st)) != cudaSuccess)
            return fail(LOC_E_CUDA, std::string("finder launch: ") + cudaGetErrorString(e));
        unsigned long long h[C_N];
        for (int tries = 0;; ++tries) {
            if (tries) cudaMemsetAsync(ctr, 0, C_N * 8, st);
            const Group a{fr, mask, n_rows, n_cols, p.words, f0, ftotal, (int *)s.runs.p, s.run_cap, s.part_cap,
                          (unsigned long long *)s.sums.p, (loc_candidate *)s.cands.p, fbase, fcount, ctr};
            k_group<<<nf, threads, run_smem, st>>>(a);
            k_offsets<<<1, 1024, 0, st>>>(fcount, nf, foff, ctr);
            if ((e = cudaGetLastError()) != cudaSuccess ||
                (e = cudaMemcpyAsync(h, ctr, sizeof h, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
                (e = cudaStreamSynchronize(st)) != cudaSuccess)
                return fail(LOC_E_CUDA, std::string("finder: ") + cudaGetErrorString(e));
            if (h[C_ERR]) return fail(LOC_E_CUDA, "finder: component linking did not settle");
            if ((long long)h[C_RUNS] <= s.run_cap && (long long)h[C_PARTS] <= s.part_cap) break;
            // more runs or particles than the tables hold: group this chunk's
            // mask again with larger ones (frames without room for their runs
            // have not counted their particles yet, so this can happen twice)
            if (tries >= 3) return fail(LOC_E_CUDA, "finder: tables did not settle");
            if ((e = s.grow((long long)h[C_RUNS], (long long)h[C_PARTS])) != cudaSuccess)
                return fail(LOC_E_NOMEM, std::string("finder particles: ") + cudaGetErrorString(e));
        }
        const long long np = (long long)h[C_TOTAL];
        loc_candidate *out = d_cands;
        long long at = total, room = max_cands;
        if (alloc) {
            room = total + np;
            if (one_chunk) {
                out = np > 0 ? (loc_candidate *)alloc(user, np) : nullptr;
                if (np > 0 && !out) return fail(LOC_E_NOMEM, "finder: the caller's allocator gave no buffer");
            } else {
                // several chunks: collected here, handed over at the end
                if (s.all.cap < (size_t)room * sizeof(loc_candidate)) {
                    Buf more;
                    if ((e = more.ensure((size_t)room * 2 * sizeof(loc_candidate))) != cudaSuccess)
                        return fail(LOC_E_NOMEM, std::string("finder particles: ") + cudaGetErrorString(e));
                    if (total > 0)
                        cudaMemcpyAsync(more.p, s.all.p, (size_t)total * sizeof(loc_candidate),
                                        cudaMemcpyDeviceToDevice, st);
                    cudaStreamSynchronize(st);
                    std::swap(more.p, s.all.p);
                    std::swap(more.cap, s.all.cap);
                }
                out = (loc_candidate *)s.all.p;
            }
        }
        if (np > 0 && out && at < room)
            k_place<<<nf, 128, 0, st>>>((const loc_candidate *)s.cands.p, fbase, fcount, foff, out, at, room);
        total += np;
        if ((e = cudaGetLastError()) != cudaSuccess)
            return fail(LOC_E_CUDA, std::string("finder launch: ") + cudaGetErrorString(e));
    }
    if (alloc && !one_chunk && total > 0) {
        void *out = alloc(user, total);
        if (!out) return fail(LOC_E_NOMEM, "finder: the caller's allocator gave no buffer");
        cudaMemcpyAsync(out, s.all.p, (size_t)total * sizeof(loc_candidate), cudaMemcpyDeviceToDevice, st);
    }
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess)
        return fail(LOC_E_CUDA, std::string("finder: ") + cudaGetErrorString(e));
    size_t kept = 0;
    for (Buf *b : {&s.mask, &s.head, &s.runs, &s.sums, &s.cands, &s.all}) kept += b->cap;
    if (kept > kKeepBytes) s.release();
    return (long)total;
}

}  // namespace

extern "C" LOC_API long loc_find_candidates(const uint16_t *d_frames, int n_frames, int n_rows, int n_cols,
                                            double pfa, double psf_width, loc_candidate *d_cands, long max_cands,
                                            void *stream)
{
    return find(d_frames, n_frames, n_rows, n_cols, pfa, psf_width, d_cands, max_cands, nullptr, nullptr,
                (cudaStream_t)stream);
}

extern "C" LOC_API long loc_find_candidates_alloc(const uint16_t *d_frames, int n_frames, int n_rows, int n_cols,
                                                  double pfa, double psf_width, loc_alloc_fn alloc, void *user,
                                                  void *stream)
{
    if (!alloc) return fail(LOC_E_INVALID, "no allocator");
    return find(d_frames, n_frames, n_rows, n_cols, pfa, psf_width, nullptr, 0, alloc, user, (cudaStream_t)stream);
}
