// Frame ingest: camera buffers of any of the reference's storage types
// (LocalizerStorageType, reference source/Defines.h:82-95) in row- or
// column-major order (BufferWithFormatToImage / CopyBufferToImage,
// source/FileIO.cpp:195-234, FileIO.h:96-116) into the fit path's uint16
// frame stack (x fastest). The reference widens every pixel to double; the
// fit path works on uint16, which holds every value of 8- and 16-bit unsigned
// cameras exactly. Other values are rounded to the nearest integer and
// clamped to [0, 65535]; the call returns how many pixels that changed, so a
// caller can tell a lossless ingest (0) from a lossy one.
//
// Column-major input is a streaming conversion; row-major input is
// transposed through 64 x 64 shared-memory tiles so that both the reads and
// the writes are coalesced. HBM-bound: element size + 2 bytes per pixel.
#include "../../include/localizer_b200.h"

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <string>
#include <type_traits>

namespace locb {
int record_error_fixed(int code, const char *msg);
}

namespace {

constexpr int kTile = 64;     // row-major transpose tile (64 x 64 pixels, 256 threads)

// types whose every value is a uint16
template <typename S> constexpr bool kExact = sizeof(S) <= 2 && !std::is_signed<S>::value;

template <typename S> __device__ __forceinline__ uint16_t to_u16(S v, unsigned &lossy)
{
    if constexpr (kExact<S>) {
        return (uint16_t)v;
    } else if constexpr (std::is_same<S, float>::value) {
        float r = rintf(v);
        r = r < 0.0f ? 0.0f : (r > 65535.0f ? 65535.0f : r);
        if (!(r == v)) ++lossy;   // rounded, clamped, or NaN (-> 0)
        return (uint16_t)(r == r ? r : 0.0f);
    } else {
        const double d = (double)v;
        double r = rint(d);
        r = r < 0.0 ? 0.0 : (r > 65535.0 ? 65535.0 : r);
        if (!(r == d)) ++lossy;
        return (uint16_t)(r == r ? r : 0.0);
    }
}

// V consecutive elements moved by one load or store (the host checks the
// alignment and the sizes before it picks V > 1)
template <typename T, int V> struct alignas(V * sizeof(T)) Vec {
    T v[V];
};

// one atomic per block: with one per warp a stack in which most pixels are
// rounded spent its time on this counter (500 float frames of 512 x 512, all rounded:
// 433 -> 163 us). Exact types have nothing to count and skip the block's waits
// (30 column-major uint16 frames of 2048 x 2048: 143 us with them, 126 us without)
template <typename S> __device__ __forceinline__ void count_lossy(unsigned lossy, unsigned long long *counter)
{
    if constexpr (kExact<S>) return;
    __shared__ unsigned block_lossy;
    if (threadIdx.x == 0) block_lossy = 0;
    __syncthreads();
    lossy = __reduce_add_sync(0xffffffffu, lossy);
    if ((threadIdx.x & 31) == 0 && lossy) atomicAdd(&block_lossy, lossy);
    __syncthreads();
    if (threadIdx.x == 0 && block_lossy) atomicAdd(counter, (unsigned long long)block_lossy);
}

// column-major: the same pixel order on both sides, V pixels per thread and trip
template <typename S, int V>
__global__ void k_ingest_cm(const S *src, uint16_t *dst, long long n, unsigned long long *lossy_count)
{
    unsigned lossy = 0;
    const long long nv = n / V;
    const Vec<S, V> *sv = reinterpret_cast<const Vec<S, V> *>(src);
    Vec<uint16_t, V> *dv = reinterpret_cast<Vec<uint16_t, V> *>(dst);
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < nv; p += (long long)gridDim.x * blockDim.x) {
        const Vec<S, V> x = sv[p];
        Vec<uint16_t, V> y;
#pragma unroll
        for (int k = 0; k < V; ++k) y.v[k] = to_u16<S>(x.v[k], lossy);
        dv[p] = y;
    }
    count_lossy<S>(lossy, lossy_count);
}

// row-major: frame buffer element (i, j) at i * n_cols + j -> pixel i + j * n_rows,
// through a 64 x 64 shared-memory tile so that reads (along j) and writes
// (along i) are both coalesced. All of a thread's loads are issued before the
// first conversion: one at a time left the memory latency in the open.

// Even n_rows and n_cols, aligned buffers: a thread reads pairs along j and
// writes pairs along i, a 64-pixel segment per warp and access (500 frames of
// 512 x 512: float 220 -> 163 us, uint16 199 -> 122 us; with the words of the
// kernel below float takes 189 us).
template <typename S>
__global__ void __launch_bounds__(256) k_ingest_rm_even(const S *src, uint16_t *dst, int n_rows, int n_cols,
                                                        unsigned long long *lossy_count)
{
    __shared__ uint16_t t[kTile][kTile + 1];
    const size_t fpx = (size_t)n_rows * n_cols;
    const S *fs = src + (size_t)blockIdx.z * fpx;
    uint16_t *fd = dst + (size_t)blockIdx.z * fpx;
    const int j0 = blockIdx.x * kTile, i0 = blockIdx.y * kTile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned lossy = 0;
    constexpr int N = kTile / 8;
    const int jr = j0 + 2 * lane;   // even, as is n_cols: jr < n_cols gives jr + 1 < n_cols
    const S *row = fs + min(jr, n_cols - 2);
    Vec<S, 2> x[N];
#pragma unroll
    for (int u = 0; u < N; ++u)
        x[u] = *reinterpret_cast<const Vec<S, 2> *>(row + (size_t)min(i0 + warp + 8 * u, n_rows - 1) * n_cols);
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const int di = warp + 8 * u;
        if (i0 + di < n_rows && jr < n_cols) {
            t[di][2 * lane] = to_u16<S>(x[u].v[0], lossy);
            t[di][2 * lane + 1] = to_u16<S>(x[u].v[1], lossy);
        }
    }
    __syncthreads();
    for (int dj = warp; dj < kTile; dj += 8) {
        const int j = j0 + dj, i = i0 + 2 * lane;
        if (j < n_cols && i < n_rows) {   // i even, n_rows even: i + 1 < n_rows
            Vec<uint16_t, 2> y;
            y.v[0] = t[2 * lane][dj];
            y.v[1] = t[2 * lane + 1][dj];
            *reinterpret_cast<Vec<uint16_t, 2> *>(fd + i + (size_t)j * n_rows) = y;
        }
    }
    count_lossy<S>(lossy, lossy_count);
}

// Any size and alignment: a thread reads the same columns of rows i and i + 1,
// whose pixels are neighbours in the output, and passes them on as one 32-bit
// word; with 16-bit words, four accesses a pixel, the load/store units set the
// time. Where an output row starts at an odd pixel the words are shifted by
// one between lanes (500 frames of 511 x 513: float 347 -> 228 us, uint8
// 275 -> 165 us).
template <typename S>
__global__ void __launch_bounds__(256) k_ingest_rm(const S *src, uint16_t *dst, int n_rows, int n_cols,
                                                   unsigned long long *lossy_count)
{
    constexpr int N = kTile / 16;                 // row pairs per thread, in two groups of columns
    __shared__ uint32_t t[kTile][kTile / 2 + 1];  // [j][pair of i]
    const size_t fpx = (size_t)n_rows * n_cols;
    const S *fs = src + (size_t)blockIdx.z * fpx;
    const int j0 = blockIdx.x * kTile, i0 = blockIdx.y * kTile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned lossy = 0;
    S x[N][2][2];
#pragma unroll
    for (int u = 0; u < N; ++u)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const S *row = fs + (size_t)min(i0 + 2 * (warp + 8 * u) + h, n_rows - 1) * n_cols;
#pragma unroll
            for (int g = 0; g < 2; ++g) x[u][h][g] = row[min(j0 + lane + 32 * g, n_cols - 1)];
        }
#pragma unroll
    for (int u = 0; u < N; ++u) {
        const int ip = warp + 8 * u;
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const int dj = lane + 32 * g;
            uint32_t w = 0;
            if (j0 + dj < n_cols) {
                if (i0 + 2 * ip < n_rows) w = to_u16<S>(x[u][0][g], lossy);
                if (i0 + 2 * ip + 1 < n_rows) w |= (uint32_t)to_u16<S>(x[u][1][g], lossy) << 16;
            }
            t[dj][ip] = w;
        }
    }
    __syncthreads();
    uint32_t out[kTile / 8];
#pragma unroll
    for (int u = 0; u < kTile / 8; ++u) out[u] = t[warp + 8 * u][lane];
#pragma unroll
    for (int u = 0; u < kTile / 8; ++u) {
        const int dj = warp + 8 * u;
        if (j0 + dj >= n_cols) break;
        uint16_t *to = dst + (size_t)blockIdx.z * fpx + (size_t)(j0 + dj) * n_rows + i0;
        const uint32_t w = out[u];
        const int left = n_rows - i0 - 2 * lane;   // pixels of the row from this lane's first on
        if ((reinterpret_cast<uintptr_t>(to) & 2) == 0) {
            if (left > 1) *reinterpret_cast<uint32_t *>(to + 2 * lane) = w;
            else if (left == 1) to[2 * lane] = (uint16_t)w;
        } else {
            const uint32_t next = __shfl_down_sync(0xffffffffu, w, 1);
            if (lane == 0) to[0] = (uint16_t)w;
            if (lane < 31 && left > 2) *reinterpret_cast<uint32_t *>(to + 2 * lane + 1) = w >> 16 | next << 16;
            else if (left > 1) to[2 * lane + 1] = (uint16_t)(w >> 16);
        }
    }
    count_lossy<S>(lossy, lossy_count);
}

template <typename S>
cudaError_t launch(const void *src, uint16_t *dst, int n_frames, int n_rows, int n_cols, int row_major,
                   unsigned long long *cnt, cudaStream_t st)
{
    const S *s = static_cast<const S *>(src);
    const uintptr_t sa = reinterpret_cast<uintptr_t>(src), da = reinterpret_cast<uintptr_t>(dst);
    if (!row_major) {
        const long long n = (long long)n_frames * n_rows * n_cols;
        const bool v4 = n % 4 == 0 && sa % (4 * sizeof(S)) == 0 && da % 8 == 0;
        const long long units = v4 ? n / 4 : n;
        const int blocks = (int)((units + 255) / 256 < 148 * 16 ? (units + 255) / 256 : 148 * 16);
        if (v4) k_ingest_cm<S, 4><<<blocks, 256, 0, st>>>(s, dst, n, cnt);
        else k_ingest_cm<S, 1><<<blocks, 256, 0, st>>>(s, dst, n, cnt);
    } else {
        const bool even = n_rows % 2 == 0 && n_cols % 2 == 0 && sa % (2 * sizeof(S)) == 0 && da % 4 == 0;
        dim3 grid((n_cols + kTile - 1) / kTile, (n_rows + kTile - 1) / kTile, n_frames);
        if (even) k_ingest_rm_even<S><<<grid, 256, 0, st>>>(s, dst, n_rows, n_cols, cnt);
        else k_ingest_rm<S><<<grid, 256, 0, st>>>(s, dst, n_rows, n_cols, cnt);
    }
    return cudaGetLastError();
}

}  // namespace

extern "C" LOC_API long long loc_ingest_frames(const void *d_src, int format, int n_frames, int n_rows, int n_cols,
                                               int row_major, uint16_t *d_dst, void *stream)
{
    if (!d_src || !d_dst || n_frames < 0 || n_rows <= 0 || n_cols <= 0)
        return locb::record_error_fixed(LOC_E_INVALID, "bad argument");
    if (n_frames > 65535 && row_major) return locb::record_error_fixed(LOC_E_UNSUPPORTED, "too many frames in one call");
    if (n_frames == 0) return 0;
    const cudaStream_t st = (cudaStream_t)stream;
    // one lossy counter per host thread and device, kept across calls (a
    // stream-ordered allocation per call would go back to the driver at every
    // synchronisation)
    struct Counter {
        unsigned long long *p = nullptr;
        int dev = -1;
        ~Counter()
        {
            if (p) cudaFree(p);
        }
    };
    static thread_local Counter counter;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess && counter.dev != dev) {
        if (counter.p) cudaFree(counter.p);
        counter.p = nullptr;
        counter.dev = -1;
        e = cudaMalloc((void **)&counter.p, sizeof(unsigned long long));
        if (e == cudaSuccess) counter.dev = dev;
    }
    if (e != cudaSuccess) return locb::record_error_fixed(LOC_E_NOMEM, "ingest counter");
    unsigned long long *cnt = counter.p;
    cudaMemsetAsync(cnt, 0, sizeof(unsigned long long), st);
    switch (format) {
    case 2: e = launch<int8_t>(d_src, d_dst, n_frames, n_rows, n_cols, row_major, cnt, st); break;
    case 3: e = launch<uint8_t>(d_src, d_dst, n_frames, n_rows, n_cols, row_major, cnt, st); break;
    case 4: e = launch<int16_t>(d_src, d_dst, n_frames, n_rows, n_cols, row_major, cnt, st); break;
    case 5: e = launch<uint16_t>(d_src, d_dst, n_frames, n_rows, n_cols, row_major, cnt, st); break;
    case 6: e = launch<int32_t>(d_src, d_dst, n_frames, n_rows, n_cols, row_major, cnt, st); break;
    case 7: e = launch<uint32_t>(d_src, d_dst, n_frames, n_rows, n_cols, row_major, cnt, st); break;
    case 8: e = launch<int64_t>(d_src, d_dst, n_frames, n_rows, n_cols, row_major, cnt, st); break;
    case 9: e = launch<uint64_t>(d_src, d_dst, n_frames, n_rows, n_cols, row_major, cnt, st); break;
    case 10: e = launch<float>(d_src, d_dst, n_frames, n_rows, n_cols, row_major, cnt, st); break;
    case 11: e = launch<double>(d_src, d_dst, n_frames, n_rows, n_cols, row_major, cnt, st); break;
    default:
        return locb::record_error_fixed(LOC_E_UNSUPPORTED, "unsupported storage format (4-bit types are not)");
    }
    unsigned long long h = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, cnt, sizeof h, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return locb::record_error_fixed(LOC_E_CUDA, (std::string("ingest: ") + cudaGetErrorString(e)).c_str());
    return (long long)h;
}
