// build_index.cu -- the CSR inverted index built on the device.
//
// Same result as build_host_index (host_index.cc): for every dim, a stable
// counting sort of the column by value, so ids ascend inside each (dim,value)
// list -- the layout of inv_list::invert + inv_table::build
// (table/inv_list.cc:295-320, table/inv_table.cu:267-350), which the reference
// runs single-threaded on the host with a copy of every list.
//
// Steps (values uploaded once, row-major n x d), one launch each for all dims:
//   k_bounds      per-dim min / max
//   (host)        key_base from the ranges (one list per value in [min,max])
//   k_columns     column-major 16-bit copy of value - min (shared-memory tiles)
//   k_hist        histogram of every chunk of a column
//   k_offsets     per dim: exclusive sums over the chunks (each chunk's start
//                 inside a list) and over the lists (key_off)
//   k_place       dims of few values: a chunk is sorted in shared memory (each
//                 warp ranks its run with match_any, 32 objects at a time, on
//                 counters of its own) and written list by list, in runs
//   k_place_wide  dims of more values, whose lists get a few ids a chunk: a
//                 warp takes a chunk in order and writes every id where it belongs
// A dim whose value range exceeds kMaxBins falls back to the host builder.
// The column is read twice and written once, the ids written once; 1,000,000 x
// 128 byte values take 1.1 ms on the device (0.7 of them placing), against 15.1 ms with a launch a
// dim for every step, a serial chain over the chunks per value and a 55-step
// sort of every 1,024 objects.
#include "capi_internal.h"

#include <algorithm>

namespace gg {
namespace {

constexpr int kMaxBins = 16384;       // values per dim the device path supports
constexpr int kFewBins = 1024;        // values per dim sorted in shared memory
constexpr int kPlaceWarps = 8;
constexpr int kWarpRun = 1024;        // objects of a chunk one warp ranks
constexpr int kChunk = kPlaceWarps * kWarpRun;
constexpr int kWideChunk = 32768;     // least objects of a chunk of a dim of many values
constexpr int kWideChunks = 128;      // most chunks of such a dim
constexpr int kHistThreads = 512;
static_assert(kChunk <= 8192, "a sorted entry holds its object in 13 bits");

// What the kernels need of a dim.
struct DimPlan {
    int32_t min, bins, chunks;
    int64_t key0;         // first list
    int64_t hist;         // first histogram word: chunk c, value v at hist + c * bins + v
    int64_t chunk;        // objects of a chunk
};

// min / max of 32 dims (blockIdx.x) over a slice of the rows
__global__ void __launch_bounds__(256) k_bounds(const int32_t *__restrict__ in, int64_t n, int32_t d, int32_t *mn, int32_t *mx) {
    __shared__ int32_t lo_s[8][32], hi_s[8][32];
    const int32_t c = (int32_t)blockIdx.x * 32 + threadIdx.x;
    int32_t lo = INT32_MAX, hi = INT32_MIN;
    if (c < d) {
#pragma unroll 4
        for (int64_t r = (int64_t)blockIdx.y * 8 + threadIdx.y; r < n; r += (int64_t)gridDim.y * 8) {
            const int32_t v = __ldg(in + r * d + c);
            lo = min(lo, v);
            hi = max(hi, v);
        }
    }
    lo_s[threadIdx.y][threadIdx.x] = lo;
    hi_s[threadIdx.y][threadIdx.x] = hi;
    __syncthreads();
    if (threadIdx.y == 0 && c < d) {
        for (int y = 1; y < 8; ++y) {
            lo = min(lo, lo_s[y][threadIdx.x]);
            hi = max(hi, hi_s[y][threadIdx.x]);
        }
        atomicMin(&mn[c], lo);
        atomicMax(&mx[c], hi);
    }
}

// out[c][r] = in[r][c] - min[c]: 64 rows x 32 dims a block
__global__ void __launch_bounds__(256) k_columns(const int32_t *__restrict__ in, const DimPlan *__restrict__ plan, int64_t n,
                                                 int32_t d, int32_t tiles_d, uint16_t *__restrict__ out) {
    __shared__ uint16_t tile[32][66];
    const int64_t r0 = (int64_t)(blockIdx.x / tiles_d) * 64;
    const int32_t c0 = (int32_t)(blockIdx.x % tiles_d) * 32;
    const int32_t x = threadIdx.x & 31, y = threadIdx.x >> 5;
    if (c0 + x < d) {
        const int32_t mn = plan[c0 + x].min;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int64_t r = r0 + y + 8 * k;
            if (r < n) tile[x][y + 8 * k] = (uint16_t)(__ldg(in + r * d + c0 + x) - mn);
        }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int32_t c = c0 + y + 8 * k;
        if (c >= d) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int64_t r = r0 + x + 32 * h;
            if (r < n) out[(int64_t)c * n + r] = tile[y + 8 * k][x + 32 * h];
        }
    }
}

// histogram of chunk blockIdx.x / d of dim blockIdx.x % d
__global__ void __launch_bounds__(kHistThreads) k_hist(const uint16_t *__restrict__ col, const DimPlan *__restrict__ plan, int64_t n,
                                                       int32_t d, uint32_t *__restrict__ H) {
    extern __shared__ uint32_t h[];
    const int32_t j = (int32_t)(blockIdx.x % (uint32_t)d);
    const int64_t c = blockIdx.x / (uint32_t)d;
    const DimPlan p = plan[j];
    if (c >= p.chunks) return;
    for (int v = threadIdx.x; v < p.bins; v += blockDim.x) h[v] = 0;
    __syncthreads();
    const int64_t i1 = min(n, (c + 1) * p.chunk);
    const uint16_t *x = col + (int64_t)j * n;
#pragma unroll 4
    for (int64_t i = c * p.chunk + threadIdx.x; i < i1; i += blockDim.x) atomicAdd(&h[__ldg(x + i)], 1u);
    __syncthreads();
    uint32_t *out = H + p.hist + c * p.bins;
    for (int v = threadIdx.x; v < p.bins; v += blockDim.x) out[v] = h[v];
}

// one dim a block: H becomes the exclusive sums over its chunks, key_off[key0
// + v] = j n + the exclusive sum of the lists' lengths
__global__ void __launch_bounds__(1024) k_offsets(uint32_t *__restrict__ H, const DimPlan *__restrict__ plan, int64_t n,
                                                  int64_t *__restrict__ key_off) {
    __shared__ int64_t warp_sum[33];
    const DimPlan p = plan[blockIdx.x];
    int64_t carry = (int64_t)blockIdx.x * n;
    for (int32_t b0 = 0; b0 < p.bins; b0 += 1024) {
        const int32_t v = b0 + threadIdx.x;
        uint32_t total = 0;
        if (v < p.bins) {
            uint32_t *h = H + p.hist + v;
            for (int32_t c0 = 0; c0 < p.chunks; c0 += 8) {
                uint32_t x[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) x[k] = c0 + k < p.chunks ? h[(int64_t)(c0 + k) * p.bins] : 0u;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    if (c0 + k < p.chunks) h[(int64_t)(c0 + k) * p.bins] = total;
                    total += x[k];
                }
            }
        }
        int64_t incl = total;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if ((threadIdx.x & 31) >= (unsigned)o) incl += y;
        }
        __syncthreads();
        if ((threadIdx.x & 31) == 31) warp_sum[threadIdx.x >> 5] = incl;
        __syncthreads();
        if (threadIdx.x < 32) {
            const int64_t w = warp_sum[threadIdx.x];
            int64_t wi = w;
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t y = __shfl_up_sync(0xffffffffu, wi, o);
                if (threadIdx.x >= (unsigned)o) wi += y;
            }
            warp_sum[threadIdx.x] = wi - w;
            if (threadIdx.x == 31) warp_sum[32] = wi;
        }
        __syncthreads();
        if (v < p.bins) key_off[p.key0 + v] = carry + warp_sum[threadIdx.x >> 5] + incl - total;
        carry += warp_sum[32];
    }
}

// Lanes of `active` holding the same value as this one, and this lane's rank among them.
__device__ __forceinline__ uint32_t rank_among(uint32_t active, uint32_t v, uint32_t &peers) {
    peers = __match_any_sync(active, v);
    return (uint32_t)__popc(peers & ((1u << (threadIdx.x & 31)) - 1u));
}

// Chunk blockIdx.x / d of dim blockIdx.x % d (at most kFewBins values) into its lists.
__global__ void __launch_bounds__(kPlaceWarps * 32, 4) k_place(const uint16_t *__restrict__ col, const DimPlan *__restrict__ plan,
                                                            int64_t n, int32_t d, const uint32_t *__restrict__ H,
                                                            const int64_t *__restrict__ key_off, uint32_t *__restrict__ ids) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t warp_sum[kPlaceWarps];
    const int32_t j = (int32_t)(blockIdx.x % (uint32_t)d);
    const int64_t c = blockIdx.x / (uint32_t)d;
    const DimPlan p = plan[j];
    if (p.bins > kFewBins || c >= p.chunks) return;
    const uint32_t bins = (uint32_t)p.bins, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    int64_t *dst = (int64_t *)smem;                              // [bins] where the chunk's ids of a list go, less its first slot
    uint32_t *sorted = (uint32_t *)(dst + bins);                 // [kChunk] value << 13 | object, in list order
    uint32_t *cnt = sorted + kChunk;                             // [warps][bins] counts, then next slots
    for (uint32_t i = tid; i < bins * kPlaceWarps; i += blockDim.x) cnt[i] = 0;
    const int64_t i0 = c * kChunk;
    const uint32_t len = (uint32_t)min((int64_t)kChunk, n - i0);
    const uint16_t *x = col + (int64_t)j * n + i0;
    // the warp's run: 32 rounds of 32 objects, two values a register
    uint32_t val[kWarpRun / 64];
#pragma unroll
    for (int r = 0; r < kWarpRun / 64; ++r) {
        const uint32_t a = w * kWarpRun + 64 * r + lane;
        val[r] = (a < len ? (uint32_t)__ldg(x + a) : 0u) | (a + 32 < len ? (uint32_t)__ldg(x + a + 32) : 0u) << 16;
    }
    __syncthreads();
    uint32_t *mine = cnt + w * bins;
#pragma unroll
    for (int r = 0; r < kWarpRun / 32; ++r) {
        const uint32_t a = w * kWarpRun + 32 * r + lane, v = (val[r / 2] >> (16 * (r & 1))) & 0xFFFFu;
        if (a < len) atomicAdd(&mine[v], 1u);
    }
    __syncthreads();
    // slots: list by list, in a list warp by warp
    uint32_t carry = 0;
    for (uint32_t b0 = 0; b0 < bins; b0 += kPlaceWarps * 32) {
        const uint32_t v = b0 + tid;
        uint32_t sum = 0;
        if (v < bins)
            for (int k = 0; k < kPlaceWarps; ++k) sum += cnt[k * bins + v];
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (lane == 31) warp_sum[w] = incl;
        __syncthreads();
        uint32_t before = carry, all = 0;
        for (uint32_t k = 0; k < kPlaceWarps; ++k) {
            if (k < w) before += warp_sum[k];
            all += warp_sum[k];
        }
        carry += all;
        if (v < bins) {
            uint32_t at = before + incl - sum;
            dst[v] = key_off[p.key0 + v] + H[p.hist + c * p.bins + v] - at;
            for (int k = 0; k < kPlaceWarps; ++k) {
                const uint32_t m = cnt[k * bins + v];
                cnt[k * bins + v] = at;
                at += m;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < kWarpRun / 32; ++r) {
        const uint32_t a = w * kWarpRun + 32 * r + lane, v = (val[r / 2] >> (16 * (r & 1))) & 0xFFFFu;
        const uint32_t active = __ballot_sync(0xffffffffu, a < len);
        if (a < len) {
            uint32_t peers;
            const uint32_t rank = rank_among(active, v, peers);
            const uint32_t at = mine[v];
            sorted[at + rank] = v << 13 | a;
            __syncwarp(active);
            if (rank == 0) mine[v] = at + (uint32_t)__popc(peers);
        }
        __syncwarp();
    }
    __syncthreads();
    for (uint32_t i = tid; i < len; i += blockDim.x) {
        const uint32_t e = sorted[i];
        ids[dst[e >> 13] + i] = (uint32_t)i0 + (e & 8191u);
    }
}

// The same for a dim of more values: one warp a chunk, in order.
__global__ void __launch_bounds__(32) k_place_wide(const uint16_t *__restrict__ col, const DimPlan *__restrict__ plan, int64_t n,
                                                   int32_t d, const uint32_t *__restrict__ H,
                                                   const int64_t *__restrict__ key_off, uint32_t *__restrict__ ids) {
    extern __shared__ uint32_t next[];         // [bins] next slot of a list, from the dim's first
    const int32_t j = (int32_t)(blockIdx.x % (uint32_t)d);
    const int64_t c = blockIdx.x / (uint32_t)d;
    const DimPlan p = plan[j];
    if (p.bins <= kFewBins || c >= p.chunks) return;
    const uint32_t lane = threadIdx.x;
    for (int32_t v = lane; v < p.bins; v += 32)
        next[v] = (uint32_t)(key_off[p.key0 + v] - (int64_t)j * n) + H[p.hist + c * p.bins + v];
    __syncwarp();
    const int64_t i0 = c * p.chunk, i1 = min(n, i0 + p.chunk);
    const uint16_t *x = col + (int64_t)j * n;
    uint32_t *out = ids + (int64_t)j * n;
    constexpr int R = 8;
    for (int64_t b = i0; b < i1; b += 32 * R) {
        uint32_t val[R];
#pragma unroll
        for (int r = 0; r < R; ++r) val[r] = b + 32 * r + lane < i1 ? (uint32_t)__ldg(x + b + 32 * r + lane) : 0u;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int64_t i = b + 32 * r + lane;
            const uint32_t active = __ballot_sync(0xffffffffu, i < i1);
            if (i < i1) {
                uint32_t peers;
                const uint32_t rank = rank_among(active, val[r], peers);
                const uint32_t at = next[val[r]];
                out[at + rank] = (uint32_t)i;
                __syncwarp(active);
                if (rank == 0) next[val[r]] = at + (uint32_t)__popc(peers);
            }
            __syncwarp();
        }
    }
}

}  // namespace

// Device build of a one-value-per-object index; false when a dim's value
// range is beyond kMaxBins (the caller then builds on the host).  Fills the
// host mirror (bounds, key offsets) and the device arrays of ix.
int build_device_index(const int32_t *values, int64_t n, int32_t d, genie_index *ix, bool *used) {
    *used = false;
    cudaError_t e = cudaSuccess;
    static thread_local int prepared_device = -1;
    int dev = 0;
    cudaGetDevice(&dev);
    const auto place_smem = [](int64_t bins) { return (size_t)bins * (8 + 4 * kPlaceWarps) + (size_t)kChunk * 4; };
    if (prepared_device != dev) {     // per-value shared counters of up to kMaxBins values
        if ((e = cudaFuncSetAttribute((const void *)k_hist, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBins * 4)) ||
            (e = cudaFuncSetAttribute((const void *)k_place_wide, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxBins * 4)) ||
            (e = cudaFuncSetAttribute((const void *)k_place, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)place_smem(kFewBins))))
            return cuda_fail(e, "device index build");
        prepared_device = dev;
    }
    const size_t cells = (size_t)n * d;
    int32_t *d_vals = nullptr, *d_bounds = nullptr;
    uint16_t *d_col = nullptr;
    DimPlan *d_plan = nullptr;
    uint32_t *d_H = nullptr;
    auto cleanup = [&] {
        cudaFree(d_vals);
        cudaFree(d_bounds);
        cudaFree(d_col);
        cudaFree(d_plan);
        cudaFree(d_H);
    };
    auto give_up = [&](const char *what) {
        cudaGetLastError();
        cleanup();
        return e == cudaErrorMemoryAllocation ? fail(GENIE_ERR_GPU_ALLOC, "device index build: out of memory")
                                              : cuda_fail(e, what);
    };
    if ((e = device_alloc((void **)&d_vals, cells * 4)) || (e = device_alloc((void **)&d_bounds, (size_t)d * 8)) ||
        (e = device_alloc((void **)&d_plan, (size_t)d * sizeof(DimPlan))))
        return give_up("device index build");
    std::vector<int32_t> bounds((size_t)d * 2, INT32_MAX);
    std::fill(bounds.begin() + d, bounds.end(), INT32_MIN);
    cudaMemcpy(d_vals, values, cells * 4, cudaMemcpyHostToDevice);
    cudaMemcpy(d_bounds, bounds.data(), (size_t)d * 8, cudaMemcpyHostToDevice);
    const unsigned tiles_d = (unsigned)((d + 31) / 32);
    const unsigned slices = (unsigned)std::min<int64_t>((n + 63) / 64, std::max<int64_t>(1, 152 * 16 / tiles_d));
    k_bounds<<<dim3(tiles_d, slices), dim3(32, 8)>>>(d_vals, n, d, d_bounds, d_bounds + d);
    if ((e = cudaMemcpy(bounds.data(), d_bounds, (size_t)d * 8, cudaMemcpyDeviceToHost))) return give_up("device index build");
    HostIndex &h = ix->host;
    h = HostIndex();
    h.n_objects = n;
    h.n_dims = d;
    h.mult_max = 1;
    h.whole = true;
    h.dim_min.assign(bounds.begin(), bounds.begin() + d);
    h.dim_max.assign(bounds.begin() + d, bounds.end());
    std::vector<DimPlan> plan((size_t)d);
    h.key_base.assign((size_t)d + 1, 0);
    int64_t hist = 0, most_chunks = 1, widest = 1, widest_few = 0, wide_chunks = 0;
    for (int32_t j = 0; j < d; ++j) {
        const int64_t bins = (int64_t)h.dim_max[j] - h.dim_min[j] + 1;
        if (bins > kMaxBins) {
            cleanup();
            return GENIE_OK;     // not used: the host builds this index
        }
        h.key_base[j + 1] = h.key_base[j] + bins;
        DimPlan &p = plan[(size_t)j];
        p.min = h.dim_min[j];
        p.bins = (int32_t)bins;
        p.key0 = h.key_base[j];
        p.hist = hist;
        p.chunk = bins <= kFewBins ? kChunk : std::max<int64_t>(kWideChunk, (n + kWideChunks - 1) / kWideChunks);
        p.chunks = (int32_t)((n + p.chunk - 1) / p.chunk);
        hist += bins * p.chunks;
        most_chunks = std::max<int64_t>(most_chunks, p.chunks);
        widest = std::max(widest, bins);
        if (bins <= kFewBins) widest_few = std::max(widest_few, bins);
        else wide_chunks = std::max<int64_t>(wide_chunks, p.chunks);
    }
    const int64_t tiles = ((n + 63) / 64) * (int64_t)tiles_d;
    if (most_chunks * d > (int64_t)0x7FFFFFFF || tiles > (int64_t)0x7FFFFFFF) {
        cleanup();
        return GENIE_OK;         // beyond a grid: the host builds this index
    }
    const int64_t nk = h.n_keys();
    if ((e = device_alloc((void **)&d_col, cells * 2)) || (e = device_alloc((void **)&d_H, (size_t)hist * 4)) ||
        (e = ix->d_key_off.reserve((size_t)(nk + 1) * 8)) ||
        (e = cudaMemcpy(d_plan, plan.data(), (size_t)d * sizeof(DimPlan), cudaMemcpyHostToDevice)))
        return give_up("device index build");
    k_columns<<<(unsigned)tiles, 256>>>(d_vals, d_plan, n, d, (int32_t)tiles_d, d_col);
    k_hist<<<(unsigned)(most_chunks * d), kHistThreads, (size_t)widest * 4>>>(d_col, d_plan, n, d, d_H);
    int64_t *d_keyoff = (int64_t *)ix->d_key_off.p;
    k_offsets<<<(unsigned)d, 1024>>>(d_H, d_plan, n, d_keyoff);
    // the values are in the columns: their room is the ids'
    cudaFree(d_vals);
    d_vals = nullptr;
    if ((e = ix->d_ids.reserve(cells * 4 + kIdsPadBytes))) return give_up("device index build");
    uint32_t *d_ids = (uint32_t *)ix->d_ids.p;
    cudaMemsetAsync(d_ids + cells, 0, kIdsPadBytes);
    if (widest_few)
        k_place<<<(unsigned)(most_chunks * d), kPlaceWarps * 32, place_smem(widest_few)>>>(d_col, d_plan, n, d, d_H, d_keyoff,
                                                                                          d_ids);
    if (wide_chunks)
        k_place_wide<<<(unsigned)(wide_chunks * d), 32, (size_t)widest * 4>>>(d_col, d_plan, n, d, d_H, d_keyoff, d_ids);
    const int64_t last = (int64_t)cells;
    cudaMemcpy(d_keyoff + nk, &last, 8, cudaMemcpyHostToDevice);
    e = cudaGetLastError();
    if (!e) e = cudaDeviceSynchronize();
    if (e) return give_up("device index build");
    cleanup();
    h.key_off.resize((size_t)nk + 1);
    if ((e = cudaMemcpy(h.key_off.data(), d_keyoff, (size_t)(nk + 1) * 8, cudaMemcpyDeviceToHost)))
        return cuda_fail(e, "device index build");
    *used = true;
    return GENIE_OK;
}

}  // namespace gg
