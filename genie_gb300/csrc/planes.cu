// planes.cu -- cumulative presence planes of a byte-valued index.
//
// For every (dim, value) of a table whose dims span at most 256 values, one
// bit per object: set when the object's value on that dim is at most the
// list's value.  An item [low, up] matches plane(up) & ~plane(low - 1), so a
// range costs two rows however many lists it covers (planes.cuh counts with
// them).  A plane row is n_objects / 8 bytes against 4 bytes a posting id, so
// the planes take (values per dim) / 32 times the ids' bytes: eight times for
// 256 values.  They are built when a quarter of the device memory that is free
// then holds all that is kept, once per index (note_search), and kept while it
// lives or until an allocation of this library finds the device full
// (give_back_planes).  The values themselves are kept too, one byte each, object by object (a 32nd of
// 256 planes): a weighted tile sums its few candidates from them, whose bytes
// of one object lie in one or two lines, where the planes would cost a line
// per item and candidate.
//
// Layout: tile by tile (kPlTile objects), in a tile one row of 16-byte vectors
// per key, so the rows that run together lie together (few pages at a time,
// and one tile's used rows fit L2), then an empty and a full row for the open
// ends.  The row of a dim's largest value (every object) is never read and not
// written.  Offsets in a tile are 32-bit bytes.
#include "capi_internal.h"

#include <algorithm>

namespace gg {
namespace {

constexpr int64_t kPlMaxValues = 256;
constexpr int kPlSubWords = 64;                          // words of a row one CTA builds (2,048 objects)
constexpr int kPlBuildThreads = 256;
constexpr size_t kPlColumnBytes = size_t(512) << 20;     // column bytes held at a time

// col[d][id] = value - dim_min of every object on dims [d0, d0 + nd) (one per
// blockIdx.y), from the posting lists.  A CTA fills kPlSpan objects of the
// column in shared memory: a thread searches each list's ids of that range,
// then warps take runs of 512 of them.  Bytes written straight to memory, one
// sector each, took 5.2 ms for 4,000,000 x 128; this takes 1.0.
constexpr uint32_t kPlSpan = 65536, kPlRun = 512;
constexpr int kPlColThreads = 512;
__global__ void __launch_bounds__(kPlColThreads) k_pl_columns(const uint32_t *__restrict__ ids, const int64_t *__restrict__ key_off,
                                                              const int64_t *__restrict__ key_base, int32_t d0, int64_t n,
                                                              uint8_t *__restrict__ col) {
    extern __shared__ __align__(16) uint8_t span[];      // [kPlSpan]
    __shared__ int64_t start[kPlMaxValues];
    __shared__ uint32_t len[kPlMaxValues], flat[kPlMaxValues + 1], tmp[48];
    const uint32_t tid = threadIdx.x, lane = lane_id();
    const int64_t kb = key_base[d0 + blockIdx.y];
    const uint32_t values = (uint32_t)(key_base[d0 + blockIdx.y + 1] - kb);
    const int64_t o0 = (int64_t)blockIdx.x * kPlSpan, o1 = min(n, o0 + (int64_t)kPlSpan);
    uint32_t runs = 0;
    if (tid < values) {
        const int64_t a = key_off[kb + tid], e = key_off[kb + tid + 1];
        const int64_t lo = lower_bound_u32(ids, a, e, (uint32_t)o0);
        const int64_t hi = o1 >= n ? e : lower_bound_u32(ids, lo, e, (uint32_t)o1);
        start[tid] = lo;
        len[tid] = (uint32_t)(hi - lo);
        runs = ((uint32_t)(hi - lo) + kPlRun - 1) / kPlRun;
    }
    uint32_t total = 0;
    const uint32_t at = block_excl_scan(runs, tmp, &total);
    if (tid < values) flat[tid] = at;
    if (tid == 0) flat[values] = total;
    __syncthreads();
    for (uint32_t f = warp_id(); f < total; f += kPlColThreads / 32) {
        uint32_t a = 0, b = values;       // last list with flat <= f: lists without runs share their successor's
        while (a + 1 < b) {
            const uint32_t mid = (a + b) >> 1;
            if (flat[mid] <= f) a = mid; else b = mid;
        }
        const uint32_t r0 = (f - flat[a]) * kPlRun, m = min(kPlRun, len[a] - r0);
        const uint32_t *p = ids + start[a] + r0;
        uint32_t x[kPlRun / 32];
#pragma unroll
        for (uint32_t r = 0; r < kPlRun / 32; ++r) x[r] = 32 * r + lane < m ? __ldg(p + 32 * r + lane) : 0u;
#pragma unroll
        for (uint32_t r = 0; r < kPlRun / 32; ++r)
            if (32 * r + lane < m) span[x[r] - (uint32_t)o0] = (uint8_t)a;
    }
    __syncthreads();
    uint8_t *out = col + (int64_t)blockIdx.y * n + o0;
    const uint32_t bytes = (uint32_t)(o1 - o0);
    if ((((uintptr_t)out) & 15u) == 0) {
        for (uint32_t i = tid; i < bytes / 16; i += kPlColThreads) ((uint4 *)out)[i] = ((const uint4 *)span)[i];
        for (uint32_t i = bytes / 16 * 16 + tid; i < bytes; i += kPlColThreads) out[i] = span[i];
    } else {
        for (uint32_t i = tid; i < bytes; i += kPlColThreads) out[i] = span[i];
    }
}

// One dim (blockIdx.y) of kPlSubWords * 32 objects (blockIdx.x): presence bits
// per value in shared memory, an OR over the values in order, rows out.  Eight
// threads share two words' values, so the running OR takes two passes.
__global__ void __launch_bounds__(kPlBuildThreads) k_pl_build(const uint8_t *__restrict__ col,
                                                              const int64_t *__restrict__ key_base, int32_t d0,
                                                              int64_t n, int64_t tile_words, uint32_t row_words,
                                                              uint32_t subs, uint32_t *__restrict__ planes) {
    extern __shared__ __align__(16) uint32_t eq[];      // [values][kPlSubWords]
    constexpr uint32_t kPairs = kPlSubWords / 2, kSegs = kPlBuildThreads / kPairs;
    __shared__ uint2 part[kSegs][kPairs];
    const int32_t d = d0 + blockIdx.y;
    const uint32_t values = (uint32_t)(key_base[d + 1] - key_base[d]);
    const uint64_t tile = blockIdx.x / subs;
    const uint32_t sub = (uint32_t)(blockIdx.x % subs);
    const int64_t o0 = (int64_t)tile * kPlTile + (int64_t)sub * kPlSubWords * 32;
    for (uint32_t i = threadIdx.x; i < values * kPlSubWords / 4; i += kPlBuildThreads) ((uint4 *)eq)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const uint8_t *c = col + (int64_t)blockIdx.y * n;
    for (int64_t i = threadIdx.x; i < kPlSubWords * 32; i += kPlBuildThreads)
        if (o0 + i < n) atomicOr(&eq[(uint32_t)c[o0 + i] * kPlSubWords + (uint32_t)(i >> 5)], 1u << (i & 31));
    __syncthreads();
    uint2 *eq2 = (uint2 *)eq;
    const uint32_t w = threadIdx.x % kPairs, seg = threadIdx.x / kPairs;
    const uint32_t per = (values + kSegs - 1) / kSegs;
    const uint32_t v0 = min(values, seg * per), v1 = min(values, v0 + per);
    uint2 acc = make_uint2(0, 0);
    for (uint32_t v = v0; v < v1; ++v) {
        const uint2 x = eq2[v * kPairs + w];
        acc.x |= x.x;
        acc.y |= x.y;
        eq2[v * kPairs + w] = acc;
    }
    part[seg][w] = acc;
    __syncthreads();
    uint2 before = make_uint2(0, 0);
    for (uint32_t g = 0; g < seg; ++g) {
        before.x |= part[g][w].x;
        before.y |= part[g][w].y;
    }
    const uint32_t word = sub * kPlSubWords + 2 * w;
    if (word >= row_words) return;             // row_words is a multiple of four
    uint2 *out = (uint2 *)(planes + tile * (uint64_t)tile_words + (uint64_t)key_base[d] * row_words + word);
    for (uint32_t v = v0; v < v1 && v + 1 < values; ++v) {
        const uint2 x = eq2[v * kPairs + w];
        out[(uint64_t)v * (row_words / 2)] = make_uint2(x.x | before.x, x.y | before.y);
    }
}

// The columns of dims [d0, d0 + nd) into the objects' rows (32 x 32 tiles through shared memory).
__global__ void k_pl_rows(const uint8_t *__restrict__ col, int32_t d0, int32_t nd, int64_t n, int32_t row,
                          uint8_t *__restrict__ vals) {
    __shared__ uint8_t tile[32][33];
    const int64_t o0 = (int64_t)blockIdx.x * 32;
    const int32_t c0 = (int32_t)blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += blockDim.y)
        if (c0 + y < nd && o0 + threadIdx.x < n) tile[y][threadIdx.x] = col[(int64_t)(c0 + y) * n + o0 + threadIdx.x];
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += blockDim.y)
        if (o0 + y < n && c0 + (int)threadIdx.x < nd) vals[(o0 + y) * row + d0 + c0 + threadIdx.x] = tile[threadIdx.x][y];
}

// The empty and the full row behind each tile's keys.
__global__ void k_pl_ends(uint4 *planes, int64_t tiles, int64_t keys, int64_t row_vec) {
    for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        uint4 *r = planes + (t * (keys + kPlExtraRows) + keys) * row_vec;
        for (int64_t i = threadIdx.x; i < row_vec; i += blockDim.x) {
            r[i] = make_uint4(0, 0, 0, 0);
            r[row_vec + i] = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
        }
    }
}

// Bytes of the index's planes; 0 when it has none.  Planes stand for one value
// per object and dim: an index from a file whose dims miss an object, list one
// twice, or hold lists outside their value range has none (k_pl_columns would
// leave a byte of a missing object unset, and k_pl_build index by it).
int64_t planes_bytes(const genie_index *ix) {
    const HostIndex &h = ix->host;
    const int64_t n = h.n_objects, nk = h.n_keys();
    if (!h.whole || ix->is_bag || ix->sub_shift >= 0 || ix->codec || n <= 0 || nk <= 0) return 0;
    for (int32_t j = 0; j < h.n_dims; ++j)
        if (h.key_base[j + 1] - h.key_base[j] > kPlMaxValues) return 0;
    const int64_t tiles = (n + kPlTile - 1) / kPlTile;
    const int64_t row_vec = tiles > 1 ? (int64_t)kPlTile / 128 : (n + 127) / 128, rows = nk + kPlExtraRows;
    if (rows * row_vec * 16 > (int64_t)0xFFFFFFFFll || tiles > (int64_t)0x7FFFFFFF) return 0;
    return tiles * rows * row_vec * 16;
}

// The indexes that have their planes.
std::mutex g_with_planes_mu;
std::vector<genie_index *> g_with_planes;

bool build(genie_index *ix) {
    const HostIndex &h = ix->host;
    const int64_t n = h.n_objects, nk = h.n_keys();
    const int64_t tiles = (n + kPlTile - 1) / kPlTile;
    const int64_t row_vec = tiles > 1 ? (int64_t)kPlTile / 128 : (n + 127) / 128, rows = nk + kPlExtraRows;
    const size_t bytes = (size_t)ix->pl_bytes.load();
    const int32_t dims_at_once = (int32_t)std::min<int64_t>(h.n_dims, std::max<int64_t>(1, (int64_t)kPlColumnBytes / n));
    const int32_t val_row = (h.n_dims + 15) & ~15;
    size_t free_b = 0, total_b = 0;
    if (cudaMemGetInfo(&free_b, &total_b)) {
        cudaGetLastError();
        return false;
    }
    const size_t val_bytes = (size_t)n * (size_t)val_row, col_bytes = (size_t)dims_at_once * (size_t)n;
    if (bytes + val_bytes > free_b / 4 || bytes + val_bytes + col_bytes > free_b / 2) return false;
    static_assert(kPlMaxValues * kPlSubWords * 4 == 65536, "shared presence bits");
    DevBuf col;
    cudaError_t e;
    if ((e = cudaFuncSetAttribute((const void *)k_pl_build, cudaFuncAttributeMaxDynamicSharedMemorySize, 65536)) ||
        (e = cudaFuncSetAttribute((const void *)k_pl_columns, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlSpan)) ||
        (e = cudaMalloc(&ix->d_planes.p, bytes)) ||
        (e = cudaMalloc(&ix->d_pl_vals.p, val_bytes)) || (e = cudaMalloc(&col.p, col_bytes))) {
        cudaGetLastError();
        ix->d_planes.release();
        ix->d_pl_vals.release();
        return false;
    }
    ix->d_planes.bytes = bytes;
    ix->d_pl_vals.bytes = val_bytes;
    const uint32_t subs = (uint32_t)((row_vec * 4 + kPlSubWords - 1) / kPlSubWords);
    for (int32_t d0 = 0; d0 < h.n_dims; d0 += dims_at_once) {
        const int32_t nd = std::min(dims_at_once, h.n_dims - d0);
        int64_t widest = 1;
        for (int32_t j = d0; j < d0 + nd; ++j) widest = std::max(widest, h.key_base[j + 1] - h.key_base[j]);
        for (int32_t j = 0; j < nd; j += 65535)
            k_pl_columns<<<dim3((unsigned)((n + kPlSpan - 1) / kPlSpan), (unsigned)std::min(65535, nd - j)), kPlColThreads, kPlSpan,
                           ix->stream>>>(ix->dev.ids, ix->dev.key_off, ix->dev.key_base, d0 + j, n,
                                         (uint8_t *)col.p + (int64_t)j * n);
        for (int32_t j = 0; j < nd; j += 32 * 65535)
            k_pl_rows<<<dim3((unsigned)((n + 31) / 32), (unsigned)((std::min(nd - j, 32 * 65535) + 31) / 32)), dim3(32, 8), 0,
                        ix->stream>>>((const uint8_t *)col.p + (int64_t)j * n, d0 + j, nd - j, n, val_row,
                                      (uint8_t *)ix->d_pl_vals.p);
        // grid y is at most 65,535 dims at once
        for (int32_t j = 0; j < nd; j += 65535)
            k_pl_build<<<dim3((unsigned)(tiles * subs), (unsigned)std::min(65535, nd - j)), kPlBuildThreads,
                         (size_t)widest * kPlSubWords * 4, ix->stream>>>(
                (const uint8_t *)col.p + (int64_t)j * n, ix->dev.key_base, d0 + j, n, rows * row_vec * 4,
                (uint32_t)(row_vec * 4), subs, (uint32_t *)ix->d_planes.p);
    }
    k_pl_ends<<<(unsigned)std::min<int64_t>(tiles, 65535), 128, 0, ix->stream>>>((uint4 *)ix->d_planes.p, tiles, nk,
                                                                                row_vec);
    e = cudaGetLastError();
    if (!e) e = cudaStreamSynchronize(ix->stream);
    cudaFree(col.p);
    if (e) {
        cudaGetLastError();
        ix->d_planes.release();
        ix->d_pl_vals.release();
        return false;
    }
    ix->pl_row_vec = row_vec;
    std::lock_guard<std::mutex> g(g_with_planes_mu);
    g_with_planes.push_back(ix);
    ++ix->pl_built;
    ix->pl_tiles = tiles;
    return true;
}

}  // namespace

// A launch in flight has its pointers already, so the device is waited for; a
// call that has a view but has not launched counts in pl_users; a batch's own
// graph is captured again without the planes (enqueue), one of a caller's
// cannot be, so those keep them.
bool give_back_planes() {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> g(g_with_planes_mu);
    bool any = false;
    for (size_t i = g_with_planes.size(); i-- > 0;) {
        genie_index *ix = g_with_planes[i];
        std::lock_guard<std::mutex> use(ix->pl_mu);
        if (ix->device != dev || ix->pl_users > 0 || ix->pl_held || cudaDeviceSynchronize()) continue;
        ix->d_planes.release();
        ix->d_pl_vals.release();
        ix->pl_touched = 0;
        ix->pl_tiles = 0;
        g_with_planes.erase(g_with_planes.begin() + (std::ptrdiff_t)i);
        any = true;
    }
    return any;
}

void forget_planes(genie_index *ix) {
    std::lock_guard<std::mutex> g(g_with_planes_mu);
    g_with_planes.erase(std::remove(g_with_planes.begin(), g_with_planes.end(), ix), g_with_planes.end());
}

PlanesUse::PlanesUse(genie_index *index) : ix(index) {
    std::lock_guard<std::mutex> g(ix->pl_mu);
    ++ix->pl_users;
}

PlanesUse::~PlanesUse() {
    std::lock_guard<std::mutex> g(ix->pl_mu);
    --ix->pl_users;
}

namespace {

// What a batch touches is told from at most 16 of its queries and 8 items of
// each (1 us): every item looked at took 3 us of a 130 us batch of 12 queries.
// One of every group, wherever in it, so that no pattern of the caller's falls
// in step with them.
struct Sample {
    int64_t n, step;
    Sample(int64_t size, int64_t most) : n(size), step(std::max<int64_t>(1, (size + most - 1) / most)) {}
    int64_t of(int64_t group) const { return std::min(step, n - group * step); }      // it stands for
    int64_t at(int64_t group) const { return group * step + (int64_t)((uint32_t)(group + 1) * 2654435761u >> 8) % of(group); }
};

int64_t sampled_ids(const HostIndex &h, const genie_queries *q, int64_t i) {
    const int64_t a = q->item_off[i];
    const Sample s(q->item_off[i + 1] - a, 8);
    int64_t total = 0;
    for (int64_t g = 0; g * s.step < s.n; ++g) {
        const int64_t j = a + s.at(g);
        int64_t s0 = 0, s1 = 0;
        if (item_span(h, q->dim[j], q->low[j], q->up[j], s0, s1)) total += (s1 - s0) * s.of(g);
    }
    return total;
}

}  // namespace

// Building the planes takes about as long as counting four times their bytes
// of posting ids without them (260,000 x 128, 1.1 GB of planes: build 1 ms,
// 2.5 GB of ids counted in 0.5 ms; 4,000,000 x 128, 17 GB: 8 ms, and 310 GB
// in 45 ms), so they are built when the index's searches have touched that
// much: a table searched once or twice never pays for them, and none pays more
// than about twice what it would have.  Past that point nothing is counted.
// Searches whose tuning keeps them off the planes do not count.
void note_search(genie_index *ix, const genie_queries *q, const Tuning &t) {
    if (!t.dense_bitmaps || ix->pl_bytes == 0 || ix->pl_tiles > 0) return;
    std::lock_guard<std::mutex> g(ix->dir_mu);
    if (ix->pl_bytes < 0) ix->pl_bytes = planes_bytes(ix);
    if (ix->pl_bytes == 0 || ix->pl_tiles > 0) return;
    const HostIndex &h = ix->host;
    const int64_t enough = ix->pl_bytes;       // ids, of four bytes
    const Sample s(q->n_queries, 16);
    for (int64_t g = 0; g * s.step < s.n && ix->pl_touched < enough; ++g)
        ix->pl_touched += sampled_ids(h, q, s.at(g)) * s.of(g);
    if (ix->pl_touched >= enough && !build(ix)) ix->pl_bytes = 0;
}

bool may_have_planes(genie_index *ix) {
    std::lock_guard<std::mutex> g(ix->dir_mu);
    if (ix->pl_bytes < 0) ix->pl_bytes = planes_bytes(ix);
    return ix->pl_bytes > 0;
}

PlanesPlan planes_plan(const genie_index *ix, const genie_queries *q) {
    PlanesPlan plan{kNeedLists, kRouteLists};
    if (ix->pl_bytes == 0) return plan;          // never any planes
    const HostIndex &h = ix->host;
    const auto takes = [&](int64_t i, bool &w, uint32_t &k, int64_t &m) {
        w = q->weighted && q->weight && q->weighted[i];
        k = q->k ? q->k[i] : q->uniform_k;
        m = q->item_off[i + 1] - q->item_off[i];
        return planes_take(m, q->item_off[i + 1], w, k, h.n_dims, h.n_objects);
    };
    bool w = false, others = false;              // others: queries that only the lists take
    uint32_t k = 0, kinds = 0;
    int64_t m = 0;
    for (int64_t i = 0; i < q->n_queries; ++i)
        if (takes(i, w, k, m)) kinds |= w ? kNeedPlanesWeighted : kNeedPlanes;
        else others = true;
    if (!kinds) return plan;
    plan.route = kRoutePlanes;
    // a table of one tile has planes no slower than its lists throughout, but for
    // the lists' kernels that other queries of the batch need (49 weighted
    // queries on 5,072 objects, half k = 10 and half 500: 180 us both ways, 160
    // on lists)
    if (h.n_objects > (int64_t)kPlTile || others) {
        int64_t planes = others ? kPlBothPs : 0, lists = 0, each = kPlBothPs;
        const Sample s(q->n_queries, 16);
        for (int64_t g = 0; g * s.step < s.n; ++g) {
            if (!takes(s.at(g), w, k, m)) continue;
            const PlanesCost cost(m, w, k, h.n_objects, q->n_queries);
            const int64_t l = cost.lists(sampled_ids(h, q, s.at(g)));
            planes += cost.planes * s.of(g);
            lists += l * s.of(g);
            each += std::min(cost.planes, l) * s.of(g);
        }
        if (lists < std::min(planes, each)) return plan = PlanesPlan{kNeedLists, kRouteLists};
        if (each < planes) plan.route = kRouteEach;
    }
    plan.need = kinds | (others || plan.route == kRouteEach ? (uint32_t)kNeedLists : 0u);
    return plan;
}

}  // namespace gg
