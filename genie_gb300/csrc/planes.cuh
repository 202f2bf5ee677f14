// planes.cuh -- k_planes: match counting on byte-valued tables from
// cumulative presence planes, counts kept bit-sliced in registers.
//
// Reference counterpart: the per-query bitmap counter of match_AT
// (matching/match_device_utils.h:422-446, match.cu:43-464), one global atomic
// per posting id.  A table whose dims span at most 256 values keeps, for every
// (dim, value), a plane of one bit per object: set when the object's value is
// at most that value (planes.cu).  An item [low, up] then matches the objects
// of plane(up) & ~plane(low - 1), whatever the range's width, and a query's
// counts are the column sums of its items' words: a carry-save adder tree sums
// eight items' words into eight bit planes of the count, held in registers.
// No posting id is read, and there are no counters to clear, scan or add to
// with atomics.
//
// What bounds it: unweighted, reading two 2 KB row slices per (item, tile) from
// L2.  A tile is 16,384 objects (128 threads, one 16-byte vector each), and
// work is taken tile-major, every query's tile t before any query's tile t + 1,
// so the rows in use are those of one or two tiles (about 30 MB of 128 byte
// dims), which L2 serves at 14-20 TB/s; at 64 MB and more it gives 8-13 TB/s
// (random 4 KB rows, one kernel reading nothing else).  At 4,000,000 x 128,
// 1,024 queries of 8-128 items: 3.6 ms, 16 TB/s; the counter tiles (k_dense)
// took 13.0 ms for them, bound by a shared atomic per posting id.  Plain 16-byte
// loads, sixteen in flight a thread, are the fastest feed found: a producer
// warp with bulk copies of rows took 5.6-6.8 ms (about 140 cycles a copy),
// cp.async of 16 bytes a thread 11 ms.
//
// Weighted queries need 31-bit sums.  Bit-sliced they would cost 62 logic
// operations per item and word, so a tile first bounds every sum from above:
// items are sorted by weight, each group of eight (sixteen past kPlGroup8
// items) counts with its largest weight in units of 2^qshift, and since the
// groups descend the bound is
//   sum over groups of (unit weight of the group - of the next) * (count so far),
// bit-sliced additions of the count planes.  Objects whose bound reaches the
// query's lower bound (at 500,000 x 128, k = 100: 90 a tile on average) are
// summed exactly from the table's value bytes.  Logic operations bound it:
// 7.9 ms for 1,024 weighted queries at 4,000,000 x 128, 31.1 ms with 4-byte
// counter tiles; groups of sixteen throughout give twice the candidates and
// 9.7 ms, 63 units instead of 31 one more plane and no fewer candidates.
//
// Results of a tile (at most k keys) go to the query's region of the part
// scratch.  lbk[q], a lower bound on the query's final k-th key, prunes: a
// tile holding k objects raises it to its own k-th key, and a histogram of
// the primaries written so far bounds it as tiles finish.  k_planes_finish
// merges.  A region holds k keys of every tile while the batch's fit 512 MB; one
// that is too small (many ties, few bounds) makes it redo the query alone, tile
// by tile, compacting the region.  A table of one tile
// needs neither: its block writes the results.
#pragma once

namespace gg {

// Blocks per SM: unweighted, five (96 registers, spilled loads) take 3.75 ms for
// the batch above and six 3.99, four 3.60; weighted, three and four take the
// same 7.6 and five (102 registers) 13.1.
constexpr int kPlBlocks = 4;
constexpr uint32_t kPlThreads = 128;                   // threads that count: four warps
constexpr uint32_t kPlTileVec = kPlThreads;            // 16-byte vectors of a full tile's row
constexpr int kPlWSum = 11;                            // planes of a weighted bound
static_assert(kPlTileVec * 128 == kPlTile, "one vector of 128 objects per thread");
static_assert(kPlMaxItems <= 255 && (kPlMaxItems + 1) % 8 == 0, "eight count planes, whole groups");
constexpr uint32_t kPlManyExact = 64;                  // objects from which, and items up to which, an exact sum
constexpr uint32_t kPlManyItems = 48;                  // takes a thread an object instead of a warp four
constexpr uint32_t kPlCand = 1024;                     // exact keys a weighted tile holds at once
static_assert(kPlMaxWeightedK * 2 <= kPlCand, "k kept keys and as many new ones fit the candidate buffer");

// State of the tile being counted.
struct PlShared {
    uint32_t red[2][4];
    uint32_t tmp[48];
    uint64_t lbk;
    uint32_t n, last_id, tile;
    uint4 entry;
};
// What a weighted tile needs beside: exact keys, and the objects to sum.
struct PlExact {
    uint64_t cand[kPlCand];
    uint16_t obj[kPlCand];
};
// The keys of a table of one tile, which need no merge; before there are any,
// the counts that pl_join adds up, in 16-byte vectors.
struct PlKeys {
    alignas(16) uint64_t cand[kCandCap];
};
static_assert(alignof(PlKeys) % sizeof(uint4) == 0, "pl_join's vectors are aligned");
static_assert(sizeof(PlKeys::cand) >= 8 * kPlThreads * sizeof(uint4), "eight planes of every thread");
// A tile's keys in shared memory: exact keys of a weighted one, the result of
// an unweighted query of a table of one tile.
template <bool WEIGHTED>
struct PlScratch {
    using type = PlExact;
};
template <>
struct PlScratch<false> {
    using type = PlKeys;
};

// One query's items, as the tiles use them.
template <bool WEIGHTED>
struct PlItems {
    uint2 rows[kPlMaxItems + 1];       // byte offsets in a tile of the rows of low - 1 and up
    uint32_t inc[WEIGHTED ? kPlMaxItems + 1 : 1];
    uint32_t test[WEIGHTED ? kPlMaxItems + 1 : 1];      // dim << 16 | low << 8 | width of the exact sums
};

// Sum over the counting warps; s.red alternates so that one barrier per call is enough.
__device__ __forceinline__ uint32_t pl_block_sum(uint32_t v, PlShared &s, uint32_t &phase) {
    const uint32_t w = __reduce_add_sync(0xffffffffu, v);
    uint32_t *r = s.red[phase & 1u];
    ++phase;
    if (lane_id() == 0) r[warp_id()] = w;
    BlockGroup::sync();
    return r[0] + r[1] + r[2] + r[3];
}

__device__ __forceinline__ uint32_t pl_popc(const uint32_t (&m)[4]) {
    return __popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3]);
}

// Objects of m whose bit-sliced value is at least c.
template <int NP>
__device__ __forceinline__ void pl_keep_ge(const uint32_t (&p)[NP][4], uint32_t c, uint32_t (&m)[4]) {
    uint32_t gt[4] = {0, 0, 0, 0};
    const bool over = (c >> NP) != 0;
#pragma unroll
    for (int b = NP - 1; b >= 0; --b) {
        if ((c >> b) & 1u) {
#pragma unroll
            for (int w = 0; w < 4; ++w) m[w] &= p[b][w];
        } else {
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                gt[w] |= m[w] & p[b][w];
                m[w] &= ~p[b][w];
            }
        }
    }
#pragma unroll
    for (int w = 0; w < 4; ++w) m[w] = over ? 0u : m[w] | gt[w];
}

// The `need` largest of the objects m (need <= their number): gt receives
// those above the need-th value, m keeps the ones equal to it; returns how
// many of the latter belong, and the value.
template <int NP>
__device__ __forceinline__ uint32_t pl_kth(const uint32_t (&p)[NP][4], uint32_t (&m)[4], uint32_t need,
                                           uint32_t (&gt)[4], uint32_t &value, PlShared &s, uint32_t &phase) {
#pragma unroll
    for (int w = 0; w < 4; ++w) gt[w] = 0;
    value = 0;
#pragma unroll
    for (int b = NP - 1; b >= 0; --b) {
        uint32_t t[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) t[w] = m[w] & p[b][w];
        const uint32_t n = pl_block_sum(pl_popc(t), s, phase);
        if (n >= need) {
            value |= 1u << b;
#pragma unroll
            for (int w = 0; w < 4; ++w) m[w] = t[w];
        } else {
            need -= n;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                gt[w] |= t[w];
                m[w] &= ~t[w];
            }
        }
    }
    return need;
}

// Keep the first `take` of this thread's objects m in id order.
__device__ __forceinline__ void pl_first(uint32_t (&m)[4], uint32_t take) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const uint32_t c = __popc(m[w]);
        if (c > take) {
            uint32_t x = m[w], kept = 0;
            for (uint32_t i = 0; i < take; ++i) {
                const uint32_t low = x & (0u - x);
                kept |= low;
                x ^= low;
            }
            m[w] = kept;
            take = 0;
        } else {
            take -= c;
        }
    }
}

__device__ __forceinline__ uint4 pl_load(const unsigned char *tile, uint32_t off) {
    return __ldg((const uint4 *)(tile + off));
}

// s += c << B on bit planes.
template <int B>
__device__ __forceinline__ void pl_add_shifted(uint32_t (&s)[kPlWSum][4], const uint32_t (&c)[8][4]) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        uint32_t carry = 0;
#pragma unroll
        for (int j = B; j < kPlWSum; ++j) {
            const uint32_t a = s[j][w];
            if (j - B < 8) {
                const uint32_t b = c[j - B][w];
                s[j][w] = a ^ b ^ carry;
                carry = (a & b) | (a & carry) | (b & carry);
            } else {
                s[j][w] = a ^ carry;
                carry &= a;
            }
        }
    }
}

// Bit planes of this thread's 128 objects: counts and, weighted, the bound.
template <bool WEIGHTED>
struct PlCounts {
    uint32_t c[8][4];
    uint32_t sum[WEIGHTED ? kPlWSum : 1][4];
    uint32_t unit;         // unit weight of the weight group being counted

    static __device__ __forceinline__ void csa(uint32_t &s, uint32_t &cr, uint32_t a, uint32_t b, uint32_t d) {
        cr = (a & b) | (a & d) | (b & d);      // one logic operation each
        s = a ^ b ^ d;
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int w = 0; w < 4; ++w) c[j][w] = 0;
        if (WEIGHTED) {
#pragma unroll
            for (int j = 0; j < kPlWSum; ++j)
#pragma unroll
                for (int w = 0; w < 4; ++w) sum[j][w] = 0;
        }
    }
    // four items' words into planes 0 and 1; t4 takes the carry
    __device__ __forceinline__ void four(const uint4 (&lo)[4], const uint4 (&up)[4], uint32_t (&t4)[4]) {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            uint32_t m[4], a, b;
#pragma unroll
            for (int i = 0; i < 4; ++i) m[i] = (&up[i].x)[w] & ~(&lo[i].x)[w];
            csa(c[0][w], a, c[0][w], m[0], m[1]);
            csa(c[0][w], b, c[0][w], m[2], m[3]);
            csa(c[1][w], t4[w], c[1][w], a, b);
        }
    }
    // eight items' carries into plane 2; t8 takes the carry
    __device__ __forceinline__ void eight(const uint32_t (&a)[4], const uint32_t (&b)[4], uint32_t (&t8)[4]) {
#pragma unroll
        for (int w = 0; w < 4; ++w) csa(c[2][w], t8[w], c[2][w], a[w], b[w]);
    }
    // a carry of weight 2^J into planes J and up
    template <int J>
    __device__ __forceinline__ void ripple(const uint32_t (&t)[4]) {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            uint32_t carry = t[w];
#pragma unroll
            for (int j = J; j < 8; ++j) {
                const uint32_t x = c[j][w];
                c[j][w] = x ^ carry;
                carry &= x;
            }
        }
    }
    __device__ __forceinline__ void sixteen(const uint32_t (&a)[4], const uint32_t (&b)[4]) {
        uint32_t t16[4];
#pragma unroll
        for (int w = 0; w < 4; ++w) csa(c[3][w], t16[w], c[3][w], a[w], b[w]);
        ripple<4>(t16);
    }
    // a weight group is counted: the bound, up to the next group's unit weight
    __device__ __forceinline__ void bound(uint32_t next) {
        if constexpr (WEIGHTED) {
            const uint32_t d = unit - next;
            unit = next;
            // differences are small: digits of four, an addition each (two copies of the code, not five)
#pragma unroll 1
            for (uint32_t i = d & 3u; i > 0; --i) pl_add_shifted<0>(sum, c);
#pragma unroll 1
            for (uint32_t i = d >> 2; i > 0; --i) pl_add_shifted<2>(sum, c);
        }
    }
};

// The sums of the block's `groups` runs of `width` threads, each of which
// counted other items of the same objects, into the first run's planes.  buf
// holds a vector per plane and thread.
__device__ __forceinline__ void pl_join(PlCounts<false> &pc, uint32_t width, uint32_t groups, uint4 *buf) {
    const uint32_t g = threadIdx.x / width;
    for (uint32_t half = groups / 2; half > 0; half /= 2) {
        if (g >= half && g < 2 * half) {
#pragma unroll
            for (int b = 0; b < 8; ++b)
                buf[b * kPlThreads + threadIdx.x - half * width] = make_uint4(pc.c[b][0], pc.c[b][1], pc.c[b][2], pc.c[b][3]);
        }
        __syncthreads();
        if (g < half) {
            uint32_t carry[4] = {0, 0, 0, 0};
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const uint4 v = buf[b * kPlThreads + threadIdx.x];
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const uint32_t x = pc.c[b][w], y = (&v.x)[w], z = carry[w];
                    pc.c[b][w] = x ^ y ^ z;
                    carry[w] = (x & y) | (x & z) | (y & z);
                }
            }
        }
        __syncthreads();
    }
}

// Unit weight of the weight group starting at item u (0 past the last).
__device__ __forceinline__ uint32_t pl_unit(const PlItems<true> &it, uint32_t u, uint32_t n, int qshift) {
    return u < n ? (it.inc[u] + ((1u << qshift) - 1u)) >> qshift : 0u;
}

// Counts of one tile over the query's items.
template <bool WEIGHTED>
__device__ __forceinline__ void pl_count(const unsigned char *__restrict__ tile, uint32_t mine, uint32_t n,
                                         int qshift, const PlItems<WEIGHTED> &it, PlCounts<WEIGHTED> &pc,
                                         uint32_t first = 0) {
    pc.clear();
    if constexpr (WEIGHTED) pc.unit = pl_unit(it, 0, n, qshift);
    auto load = [&](uint32_t u, uint4 (&lo)[4], uint4 (&up)[4]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint2 r = it.rows[first + u + i];
            lo[i] = __ldg((const uint4 *)(tile + (r.x + mine)));
            up[i] = __ldg((const uint4 *)(tile + (r.y + mine)));
        }
    };
    uint4 lo0[4], up0[4], lo1[4], up1[4];
    auto eight = [&](uint32_t u, uint32_t (&t8)[4]) {
        uint32_t a[4], b[4];
        load(u, lo0, up0);
        load(u + 4, lo1, up1);
        pc.four(lo0, up0, a);
        pc.four(lo1, up1, b);
        pc.eight(a, b, t8);
    };
    const bool by8 = WEIGHTED && n <= kPlGroup8;
    uint32_t held[4] = {0, 0, 0, 0};
    bool half = false;             // held is the carry of the first eight of sixteen
#pragma unroll 1
    for (uint32_t u0 = 0; u0 < n; u0 += 8) {
        uint32_t t8[4];
        eight(u0, t8);
        if (by8) {
            pc.template ripple<3>(t8);
        } else if (!half && u0 + 8 < n) {
#pragma unroll
            for (int w = 0; w < 4; ++w) held[w] = t8[w];
            half = true;
            continue;
        } else {
            pc.sixteen(held, t8);
#pragma unroll
            for (int w = 0; w < 4; ++w) held[w] = 0;
            half = false;
        }
        if constexpr (WEIGHTED) pc.bound(pl_unit(it, u0 + 8, n, qshift));
    }
}

// Exact sums of X objects a warp, from object c of the list on: a lane every
// 32nd item.
template <int X>
__device__ __forceinline__ void pl_exact_warp(const uint8_t *base, uint32_t row_bytes, uint32_t tile_lo, uint32_t c,
                                              uint32_t n, uint32_t n_items, uint64_t lbk, const PlItems<true> &it,
                                              PlExact &ex, PlShared &s) {
    const uint32_t lane = lane_id();
    const uint8_t *row[X];
    uint32_t sum[X];
#pragma unroll
    for (int x = 0; x < X; ++x) {
        row[x] = base + (uint32_t)ex.obj[min(c + x, n - 1)] * row_bytes;
        sum[x] = 0;
    }
    for (uint32_t i0 = 0; i0 < n_items; i0 += 64) {
        uint32_t v[2][X], test[2], inc[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t i = i0 + 32 * h + lane;
            test[h] = i < n_items ? it.test[i] : 0u;
            inc[h] = i < n_items ? it.inc[i] : 0u;
#pragma unroll
            for (int x = 0; x < X; ++x) v[h][x] = __ldg(row[x] + (test[h] >> 16));
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int x = 0; x < X; ++x)
                sum[x] += v[h][x] - ((test[h] >> 8) & 255u) <= (test[h] & 255u) ? inc[h] : 0u;
    }
    uint32_t mine = 0;      // lane x: object c + x's sum
#pragma unroll
    for (int x = 0; x < X; ++x) {
        const uint32_t total = __reduce_add_sync(0xffffffffu, sum[x]);
        if (lane == (uint32_t)x) mine = total;
    }
    if (lane < (uint32_t)X && c + lane < n) {
        const uint64_t key = make_key(mine, tile_lo + ex.obj[c + lane]);
        if (key >= lbk) ex.cand[atomicAdd(&s.n, 1u)] = key;
    }
}

// Exact sums of the listed objects (x.obj[0, n), local to the tile) from the
// objects' value rows: keys at or above lbk are appended to x.cand at s.n.  A
// warp sums four objects at a time, eight when there are many (twice the loads
// in flight).  Many objects (a first tile) of few items: a thread an object,
// whose row stays in L1 while its items are read one after the other (64
// queries of up to 20 items, k = 100, 20,000 objects: 393 us a call with a warp
// four, 210 so; of up to 120 items 183 and 224).
__device__ __forceinline__ void pl_exact(const DevIndex &ix, uint32_t tile_lo, uint32_t n, uint32_t n_items,
                                         uint64_t lbk, const PlItems<true> &it, PlExact &ex, PlShared &s) {
    const uint32_t row_bytes = (uint32_t)ix.pl_val_row;
    const uint8_t *base = ix.pl_vals + (uint64_t)tile_lo * (uint64_t)row_bytes;
    constexpr uint32_t kWarps = kPlThreads / 32;
    if (n >= kPlManyExact && n_items <= kPlManyItems) {
        for (uint32_t c = threadIdx.x; c < n; c += kPlThreads) {
            const uint32_t o = ex.obj[c];
            const uint8_t *row = base + o * row_bytes;
            uint32_t total = 0;
#pragma unroll 8
            for (uint32_t i = 0; i < n_items; ++i) {
                const uint32_t test = it.test[i];
                total += __ldg(row + (test >> 16)) - ((test >> 8) & 255u) <= (test & 255u) ? it.inc[i] : 0u;
            }
            const uint64_t key = make_key(total, tile_lo + o);
            if (key >= lbk) ex.cand[atomicAdd(&s.n, 1u)] = key;
        }
    } else if (n > 4 * kWarps) {
        for (uint32_t c = warp_id() * 8; c < n; c += 8 * kWarps)
            pl_exact_warp<8>(base, row_bytes, tile_lo, c, n, n_items, lbk, it, ex, s);
    } else if (warp_id() * 4 < n) {
        pl_exact_warp<4>(base, row_bytes, tile_lo, warp_id() * 4, n, n_items, lbk, it, ex, s);
    }
}

struct PlQuery {
    uint32_t q, k, n_items;
    int qshift;
    uint64_t *region;      // the query's keys
    uint32_t cap;          // keys it holds
    uint32_t *hist;        // [256] primaries written so far
    bool several;          // more than one tile: bounds help
};

// Places of the region (of a table of one tile: of the block's keys) for a
// warp's keys, `mine` per lane: this lane's first.
__device__ __forceinline__ uint32_t pl_claim(const Work &W, const PlQuery &pq, uint32_t mine, PlShared &s) {
    const uint32_t incl = warp_incl_scan(mine);
    uint32_t at = 0;
    if (lane_id() == 31 && incl) at = atomicAdd(pq.several ? &W.pl_cur[pq.q] : &s.n, incl);
    return __shfl_sync(0xffffffffu, at, 31) + incl - mine;
}

// The bound that the histogram of what a query's tiles wrote gives: the
// largest primary with k keys at or above it (one warp; 0: fewer than k keys).
// load() reads the histogram, key() (later) evaluates it.
struct PlBound {
    uint4 hi, lo;          // bins 255 - 8 lane .. 248 - 8 lane
    uint64_t lbk;
    __device__ __forceinline__ void load(const Work &W, const PlQuery &pq) {
        lbk = *(volatile uint64_t *)&W.lbk[pq.q];
        if (!pq.several) return;
        const uint4 *h = (const uint4 *)(pq.hist + (248u - 8u * lane_id()));
        lo = __ldcg(h);
        hi = __ldcg(h + 1);
    }
    template <bool WEIGHTED>
    __device__ __forceinline__ uint64_t key(const PlQuery &pq) const {
        if (!pq.several) return lbk;
        const uint32_t bins[8] = {hi.w, hi.z, hi.y, hi.x, lo.w, lo.z, lo.y, lo.x};
        uint32_t sum = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) sum += bins[j];
        const uint32_t incl = warp_incl_scan(sum);
        uint32_t cum = incl - sum, found = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (cum < pq.k && cum + bins[j] >= pq.k) found = 255u - (8u * lane_id() + j);
            cum += bins[j];
        }
        const uint64_t prim = __reduce_max_sync(0xffffffffu, found);
        const uint64_t k = (WEIGHTED ? prim << 23 : prim) << 32;
        return k > lbk ? k : lbk;
    }
};

// One counted tile of one query: its keys (at most k, every key that can still
// place) into the query's region.  s.lbk holds a lower bound of the query and
// s.n is 0.
template <bool WEIGHTED>
__device__ void pl_select(const DevIndex &ix, const Work &W, const PlQuery &pq, uint64_t tile, PlCounts<WEIGHTED> &pc, const PlItems<WEIGHTED> &it,
                          typename PlScratch<WEIGHTED>::type &ex, PlShared &s) {
    const uint32_t tid = threadIdx.x;
    uint32_t phase = 0;
    const uint32_t tile_lo = (uint32_t)(tile * kPlTile);
    // objects that exist
    uint32_t m[4];
    const int64_t left = (int64_t)ix.n_objects - (int64_t)tile_lo - (int64_t)tid * 128;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const int64_t r = left - 32 * w;
        m[w] = r >= 32 ? 0xFFFFFFFFu : (r <= 0 ? 0u : (1u << r) - 1u);
    }
    uint64_t lbk = s.lbk;
    if constexpr (!WEIGHTED) {
        // a primary at the bound places only with an id up to the bound's
        const uint32_t lp = key_prim(lbk);
        uint32_t c_min = lp > 1u ? lp : 1u;
        if (lp >= 1u && tile_lo > key_id(lbk)) c_min = lp + 1;
        pl_keep_ge<8>(pc.c, c_min, m);
        const uint32_t n = pl_block_sum(pl_popc(m), s, phase);
        if (n == 0) return;
        if (n > pq.k) {
            uint32_t gt[4], value, tot;
            const uint32_t need = pl_kth<8>(pc.c, m, pq.k, gt, value, s, phase);
            const uint32_t ties = pl_popc(m);
            const uint32_t at = group_excl_scan<BlockGroup>(ties, s.tmp, &tot);      // ties of lower ids
            const uint32_t take = at < need ? min(ties, need - at) : 0u;
            pl_first(m, take);
            if (take && at + take == need) {       // the k-th key's id
                uint32_t id = 0;
#pragma unroll
                for (int w = 0; w < 4; ++w)
                    if (m[w]) id = tile_lo + tid * 128u + 32u * w + 31u - __clz((int)m[w]);
                s.last_id = id;
            }
            BlockGroup::sync();
            if (tid == 0)
                atomicMax((unsigned long long *)&W.lbk[pq.q], (unsigned long long)make_key(value, s.last_id));
#pragma unroll
            for (int w = 0; w < 4; ++w) m[w] |= gt[w];
        }
        uint32_t at = pl_claim(W, pq, pl_popc(m), s);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            uint32_t x = m[w];
            while (x) {
                const uint32_t bit = (uint32_t)__ffs((int)x) - 1u;
                x &= x - 1u;
                uint32_t cnt = 0;
#pragma unroll
                for (int b = 0; b < 8; ++b) cnt |= ((pc.c[b][w] >> bit) & 1u) << b;
                const uint64_t key = make_key(cnt, tile_lo + tid * 128u + 32u * w + bit);
                if (!pq.several) {
                    ex.cand[at] = key;
                } else {
                    if (at < pq.cap) __stcg(pq.region + at, key);
                    atomicAdd(&pq.hist[cnt], 1u);
                }
                ++at;
            }
        }
    } else {
        const uint32_t up = pq.qshift > 0 ? (1u << pq.qshift) - 1u : 0u;
        auto units = [&](uint32_t prim) { return prim ? (uint32_t)(((uint64_t)prim + up) >> pq.qshift) : 1u; };
        pl_keep_ge<kPlWSum>(pc.sum, units(key_prim(lbk)), m);
        uint32_t nr = 0;
        bool first = true;
        for (;;) {
            const uint32_t n = pl_block_sum(pl_popc(m), s, phase);
            if (n == 0) break;
            uint32_t take[4], taken;
            const uint32_t room = kPlCand - nr;
            if (first && n > pq.k + 16u) {
                // the k with the largest bounds: their exact k-th prunes the rest
                uint32_t eq[4], value, tot;
#pragma unroll
                for (int w = 0; w < 4; ++w) eq[w] = m[w];
                const uint32_t need = pl_kth<kPlWSum>(pc.sum, eq, pq.k, take, value, s, phase);
                const uint32_t ties = pl_popc(eq);
                const uint32_t at = group_excl_scan<BlockGroup>(ties, s.tmp, &tot);
                pl_first(eq, at < need ? min(ties, need - at) : 0u);
#pragma unroll
                for (int w = 0; w < 4; ++w) take[w] |= eq[w];
                taken = pq.k;
            } else {
                uint32_t tot;
                const uint32_t mine = pl_popc(m);
                const uint32_t at = group_excl_scan<BlockGroup>(mine, s.tmp, &tot);
#pragma unroll
                for (int w = 0; w < 4; ++w) take[w] = m[w];
                pl_first(take, at < room ? min(mine, room - at) : 0u);
                taken = min(n, room);
            }
            first = false;
            uint32_t tot;
            uint32_t at = group_excl_scan<BlockGroup>(pl_popc(take), s.tmp, &tot);
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                m[w] &= ~take[w];
                uint32_t x = take[w];
                while (x) {
                    const uint32_t bit = (uint32_t)__ffs((int)x) - 1u;
                    x &= x - 1u;
                    ex.obj[at++] = (uint16_t)(tid * 128u + 32u * w + bit);
                }
            }
            BlockGroup::sync();
            pl_exact(ix, tile_lo, taken, pq.n_items, lbk, it, ex, s);
            BlockGroup::sync();
            nr = s.n;
            if (taken < n || nr > pq.k) {
                const uint32_t np2 = next_pow2(nr);
                for (uint32_t i = nr + tid; i < np2; i += kPlThreads) ex.cand[i] = 0ull;
                bitonic_sort_desc<BlockGroup>(ex.cand, np2);
                if (nr >= pq.k) {
                    nr = pq.k;
                    if (ex.cand[nr - 1] > lbk) lbk = ex.cand[nr - 1];
                    pl_keep_ge<kPlWSum>(pc.sum, units(key_prim(lbk)), m);
                }
                BlockGroup::sync();
                if (tid == 0) {
                    s.n = nr;
                    if (nr == pq.k) atomicMax((unsigned long long *)&W.lbk[pq.q], (unsigned long long)lbk);
                }
                BlockGroup::sync();
            }
        }
        for (uint32_t b = 0; pq.several && b < nr; b += kPlThreads) {
            const uint32_t i = b + tid;
            const uint32_t at = pl_claim(W, pq, i < nr ? 1u : 0u, s);
            if (i >= nr) continue;
            if (at < pq.cap) __stcg(pq.region + at, ex.cand[i]);
            atomicAdd(&pq.hist[min(key_prim(ex.cand[i]) >> 23, 255u)], 1u);
        }
        BlockGroup::sync();       // the next tile reuses the candidates and s.n
    }
}

// Keys a query's region holds per result slot (the scratch is shared evenly).
__device__ __forceinline__ uint64_t pl_region_k(const DevQueries &Q, const Work &W) {
    const int64_t total_k = Q.out_off[Q.dyn ? (int64_t)Q.dyn[0] : (int64_t)Q.n_queries];
    const uint64_t slots = (uint64_t)W.scratch_keys / (uint64_t)(total_k > 0 ? total_k : 1);
    return slots < 65536 ? slots : 65536;
}

__device__ __forceinline__ PlQuery pl_query(const DevIndex &ix, const DevQueries &Q, const Work &W, uint32_t q,
                                            uint64_t region_k) {
    const QInfo qi = W.qinfo[q];
    PlQuery pq;
    pq.q = q;
    pq.k = qi.k;
    pq.n_items = (uint32_t)qi.n_units;
    pq.qshift = qi.qshift;
    pq.region = W.scratch + (uint64_t)Q.out_off[q] * region_k;
    pq.cap = (uint32_t)umin64((uint64_t)qi.k * region_k, 0x7FFFFFFFull);
    pq.hist = W.pl_hist + (size_t)q * 256;
    pq.several = ix.pl_tiles > 1;
    return pq;
}

// The items of a query into shared memory, padded with empty rows to a multiple of eight.
template <bool WEIGHTED>
__device__ __forceinline__ void pl_items(const DevIndex &ix, const Work &W, int64_t unit0, uint32_t n, uint32_t rank,
                                         uint32_t size, PlItems<WEIGHTED> &it) {
    const uint32_t none = (uint32_t)ix.pl_keys * (uint32_t)ix.pl_row_vec * 16u;
    for (uint32_t i = rank; i < ((n + 7u) & ~7u); i += size) {
        it.rows[i] = i < n ? *(const uint2 *)&W.span_start[unit0 + i] : make_uint2(none, none);
        if (WEIGHTED) {
            it.inc[i] = i < n ? W.inc[unit0 + i] : 0u;
            it.test[i] = i < n ? W.item_nk[unit0 + i] : 0u;
        }
    }
}

// SPLIT: a row of a small table is shorter than the block; then runs of threads
// count a part of the items each, and their counts are added up (1,000 x 128,
// one query of 128 items: 49 us a call with all items in every thread, 38 so).
// Weighted bounds need a query's items in order.
template <bool WEIGHTED, bool SPLIT>
__global__ void __launch_bounds__(kPlThreads, kPlBlocks) k_planes(DevIndex ix, DevQueries Q, Work W) {
    __shared__ PlItems<WEIGHTED> items;
    __shared__ PlShared s;
    __shared__ typename PlScratch<WEIGHTED>::type keys;
    const uint32_t tid = threadIdx.x, lane = lane_id();
    const int list = WEIGHTED ? kListPlanesWeighted : kListPlanes;
    const uint32_t nq = W.ctr[2 * list];
    if (nq == 0) return;
    const uint64_t region_k = pl_region_k(Q, W), n_work = (uint64_t)nq * (uint64_t)ix.pl_tiles;
    unsigned long long *taken = (unsigned long long *)&W.ctr[kCtrPlanes + (WEIGHTED ? 2 : 0)];
    const uint4 *entries = (const uint4 *)(W.work + (size_t)list * W.work_stride);
    const uint32_t width = SPLIT ? next_pow2((uint32_t)ix.pl_row_vec) : kPlThreads, groups = kPlThreads / width;
    const uint32_t mine = min(SPLIT ? tid % width : tid, (uint32_t)ix.pl_row_vec - 1u) * 16u;
    // the pair after this one is claimed while this one is counted
    unsigned long long w = 0;
    if (tid == 0) w = atomicAdd(taken, 1ull);
    for (;;) {
        if (tid == 0) {
            uint4 e = make_uint4(0xFFFFFFFFu, 0u, 0u, 0u);
            uint32_t t = 0;
            if (w < n_work) {
                t = (uint32_t)(w / nq);
                e = __ldg(entries + (w - (uint64_t)t * nq));
            }
            s.entry = e;
            s.tile = t;
        }
        __syncthreads();
        const uint4 e = s.entry;
        const uint32_t tile = s.tile;
        if (e.x == 0xFFFFFFFFu || !GG_OK(e.x, W.q_cap, 12)) return;
        PlQuery pq;
        pq.q = e.x;
        pq.n_items = e.z & 0xFFFFu;
        pq.k = e.z >> 16;
        pq.qshift = (int)e.w;
        pq.hist = W.pl_hist + (size_t)pq.q * 256;
        pq.several = ix.pl_tiles > 1;
        const int64_t out_off = Q.out_off[pq.q];
        pl_items<WEIGHTED>(ix, W, (int64_t)e.y, pq.n_items, tid, kPlThreads, items);
        PlBound bound;                                         // read now, used after the count
        if (warp_id() == 0) bound.load(W, pq);
        __syncthreads();
        if (tid == 0) w = atomicAdd(taken, 1ull);
        PlCounts<WEIGHTED> pc;
        const unsigned char *base = (const unsigned char *)(ix.planes + (uint64_t)tile * (uint64_t)ix.pl_tile_vec);
        if constexpr (SPLIT) {
            const uint32_t per = (pq.n_items + 8 * groups - 1) / (8 * groups) * 8;
            const uint32_t a = min(pq.n_items, tid / width * per), e = min(pq.n_items, a + per);
            pl_count<WEIGHTED>(base, mine, e - a, pq.qshift, items, pc, a);
            pl_join(pc, width, groups, reinterpret_cast<uint4 *>(keys.cand));
        } else {
            pl_count<WEIGHTED>(base, mine, pq.n_items, pq.qshift, items, pc);
        }
        pq.region = W.scratch + (uint64_t)out_off * region_k;
        pq.cap = (uint32_t)umin64((uint64_t)pq.k * region_k, 0x7FFFFFFFull);
        if (warp_id() == 0) {
            const uint64_t lbk = bound.template key<WEIGHTED>(pq);
            if (lane == 0) {
                s.lbk = lbk;
                s.n = 0;
            }
        }
        __syncthreads();
        pl_select<WEIGHTED>(ix, W, pq, tile, pc, items, keys, s);
        if (!pq.several) {       // one tile: its keys are the result
            __syncthreads();
            const uint32_t n = s.n, np2 = next_pow2(n);
            for (uint32_t i = n + tid; i < np2; i += kPlThreads) keys.cand[i] = 0ull;
            bitonic_sort_desc(keys.cand, np2);
            write_results(W, out_off, pq.k, keys.cand, min(n, pq.k), WEIGHTED, WEIGHTED ? W.qinfo[pq.q].scale : 0);
        }
    }
}

// ------------------------------------------------------------------ finish

// A query's region as a set, without the keys below its final bound.
struct PlSet {
    const uint64_t *keys;
    uint32_t n;
    uint64_t lbk;
    template <class F>
    __device__ void for_each(F f) const {
        for (uint32_t b = 0; b < n; b += blockDim.x) {
            const uint32_t i = b + threadIdx.x;
            const uint64_t key = i < n ? __ldcg(keys + i) : 0ull;
            f(i < n && key >= lbk, key_prim(key), key_id(key));
        }
    }
};

// The query again, tile by tile, its region compacted whenever a tile might
// not fit (its tiles wrote more keys than the region holds).  128 threads.
template <bool WEIGHTED>
__device__ uint32_t pl_redo(const DevIndex &ix, const Work &W, const PlQuery &pq, int64_t unit0, PlItems<WEIGHTED> &it,
                            uint64_t *cand, typename PlScratch<WEIGHTED>::type &ex, PlShared &s, SelectScratch &ss) {
    const uint32_t tid = threadIdx.x;
    const uint32_t mine = min(tid, (uint32_t)ix.pl_row_vec - 1u) * 16u;
    pl_items<WEIGHTED>(ix, W, unit0, pq.n_items, tid, kPlThreads, it);
    if (tid == 0) W.pl_cur[pq.q] = 0;
    for (uint32_t i = tid; i < 256; i += kPlThreads) pq.hist[i] = 0;
    uint32_t n = 0;
    for (uint64_t t = 0; t < (uint64_t)ix.pl_tiles; ++t) {
        __threadfence();
        __syncthreads();
        PlCounts<WEIGHTED> pc;
        pl_count<WEIGHTED>((const unsigned char *)(ix.planes + t * (uint64_t)ix.pl_tile_vec), mine, pq.n_items,
                                  pq.qshift, it, pc);
        if (warp_id() == 0) {
            PlBound bound;
            bound.load(W, pq);
            const uint64_t lbk = bound.template key<WEIGHTED>(pq);
            if (tid == 0) {
                s.lbk = lbk;
                s.n = 0;
            }
        }
        __syncthreads();
        pl_select<WEIGHTED>(ix, W, pq, t, pc, it, ex, s);
        __threadfence();
        __syncthreads();
        n = __ldcg(&W.pl_cur[pq.q]);
        if (n + pq.k > pq.cap) {
            n = select_topk(PlSet{pq.region, n, 0ull}, pq.k, WEIGHTED ? 32 : 8, cand, kCandCap, ss);
            for (uint32_t i = tid; i < n; i += kPlThreads) __stcg(pq.region + i, cand[i]);
            if (tid == 0) W.pl_cur[pq.q] = n;
        }
    }
    __syncthreads();
    return n;
}

// Merges every query's keys and writes its results, one CTA per query in turn.
// Once every tile has been counted, the histogram's bound is the k-th primary
// itself (its bucket, weighted), so the keys at or above it are k and a few
// ties: they are collected and sorted.  When the buffer fills (a few queries
// with a large k, whose tiles were all counted before any bound was known, and
// many equal counts) it is sorted and its k-th key becomes the bound: tiles
// write lower ids first, so little more passes.  Selecting from all of a
// query's keys again and again with 128 threads took most of the call (k = 500,
// one query of 16 items in 2,000,000 x 128: 978 us a call, 243 so).  Only a k
// that leaves the buffer no room for a step goes through the general selection.
__global__ void __launch_bounds__(kPlThreads) k_planes_finish(DevIndex ix, DevQueries Q, Work W) {
    __shared__ PlShared s;
    __shared__ uint64_t cand[kCandCap];
    __shared__ union Redo {
        PlExact exact;
        PlKeys keys;
        __device__ Redo() {}
    } redo;
    __shared__ PlItems<true> items_w;
    __shared__ PlItems<false> items_c;
    __shared__ SelectScratch ss;
    const uint32_t tid = threadIdx.x;
    const uint32_t n0 = W.ctr[2 * kListPlanes], n1 = W.ctr[2 * kListPlanesWeighted];
    const uint64_t region_k = n0 + n1 ? pl_region_k(Q, W) : 0;
    for (uint32_t w = blockIdx.x; w < n0 + n1; w += gridDim.x) {
        const bool weighted = w >= n0;
        const int list = weighted ? kListPlanesWeighted : kListPlanes;
        const uint32_t q = ((const uint4 *)(W.work + (size_t)list * W.work_stride))[weighted ? w - n0 : w].x;
        if (!GG_OK(q, W.q_cap, 12)) break;
        const QInfo qi = W.qinfo[q];
        const PlQuery pq = pl_query(ix, Q, W, q, region_k);
        uint32_t n = W.pl_cur[q];
        if (n > pq.cap)
            n = weighted ? pl_redo<true>(ix, W, pq, qi.unit0, items_w, cand, redo.exact, s, ss)
                         : pl_redo<false>(ix, W, pq, qi.unit0, items_c, cand, redo.keys, s, ss);
        if (warp_id() == 0) {
            PlBound bound;
            bound.load(W, pq);
            const uint64_t lbk = weighted ? bound.template key<true>(pq) : bound.template key<false>(pq);
            if (tid == 0) {
                s.lbk = lbk;
                s.n = 0;
            }
        }
        __syncthreads();
        uint64_t lbk = s.lbk;
        constexpr uint32_t kAhead = 8, kStep = kAhead * kPlThreads;
        // what is kept and a step's keys fit the buffer
        const bool prune = pq.k + kStep <= (uint32_t)kCandCap;
        uint64_t key[kAhead];
        const auto load = [&](uint32_t b) {
#pragma unroll
            for (uint32_t j = 0; j < kAhead; ++j) {
                const uint32_t i = b + j * kPlThreads + tid;
                key[j] = i < n ? __ldcg(pq.region + i) : 0ull;
            }
        };
        load(0);
        for (uint32_t b = 0; b < n; b += kStep) {
#pragma unroll
            for (uint32_t j = 0; j < kAhead; ++j)
                if (key[j] && key[j] >= lbk) {
                    const uint32_t at = atomicAdd(&s.n, 1u);
                    if (at < (uint32_t)kCandCap) cand[at] = key[j];
                }
            load(b + kStep);
            if (!prune || b + kStep >= n) continue;
            __syncthreads();
            const uint32_t have = s.n;
            if (have + kStep > (uint32_t)kCandCap) {      // more than k
                const uint32_t np2 = next_pow2(have);
                for (uint32_t i = have + tid; i < np2; i += kPlThreads) cand[i] = 0ull;
                bitonic_sort_desc(cand, np2);
                lbk = cand[pq.k - 1];
                __syncthreads();
                if (tid == 0) s.n = pq.k;
            }
            __syncthreads();
        }
        __syncthreads();
        uint32_t got = s.n;
        if (got <= (uint32_t)kCandCap) {
            const uint32_t np2 = next_pow2(got);
            for (uint32_t i = got + tid; i < np2; i += kPlThreads) cand[i] = 0ull;
            bitonic_sort_desc(cand, np2);
            got = min(got, pq.k);
        } else {
            got = select_topk(PlSet{pq.region, n, lbk}, pq.k, weighted ? 32 : 8, cand, kCandCap, ss);
        }
        write_results(W, Q.out_off[q], pq.k, cand, got, weighted, qi.scale);
        __syncthreads();
    }
}

}  // namespace gg
