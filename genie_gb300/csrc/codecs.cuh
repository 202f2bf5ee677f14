// codecs.cuh -- warp-level decoders of the reference posting-list codecs,
// emitting values in sequence order straight into the counting loop.
//
// Formats (byte-compatible with the reference's host encoders):
//   COPY     words are the values                       (DeviceCodecs.h:113-154)
//   DELTA    words are differences, first from 0        (DeviceCodecs.cu:89-139)
//   BP32     [n][w0<<24|w1<<16|w2<<8|w3][w0 words]..[w3 words] per 128 values;
//            value j of a 32-value miniblock sits at bits [j*w, j*w+w), LSB
//            first; a short tail packs ceil(rem/32) zero-padded miniblocks
//                                                      (DeviceBitPackingCodec.cu:15-58)
//   VARINT   7-bit groups, low first, the LAST byte of a value has bit 7 set,
//            zero-padded to whole words                 (DeviceVarintCodec.cu:14-78)
//   COMP(BP32,C2)  [len1][BP32 over floor(n/8)*8 values][C2 over the rest]
//                                                      (DeviceCompositeCodec.cu:28-58)
//   SERIAL(C1,C2)  C2 decoded first, then C1            (DeviceSerialCodec.cu:67-137)
//
// The reference decodes one segment per 256-thread block through shared
// memory with a sequential header parse on thread 0
// (DeviceBitPackingCodec.cu:160-200) and block-wide scans (utility/scan.cu).
// Here one warp decodes one segment: miniblock offsets come from the header
// bytes, varint boundaries from the terminal bits of each lane's word, and
// delta runs as a warp prefix sum with a carry.
#pragma once
#include "codecs_host.h"
#include "device.cuh"

namespace gg {

// Emits a group of values: lane l holds `cnt` values val[0..cnt) whose
// sequence positions are base + before(l) + 0..cnt-1 (before = exclusive
// prefix of cnt over lanes).  The emitter applies the delta stages in
// sequence order and hands each value to `visit`.
template <class V, bool POS = true>
struct Emitter {
    int deltas;
    uint32_t carry1 = 0, carry2 = 0;
    uint32_t emitted = 0;      // values emitted so far (sequence position of the next)
    V &visit;
    __device__ Emitter(int d, V &v) : deltas(d), visit(v) {}
    __device__ __forceinline__ void emit(const uint32_t *val, int cnt) {
        uint32_t v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = j < cnt ? val[j] : 0u;
        emit_mask(v, (1u << cnt) - 1u);
    }
    // the same for the values j with bit j of `has` set (the others are 0): in
    // a lane they keep their order, without being moved together
    __device__ __forceinline__ void emit_mask(const uint32_t (&val)[4], uint32_t has) {
        // sequence position of this lane's first value (skipped when the
        // visitor does not use positions)
        uint32_t pos0 = 0;
        if (POS) {
            const uint32_t cnt = __popc(has), cincl = warp_incl_scan(cnt);
            pos0 = emitted + cincl - cnt;
            emitted += __shfl_sync(0xffffffffu, cincl, 31);
        }
        uint32_t v[4] = {val[0], val[1], val[2], val[3]};
        delta(v, has);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if ((has >> j) & 1u) visit(v[j], pos0 + __popc(has & ((1u << j) - 1u)));
    }
    // a whole block, four values in every lane; the visitor takes a lane's four at once
    __device__ __forceinline__ void emit_block(uint32_t (&v)[4]) {
        delta(v);
        visit.four(v, emitted + 4u * lane_id());
        emitted += 128;
    }
    // running sums over the lane's values, then across lanes; absent values
    // are 0 and their sums unused, and before the second stage
    // (SERIAL_DELTA_DELTA) 0 again
    __device__ __forceinline__ void delta(uint32_t (&v)[4], uint32_t has = 15u) {
        if (deltas == 0) return;
        sum(v, carry1);
        if (deltas == 1) return;
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = (has >> j) & 1u ? v[j] : 0u;
        sum(v, carry2);
    }
    __device__ __forceinline__ void sum(uint32_t (&v)[4], uint32_t &carry) {
        v[1] += v[0];
        v[2] += v[1];
        v[3] += v[2];
        const uint32_t incl = warp_incl_scan(v[3]);
        const uint32_t pre = carry + incl - v[3];
        carry += __shfl_sync(0xffffffffu, incl, 31);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] += pre;
    }
};

// Word sources of the decoders.  Every lane of the warp calls word() the
// same number of times (the register source shuffles).
struct GlobalWords {      // words read from global memory
    const uint32_t *__restrict__ w;
    __device__ __forceinline__ uint32_t word(int64_t i) const { return __ldg(w + i); }
    // word i where cond holds, else 0 (read only where cond holds)
    __device__ __forceinline__ uint32_t word_if(int64_t i, bool cond) const { return cond ? __ldg(w + i) : 0u; }
};
struct RegWords {         // a segment of <= 64 words held two per lane
    int64_t base;
    uint32_t r0, r1;
    __device__ __forceinline__ uint32_t word(int64_t i) const {
        const uint32_t rel = (uint32_t)(i - base);
        const uint32_t a = __shfl_sync(0xffffffffu, r0, rel & 31u);
        const uint32_t b = __shfl_sync(0xffffffffu, r1, rel & 31u);
        return rel < 32u ? a : (rel < 64u ? b : 0u);
    }
    __device__ __forceinline__ uint32_t word_if(int64_t i, bool cond) const {
        const uint32_t x = word(i);      // every lane shuffles
        return cond ? x : 0u;
    }
};

struct SmemWords {        // a segment staged in shared memory; positions past it read its last word
    const uint32_t *s;
    int64_t base;
    uint32_t last;
    __device__ __forceinline__ uint32_t word(int64_t i) const { return s[min((uint32_t)(i - base), last)]; }
    __device__ __forceinline__ uint32_t word_if(int64_t i, bool cond) const { return cond ? word(i) : 0u; }
};

// Words [w0, w1) as values, 32 per step.
template <class S, class E>
__device__ __forceinline__ void dec_copy(const S &src, int64_t w0, int64_t w1, E &em) {
    for (int64_t b = w0; b < w1; b += 32) {
        int64_t i = b + lane_id();
        const uint32_t x = src.word(i < w1 ? i : w0);
        uint32_t v[1] = {i < w1 ? x : 0u};
        em.emit(v, i < w1 ? 1 : 0);
    }
}

// One BP32 stream starting at word w0 ([n][blocks...]); returns the word
// after it.  Lane l decodes values 4l..4l+3 of each 128-value block (all in
// miniblock l/8), so one emit (one prefix scan) covers the whole block.
template <class S, class E>
__device__ __forceinline__ int64_t dec_bp32(const S &src, int64_t w0, E &em) {
    const uint32_t lane = lane_id();
    const uint32_t n = src.word(w0);
    int64_t p = w0 + 1;
    for (uint32_t done = 0; done < n; done += 128) {
        const uint32_t hdr = src.word(p);
        const uint32_t rem = n - done;
        const uint32_t howmany = rem >= 128 ? 4u : (rem + 31) / 32;
        // widths of the miniblocks present (a short tail packs fewer)
        uint32_t bw[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) bw[m] = (uint32_t)m < howmany ? (hdr >> (24 - 8 * m)) & 255u : 0u;
        const uint32_t mb = lane >> 3;
        uint32_t b = bw[0], before = 0;
#pragma unroll
        for (int m = 1; m < 4; ++m)
            if ((uint32_t)m <= mb) {
                before += bw[m - 1];
                b = bw[m];
            }
        const int64_t off = p + 1 + before;
        const uint32_t j0 = (lane & 7u) * 4u;
        const uint32_t mask = b >= 32 ? 0xFFFFFFFFu : (1u << b) - 1u;
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t bit = (j0 + k) * b, wi = bit >> 5, sh = bit & 31;
            const uint32_t lo = src.word_if(off + wi, b > 0);
            const uint32_t hi = src.word_if(off + wi + 1, b > 0 && sh + b > 32);
            v[k] = (uint32_t)((((uint64_t)hi << 32) | lo) >> sh) & mask;
        }
        const int have = (int)min(4u, rem > 4 * lane ? rem - 4 * lane : 0u);
        em.emit(v, have);
        p += 1 + bw[0] + bw[1] + bw[2] + bw[3];
    }
    return p;
}

// The same from shared memory: a value is cut from its two words by one funnel
// shift, unconditionally (a width of 0 masks everything away; bits past the
// value's own are masked).
template <class E>
__device__ __forceinline__ int64_t dec_bp32(const SmemWords &src, int64_t w0, E &em) {
    const uint32_t lane = lane_id(), mb = lane >> 3;
    const uint32_t n = src.word(w0);
    uint32_t p = (uint32_t)(w0 + 1 - src.base);
    for (uint32_t done = 0; done < n && p <= src.last; done += 128) {
        const uint32_t hdr = src.s[p];
        const uint32_t rem = n - done;
        const uint32_t used = rem >= 97 ? hdr : hdr & ~(0xFFFFFFFFu >> (8u * ((rem + 31) / 32)));
        const uint32_t b = (used >> (24u - 8u * mb)) & 255u;
        // words of the miniblocks before this lane's: the header's higher bytes
        const uint32_t over = mb ? used >> (32u - 8u * mb) : 0u;
        const uint32_t before = (over & 255u) + ((over >> 8) & 255u) + (over >> 16);
        // every word a value touches lies before p + 1 + all (or, masked away, on it)
        const uint32_t all = (used & 255u) + ((used >> 8) & 255u) + ((used >> 16) & 255u) + (used >> 24);
        if (p + all > src.last) break;
        const uint32_t mask = b >= 32 ? 0xFFFFFFFFu : (1u << b) - 1u;
        const uint32_t *at = src.s + p + 1 + before;
        uint32_t bit = (lane & 7u) * 4u * b;
        uint32_t v[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t wi = bit >> 5;
            v[k] = __funnelshift_r(at[wi], at[wi + 1], bit) & mask;
            bit += b;
        }
        if (rem >= 128) em.emit_block(v);
        else em.emit(v, (int)min(4u, rem > 4 * lane ? rem - 4 * lane : 0u));
        p += 1 + all;
    }
    return src.base + p;
}

// Varint bytes of words [w0, w1): a lane owns one word; each byte with bit 7
// set ends a value of at most five bytes, so a value spans at most this word
// and the previous one.
template <class S, class E>
__device__ __forceinline__ void dec_varint(const S &src, int64_t w0, int64_t w1, E &em) {
    const uint32_t lane = lane_id();
    uint32_t prev_last = 0;            // previous chunk's last word
    bool have_prev = false;
    for (int64_t b = w0; b < w1; b += 32) {
        const int64_t i = b + lane;
        const uint32_t raw = src.word(i < w1 ? i : w0);
        const uint32_t cur = i < w1 ? raw : 0u;
        uint32_t prv = __shfl_up_sync(0xffffffffu, cur, 1);
        if (lane == 0) prv = have_prev ? prev_last : 0u;
        const bool prv_valid = lane > 0 || have_prev;
        // the window's bytes in order: seven bits each into the running value,
        // which a terminal byte ends; before this word's bytes only the value
        // that the previous word leaves open counts
        uint32_t vals[4], has = 0, acc = 0, sh = 0;
#pragma unroll
        for (int t = 0; t < 8; ++t) {
            const uint32_t byte = ((t < 4 ? prv >> (8 * t) : cur >> (8 * (t - 4)))) & 255u;
            acc |= sh < 32u ? (byte & 0x7Fu) << sh : 0u;
            sh += 7;
            if (t >= 4) vals[t - 4] = (byte & 0x80u) ? acc : 0u;
            if ((byte & 0x80u) || (t == 3 && !prv_valid)) {
                if (t >= 4) has |= 1u << (t - 4);
                acc = 0;
                sh = 0;
            }
        }
        em.emit_mask(vals, has);
        prev_last = __shfl_sync(0xffffffffu, cur, 31);
        have_prev = true;
    }
}

// Decode one encoded segment (words [w0, w1)) from a word source and visit
// its values in order.
template <bool POS, class S, class V>
__device__ __forceinline__ void decode_words(int codec, const S &src, int64_t w0, int64_t w1, V &visit) {
    int deltas, inner;
    codec_parts(codec, deltas, inner);
    Emitter<V, POS> em(deltas, visit);
    switch (inner) {
    case kInnerCopy:
        dec_copy(src, w0, w1, em);
        break;
    case kInnerBP32:
        dec_bp32(src, w0, em);
        break;
    case kInnerVarint:
        dec_varint(src, w0, w1, em);
        break;
    default: {     // composite: [len1][BP32 (len1 words)][tail]
        const uint32_t len1 = src.word(w0);
        int64_t p = w0 + 1;
        if (len1) dec_bp32(src, p, em);
        p += len1;
        if (p < w1) {
            if (inner == kInnerCompCopy) dec_copy(src, p, w1, em);
            else dec_varint(src, p, w1, em);
        }
    }
    }
}

// Longest segment decoded from shared memory; the buffer holds two words more
// (a value's second word may lie past the segment).
constexpr uint32_t kStageWords = 1150;

// Decode one encoded segment and visit (value, sequence position) in order,
// and whole lanes of four by visit.four(values, position).  The segment's words
// are first copied to shared memory in coalesced steps, so the chain of block
// headers (each tells where the next one is) costs shared loads; a longer
// segment is read word by word.
template <class V>
__device__ __forceinline__ void decode_segment(int codec, const uint32_t *__restrict__ w, int64_t w0, int64_t w1,
                                               uint32_t *stage, V &visit) {
    if (w1 - w0 <= (int64_t)kStageWords) {
        const uint32_t n = (uint32_t)(w1 - w0), lane = lane_id();
        if (n == 0) return;
        __syncwarp();
        for (uint32_t b = 0; b < n; b += 32 * 8) {
            uint32_t x[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) x[r] = b + 32 * r + lane < n ? __ldg(w + w0 + b + 32 * r + lane) : 0u;
#pragma unroll
            for (int r = 0; r < 8; ++r)
                if (b + 32 * r + lane < n) stage[b + 32 * r + lane] = x[r];
        }
        if (lane < 2) stage[n + lane] = 0;
        __syncwarp();
        decode_words<true>(codec, SmemWords{stage, w0, n - 1}, w0, w1, visit);
    } else {
        decode_words<true>(codec, GlobalWords{w}, w0, w1, visit);
    }
}

// The same for a visitor of values only (no sequence positions).
template <class V>
__device__ __forceinline__ void decode_segment_values(int codec, const uint32_t *__restrict__ w, int64_t w0,
                                                      int64_t w1, V &visit) {
    if (w1 - w0 <= 64) {
        const uint32_t lane = lane_id();
        RegWords src{w0, w0 + lane < w1 ? __ldg(w + w0 + lane) : 0u,
                     w0 + 32 + lane < w1 ? __ldg(w + w0 + 32 + lane) : 0u};
        decode_words<false>(codec, src, w0, w1, visit);
    } else {
        decode_words<false>(codec, GlobalWords{w}, w0, w1, visit);
    }
}

}  // namespace gg
