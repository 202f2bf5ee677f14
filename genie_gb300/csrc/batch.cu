// batch.cu -- batched search: fixed-capacity buffers, pinned staging, the
// device work of a batch captured once as a CUDA graph, and the autotuner.
//
// The reference runs one synchronous pipeline per batch: host query compile,
// H2D of the compiled spans, match_AT, a host-synchronising overflow check,
// heap_count_topk with cudaMalloc/cudaFree, D2H (matching/knn.cu:106-183,
// match.cu:224-464).  Here the batch size lives in device memory, so the same
// graph (memset, plan and the persistent kernels of the lists, of an index's
// planes, or both) serves every batch that needs no other kernels.
#include "capi_internal.h"

#include <cstring>
#include <vector>

using namespace gg;

struct genie_batch {
    genie_index *ix = nullptr;
    genie_batch_config cfg{};
    Workspace ws;
    DevBuf dyn;
    Tuning tuning{};
    cudaStream_t stream = nullptr;
    cudaGraphExec_t gexec = nullptr;
    bool graph_valid = false;
    int64_t graph_planes = 0;        // which planes of the index the graph was captured with (0: none)
    uint32_t need = 0, graph_need = 0;   // LaunchNeed of the batches staged so far, and of the graph
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t stage_ev[kStages + 1] = {};
    // pinned staging
    int64_t *h_out_off = nullptr;
    uint8_t *h_weighted = nullptr;
    uint32_t *h_k = nullptr, *h_dyn = nullptr, *h_err = nullptr;
    int32_t staged_q = 0;
    int64_t staged_sumk = 0;
    int last_kernels = 0;
    bool launched = false;
    ~genie_batch();
};

genie_batch::~genie_batch() {
    if (ix) cudaSetDevice(ix->device);
    if (gexec) cudaGraphExecDestroy(gexec);
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    for (cudaEvent_t e : stage_ev)
        if (e) cudaEventDestroy(e);
    if (stream) cudaStreamDestroy(stream);
    void *pinned[] = {h_out_off, h_weighted, h_k, h_dyn, h_err};
    for (void *p : pinned)
        if (p) cudaFreeHost(p);
    ws.release();
    dyn.release();
}

namespace {

template <class T>
cudaError_t pin(T *&p, size_t n) {
    return cudaMallocHost((void **)&p, n * sizeof(T) + 64);
}

DevQueries device_queries(const genie_batch *b) {
    DevQueries q;
    q.n_queries = b->cfg.max_queries;
    q.item_off = (const int64_t *)b->ws.item_off.p;
    q.dim = (const int32_t *)b->ws.dim.p;
    q.low = (const int32_t *)b->ws.low.p;
    q.up = (const int32_t *)b->ws.up.p;
    q.weight = (const float *)b->ws.weight.p;
    q.weighted = (const uint8_t *)b->ws.weighted.p;
    q.k = (const uint32_t *)b->ws.k.p;
    q.uniform_k = 0;
    q.out_off = (const int64_t *)b->ws.out_off.p;
    q.dyn = (const uint32_t *)b->dyn.p;
    q.route = 0;
    return q;
}

bool caller_captures(const genie_batch *b, cudaStream_t s) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (s != b->stream) cudaStreamIsCapturing(s, &status);
    return status != cudaStreamCaptureStatusNone;
}

int enqueue(genie_batch *b, cudaStream_t s) {
    DeviceContext &ctx = device_context(b->ix->device);
    const PlanesUse use(b->ix);
    const int64_t planes = b->ix->pl_tiles > 0 && b->tuning.dense_bitmaps && b->ws.planes.p ? b->ix->pl_built.load() : 0;
    // A caller that captures a launch replays it for whatever it stages later:
    // no kernel is left out, and the planes stay.
    const bool captured = caller_captures(b, s);
    const uint32_t need = captured ? (uint32_t)kNeedAll : b->need;
    if (captured && planes) {
        std::lock_guard<std::mutex> g(b->ix->pl_mu);
        b->ix->pl_held = true;
    }
    if (b->graph_valid && b->cfg.use_graph && b->graph_planes == planes && (!planes || b->graph_need == need)) {
        cudaError_t e = cudaGraphLaunch(b->gexec, s);
        return e ? cuda_fail(e, "graph launch") : GENIE_OK;
    }
    const DevQueries q = device_queries(b);
    DevIndex d = index_view(b->ix, b->tuning);           // directories built before a capture
    if (!planes) d.planes = nullptr;
    const Work w = b->ws.view(b->cfg.max_queries, true);
    if (!b->cfg.use_graph) {
        // direct launches, with an event after every stage for per-kernel timing
        b->last_kernels = launch_match(d, q, w, b->tuning, ctx.num_sms, s, captured ? nullptr : b->stage_ev, need);
        cudaError_t e = cudaGetLastError();
        return e ? cuda_fail(e, "batch launch") : GENIE_OK;
    }
    if (!b->graph_valid || b->graph_planes != planes || (planes && b->graph_need != need)) {
        b->graph_valid = false;
        if (b->gexec) cudaGraphExecDestroy(b->gexec);
        b->gexec = nullptr;
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal);
        if (e) return cuda_fail(e, "graph capture");
        b->last_kernels = launch_match(d, q, w, b->tuning, ctx.num_sms, b->stream, nullptr, need);
        cudaError_t le = cudaGetLastError();
        e = cudaStreamEndCapture(b->stream, &g);
        if (le) {
            if (g) cudaGraphDestroy(g);
            return cuda_fail(le, "graph capture launch");
        }
        if (e) return cuda_fail(e, "graph capture end");
        e = cudaGraphInstantiate(&b->gexec, g, 0);
        cudaGraphDestroy(g);
        if (e) return cuda_fail(e, "graph instantiate");
        b->graph_valid = true;
        b->graph_planes = planes;
        b->graph_need = need;
    }
    cudaError_t e = cudaGraphLaunch(b->gexec, s);
    return e ? cuda_fail(e, "graph launch") : GENIE_OK;
}

// Validate and copy a batch into pinned staging, then to the device (async on s).
int stage_async(genie_batch *b, const genie_queries *q, cudaStream_t s) {
    std::vector<int64_t> out_off;
    int64_t n_items = 0;
    int rc = validate_queries(q, out_off, n_items);
    if (rc) return rc;
    const int64_t Q = q->n_queries;
    if (Q > b->cfg.max_queries) return fail(GENIE_ERR_INVALID_ARG, "%lld queries exceed the batch capacity %d", (long long)Q, b->cfg.max_queries);
    if (n_items > b->cfg.max_items) return fail(GENIE_ERR_INVALID_ARG, "%lld items exceed the batch capacity %lld", (long long)n_items, (long long)b->cfg.max_items);
    for (int64_t i = 0; i < Q; ++i) {
        const uint32_t k = q->k ? q->k[i] : q->uniform_k;
        if (k > b->cfg.max_k) return fail(GENIE_ERR_INVALID_ARG, "k=%u exceeds the batch capacity %u", k, b->cfg.max_k);
    }
    note_search(b->ix, q, b->tuning);
    // The caller's item arrays are uploaded from where they are: a copy from
    // pageable memory returns once the source may be reused, and on a
    // coherently attached host it moves the bytes without a staging memcpy,
    // which is faster than one through pinned buffers.  The arrays built here
    // (k, result offsets, batch size) go through pinned staging.
    // Exact-match items (up is the low array itself) travel once.
    const bool exact = q->up == q->low;
    const bool weighted = q->weighted && q->weight;
    if (!weighted) memset(b->h_weighted, 0, Q);
    for (int64_t i = 0; i < Q; ++i) b->h_k[i] = q->k ? q->k[i] : q->uniform_k;
    memcpy(b->h_out_off, out_off.data(), (Q + 1) * 8);
    b->h_dyn[0] = (uint32_t)Q;
    b->h_dyn[1] = q->uniform_k;
    b->h_dyn[2] = exact ? 1u : 0u;
    const PlanesPlan plan = planes_plan(b->ix, q);
    b->need |= plan.need;
    b->h_dyn[3] = plan.route;
    cudaError_t e = cudaSuccess;
    Workspace &ws = b->ws;
    auto h2d = [&](void *dst, const void *src, size_t n) {
        if (n && !e) e = cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, s);
    };
    h2d(ws.item_off.p, q->item_off, (Q + 1) * 8);
    h2d(ws.dim.p, q->dim, n_items * 4);
    h2d(ws.low.p, q->low, n_items * 4);
    if (!exact) h2d(ws.up.p, q->up, n_items * 4);
    if (weighted) h2d(ws.weight.p, q->weight, n_items * 4);
    h2d(ws.weighted.p, weighted ? (const void *)q->weighted : (const void *)b->h_weighted, Q);
    h2d(ws.k.p, b->h_k, Q * 4);
    h2d(ws.out_off.p, b->h_out_off, (Q + 1) * 8);
    h2d(b->dyn.p, b->h_dyn, 16);
    if (e) return cuda_fail(e, "batch upload");
    b->staged_q = (int32_t)Q;
    b->staged_sumk = out_off[Q];
    return GENIE_OK;
}

// The error word of the last launch into pinned memory (async on s); the
// results themselves are downloaded by finish_fetch into the caller's buffers.
int fetch_async(genie_batch *b, cudaStream_t s, bool scores) {
    (void)scores;
    const Work w = b->ws.view(b->cfg.max_queries, true);
    cudaError_t e = cudaMemcpyAsync(b->h_err, w.ctr + kCtrError, 4, cudaMemcpyDeviceToHost, s);
    return e ? cuda_fail(e, "batch download") : GENIE_OK;
}

int finish_fetch(genie_batch *b, uint32_t *ids, uint32_t *counts, float *scores) {
    cudaError_t e = cudaStreamSynchronize(b->stream);
    if (e) return cuda_fail(e, "batch");
    int rc = check_device_error(*b->h_err);
    if (rc) return rc;
    // results straight into the caller's buffers (faster than a download
    // into pinned staging and a host copy out of it)
    const size_t n = (size_t)b->staged_sumk;
    const Work w = b->ws.view(b->cfg.max_queries, true);
    if (ids && n) e = cudaMemcpy(ids, w.out_ids, n * 4, cudaMemcpyDeviceToHost);
    if (!e && counts && n) e = cudaMemcpy(counts, w.out_counts, n * 4, cudaMemcpyDeviceToHost);
    if (!e && scores && n) e = cudaMemcpy(scores, w.out_scores, n * 4, cudaMemcpyDeviceToHost);
    if (e) return cuda_fail(e, "batch download");
    return GENIE_OK;
}

Tuning from_public(const Tuning &base, const genie_tuning &t) {
    Tuning r = base;
    if (t.sparse_slots > 0) {
        r.sparse_slots_packed = (t.sparse_slots + 31) & ~31;
        r.sparse_slots_wide = ((t.sparse_slots / 2) + 31) & ~31;
    }
    if (t.sparse_ctas_per_sm > 0) {
        r.sparse_ctas_per_sm = t.sparse_ctas_per_sm == 1 ? 1 : 2;
        r.sparse_threads = t.sparse_ctas_per_sm == 1 ? 1024 : 512;
    }
    if (t.sparse_load_pct > 0) r.sparse_load_pct = t.sparse_load_pct;
    if (t.dense_tile > 0) {
        r.dense_tile_u8 = (t.dense_tile + 255) & ~255;
        r.dense_tile_u32 = ((t.dense_tile / 4) + 63) & ~63;
    }
    if (t.dense_threads > 0) r.dense_threads = t.dense_threads;
    if (t.sparse_max_total > 0) r.sparse_max_total = t.sparse_max_total;
    if (t.dense_part_work > 0) r.dense_part_work = t.dense_part_work;
    if (t.bitmap_bits > 0) r.bitmap_bits = t.bitmap_bits;
    if (t.bitmap_bits < 0) r.bitmap_bits = 0;
    if (t.dense_bitmaps > 0) r.dense_bitmaps = t.dense_bitmaps & 3;
    if (t.dense_bitmaps < 0) r.dense_bitmaps = 0;
    return r;
}

void to_public(const Tuning &r, genie_tuning &t) {
    t.sparse_slots = r.sparse_slots_packed;
    t.sparse_ctas_per_sm = r.sparse_ctas_per_sm;
    t.dense_tile = r.dense_tile_u8;
    t.dense_threads = r.dense_threads;
    t.sparse_max_total = r.sparse_max_total;
    t.dense_part_work = r.dense_part_work;
    t.sparse_load_pct = r.sparse_load_pct;
    t.bitmap_bits = r.bitmap_bits > 0 ? r.bitmap_bits : -1;
    t.dense_bitmaps = r.dense_bitmaps > 0 ? r.dense_bitmaps : -1;
}

}  // namespace

extern "C" {

int genie_batch_create(genie_index *ix, const genie_batch_config *cfg, genie_batch **out) {
    if (!ix || !cfg || !out) return fail(GENIE_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    if (cfg->max_queries <= 0 || cfg->max_items < 0 || cfg->max_k == 0 || cfg->max_k > (uint32_t)kMaxK)
        return fail(GENIE_ERR_INVALID_ARG, "batch capacity must hold >= 1 query and 1 <= max_k <= %d", kMaxK);
    if (ix->sub_shift >= 0)
        return fail(GENIE_ERR_NOT_IMPLEMENTED, "a subsequence index is searched through genie_search");
    if ((int64_t)cfg->max_queries * kMaxDenseParts >= ((int64_t)1 << 32))
        return fail(GENIE_ERR_INVALID_ARG, "at most %lld queries per batch", (long long)(((int64_t)1 << 32) / kMaxDenseParts - 1));
    cudaSetDevice(ix->device);
    genie_batch *b = new genie_batch();
    b->ix = ix;
    b->cfg = *cfg;
    b->tuning = ix->tuning;
    const int64_t Q = cfg->max_queries, I = cfg->max_items > 0 ? cfg->max_items : 1, K = (int64_t)Q * cfg->max_k;
    const int64_t U = cfg->max_units > 0 ? cfg->max_units : 16 * I;
    // what the planes need is there before they are: a launch allocates nothing
    // and every launch of a batch, also one its caller captured, uses the same
    // buffers.  Without the memory for it the batch stays on the lists.
    if (may_have_planes(ix) && b->ws.reserve_planes(Q, K, ix->host.n_objects)) {
        cudaGetLastError();
        b->ws.planes.release();
    }
    cudaError_t e = b->ws.reserve(Q, I, U, K);
    if (!e) e = b->dyn.reserve(16);
    if (!e) e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
    if (!e) e = cudaEventCreate(&b->ev0);
    if (!e) e = cudaEventCreate(&b->ev1);
    for (int i = 0; i <= kStages && !e; ++i) e = cudaEventCreate(&b->stage_ev[i]);
    if (!e) e = pin(b->h_out_off, Q + 1);
    if (!e) e = pin(b->h_weighted, Q);
    if (!e) e = pin(b->h_k, Q);
    if (!e) e = pin(b->h_dyn, 4);
    if (!e) e = pin(b->h_err, 4);
    if (e) {
        delete b;
        return cuda_fail(e, "batch buffers");
    }
    *out = b;
    return GENIE_OK;
}

int genie_batch_destroy(genie_batch *b) {
    delete b;
    return GENIE_OK;
}

int genie_batch_stage(genie_batch *b, const genie_queries *q) {
    if (!b) return fail(GENIE_ERR_INVALID_ARG, "batch is NULL");
    cudaSetDevice(b->ix->device);
    int rc = stage_async(b, q, b->stream);
    if (rc) return rc;
    cudaError_t e = cudaStreamSynchronize(b->stream);
    return e ? cuda_fail(e, "batch upload") : GENIE_OK;
}

int genie_batch_launch(genie_batch *b, void *stream) {
    if (!b) return fail(GENIE_ERR_INVALID_ARG, "batch is NULL");
    cudaSetDevice(b->ix->device);
    cudaStream_t s = stream ? (cudaStream_t)stream : b->stream;
    if (caller_captures(b, s)) return enqueue(b, s);      // nothing runs yet that the events could time
    cudaEventRecord(b->ev0, s);
    int rc = enqueue(b, s);
    cudaEventRecord(b->ev1, s);
    b->launched = rc == GENIE_OK;
    return rc;
}

int genie_batch_fetch(genie_batch *b, uint32_t *out_ids, uint32_t *out_counts, float *out_scores) {
    if (!b) return fail(GENIE_ERR_INVALID_ARG, "batch is NULL");
    cudaSetDevice(b->ix->device);
    cudaStreamWaitEvent(b->stream, b->ev1, 0);
    int rc = fetch_async(b, b->stream, out_scores != nullptr);
    if (rc) return rc;
    return finish_fetch(b, out_ids, out_counts, out_scores);
}

int genie_batch_run(genie_batch *b, const genie_queries *q, uint32_t *out_ids, uint32_t *out_counts,
                    float *out_scores) {
    if (!b) return fail(GENIE_ERR_INVALID_ARG, "batch is NULL");
    cudaSetDevice(b->ix->device);
    int rc = stage_async(b, q, b->stream);
    if (rc) return rc;
    if (b->staged_q == 0) return GENIE_OK;
    cudaEventRecord(b->ev0, b->stream);
    rc = enqueue(b, b->stream);
    cudaEventRecord(b->ev1, b->stream);
    b->launched = rc == GENIE_OK;
    if (rc) return rc;
    rc = fetch_async(b, b->stream, out_scores != nullptr);
    if (rc) return rc;
    return finish_fetch(b, out_ids, out_counts, out_scores);
}

int genie_batch_get_tuning(const genie_batch *b, genie_tuning *out) {
    if (!b || !out) return fail(GENIE_ERR_INVALID_ARG, "NULL argument");
    to_public(b->tuning, *out);
    return GENIE_OK;
}

int genie_batch_set_tuning(genie_batch *b, const genie_tuning *t) {
    if (!b || !t) return fail(GENIE_ERR_INVALID_ARG, "NULL argument");
    Tuning r = from_public(b->tuning, *t);
    const size_t smem_cap = kSmemCap;
    if (r.sparse_slots_packed < 1024 || sparse_smem_bytes(r, true) > smem_cap ||
        sparse_smem_bytes(r, false) > smem_cap || r.dense_tile_u8 < 4096 ||
        dense_smem_bytes(r, true) > smem_cap || dense_smem_bytes(r, false) > smem_cap ||
        (r.dense_threads != 512 && r.dense_threads != 1024) || r.sparse_load_pct < 25 ||
        r.sparse_load_pct > 90 || (r.bitmap_bits > 0 && (r.bitmap_bits < 8192 || r.bitmap_bits > (1 << 24))))
        return fail(GENIE_ERR_INVALID_ARG, "tuning outside the supported shapes");
    b->tuning = r;
    b->graph_valid = false;
    return GENIE_OK;
}

int genie_batch_last_stats(const genie_batch *b, int32_t *kernels, float *device_ms) {
    if (!b) return fail(GENIE_ERR_INVALID_ARG, "batch is NULL");
    if (kernels) *kernels = b->last_kernels;
    if (device_ms) {
        *device_ms = 0.0f;
        if (b->launched) {
            cudaEventSynchronize(b->ev1);
            cudaEventElapsedTime(device_ms, b->ev0, b->ev1);
        }
    }
    return GENIE_OK;
}

int genie_batch_stage_ms(const genie_batch *b, float *ms) {
    if (!b || !ms) return fail(GENIE_ERR_INVALID_ARG, "NULL argument");
    if (b->cfg.use_graph) return fail(GENIE_ERR_INVALID_ARG, "per-kernel times need a batch created with use_graph = 0");
    if (!b->launched) return fail(GENIE_ERR_INVALID_ARG, "no launch yet");
    cudaEventSynchronize(b->stage_ev[kStages]);
    for (int i = 0; i < kStages; ++i) {
        ms[i] = 0.0f;
        cudaEventElapsedTime(&ms[i], b->stage_ev[i], b->stage_ev[i + 1]);
    }
    return GENIE_OK;
}

// Times each candidate shape on the sample (one warm-up, three timed graph
// launches) and keeps the fastest.  Candidates vary the hash slots per CTA
// (hence CTAs per SM), the dense tile, the sparse/dense crossover, the
// presence-bitmap kernel (on with a bitmap size, or off) and the dense lists'
// bitmaps (on or off; always on for a table that may have planes: off keeps the
// batch off those too, whereas the sample is timed on whatever exists by then).
int genie_batch_autotune(genie_batch *b, const genie_queries *sample, genie_tuning *chosen) {
    if (!b || !sample) return fail(GENIE_ERR_INVALID_ARG, "NULL argument");
    cudaSetDevice(b->ix->device);
    int rc = genie_batch_stage(b, sample);
    if (rc) return rc;
    const Tuning base = b->tuning;
    // hash slots, CTAs per SM (2: 512 threads, 1: 1024 threads), load %, dense tile,
    // crossover, largest id space of the bitmap kernel (-1: bitmap kernel off),
    // counter widths whose dense lists use their bitmaps (-1: none)
    struct Cand { int32_t slots, ctas, load, tile; int64_t smax; int32_t bits, dbm; };
    const Cand cands[] = {
        {22528, 2, 50, 147456, 270336, -1, 1}, {11264, 2, 50, 147456, 270336, -1, 1},
        {22528, 2, 60, 147456, 270336, -1, 1}, {45056, 1, 50, 147456, 270336, -1, 1},
        {53248, 1, 56, 147456, 270336, -1, 1}, {53248, 1, 62, 147456, 270336, -1, 1},
        {22528, 2, 50, 98304, 270336, -1, 1},  {22528, 2, 50, 147456, 67584, -1, 1},
        {53248, 1, 62, 147456, 1081344, -1, 1},
        {53248, 1, 56, 147456, 270336, 1179648, 1}, {53248, 1, 56, 147456, 1081344, 1179648, 1},
        {22528, 2, 50, 147456, 270336, 1179648, 1},
        {22528, 2, 50, 172032, 270336, -1, 1}, {22528, 2, 50, 147456, 270336, -1, -1},
        {22528, 2, 50, 172032, 270336, -1, -1},
    };
    float best_ms = 1e30f;
    Tuning best = base;
    // three timed launches of the current tuning after one untimed; a tuning
    // whose launch fails is skipped, a device error ends the search
    auto try_current = [&]() -> int {
        float total = 0.0f;
        bool ok = true;
        for (int it = 0; it < 4 && ok; ++it) {
            if (genie_batch_launch(b, nullptr)) {
                ok = false;
                break;
            }
            float ms = 0.0f;
            genie_batch_last_stats(b, nullptr, &ms);
            if (it > 0) total += ms;
        }
        cudaError_t e = cudaStreamSynchronize(b->stream);
        if (e) return cuda_fail(e, "autotune");
        if (ok && total < best_ms) {
            best_ms = total;
            best = b->tuning;
        }
        return GENIE_OK;
    };
    for (const Cand &c : cands) {
        if (c.dbm < 0 && may_have_planes(b->ix)) continue;
        genie_tuning t{};
        t.sparse_slots = c.slots;
        t.sparse_ctas_per_sm = c.ctas;
        t.sparse_load_pct = c.load;
        t.dense_tile = c.tile;
        t.sparse_max_total = c.smax;
        t.bitmap_bits = c.bits;
        t.dense_bitmaps = c.dbm;
        if (genie_batch_set_tuning(b, &t)) continue;
        if ((rc = try_current())) return rc;
        b->tuning = base;
    }
    // then the objects per dense part, in whole tiles of the chosen tile size
    const Tuning first = best;
    for (int64_t tiles = 1; tiles <= 4; ++tiles) {
        b->tuning = first;
        b->tuning.dense_part_work = tiles * first.dense_tile_u8;
        b->graph_valid = false;
        if ((rc = try_current())) return rc;
    }
    b->tuning = best;
    b->graph_valid = false;
    if (chosen) to_public(best, *chosen);
    return GENIE_OK;
}

}  // extern "C"

// ---------------------------------------------------------------- serving steps

int gg::batch_submit_async(genie_batch *b, const genie_queries *q, bool scores) {
    cudaSetDevice(b->ix->device);
    int rc = stage_async(b, q, b->stream);
    if (rc) return rc;
    cudaEventRecord(b->ev0, b->stream);
    rc = enqueue(b, b->stream);
    b->launched = rc == GENIE_OK;
    if (rc) return rc;
    rc = fetch_async(b, b->stream, scores);
    if (rc) return rc;
    cudaError_t e = cudaEventRecord(b->ev1, b->stream);
    return e ? cuda_fail(e, "batch event") : GENIE_OK;
}

int gg::batch_ready(genie_batch *b) {
    cudaError_t e = cudaEventQuery(b->ev1);
    if (e == cudaSuccess) return 1;
    if (e == cudaErrorNotReady) return 0;
    return -cuda_fail(e, "batch");
}

int gg::batch_collect(genie_batch *b, uint32_t *ids, uint32_t *counts, float *scores) {
    return finish_fetch(b, ids, counts, scores);
}

extern "C" int genie_batch_submit(genie_batch *b, const genie_queries *q, int32_t want_scores) {
    if (!b || !q) return fail(GENIE_ERR_INVALID_ARG, "NULL argument");
    cudaSetDevice(b->ix->device);
    cudaError_t e = cudaStreamSynchronize(b->stream);     // the staging buffers are free again
    if (e) return cuda_fail(e, "batch");
    b->staged_sumk = 0;
    return batch_submit_async(b, q, want_scores != 0);
}

extern "C" int genie_batch_collect(genie_batch *b, uint32_t *out_ids, uint32_t *out_counts, float *out_scores) {
    if (!b) return fail(GENIE_ERR_INVALID_ARG, "batch is NULL");
    cudaSetDevice(b->ix->device);
    return batch_collect(b, out_ids, out_counts, out_scores);
}
