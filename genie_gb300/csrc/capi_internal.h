// capi_internal.h -- host-side state behind the C ABI handles.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <cmath>
#include <cstdint>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/genie_gb300.h"
#include "host_index.h"
#include "match.cuh"

namespace gg {

int fail(int code, const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);

// cudaMalloc; when the device is full, once more after the planes (planes.cu)
// of the indexes that no call is using have been given back.
cudaError_t device_alloc(void **p, size_t bytes);

// One growable device allocation.
struct DevBuf {
    void *p = nullptr;
    size_t bytes = 0;
    cudaError_t reserve(size_t want);
    void release();
};

struct DeviceContext {
    bool ready = false;
    int num_sms = 0;
    cudaError_t prepare_error = cudaSuccess;
    Tuning tuning;
};
DeviceContext &device_context(int dev);

// Device buffers of one in-flight search (query inputs, plan, work lists,
// part scratch, results), grown on demand.
struct Workspace {
    DevBuf item_off, dim, low, up, weight, weighted, k, out_off;
    DevBuf item_k0, item_nk, item_inc;
    DevBuf span_start, span_len, inc, qinfo, work, ctr, qstate, done, lb, part_cnt, scratch;
    DevBuf out_ids, out_counts, out_scores;
    DevBuf counters;                 // per-object counters of a subsequence search
    DevBuf unit_key;
    DevBuf call;                     // inputs, counters and results of a small call
    DevBuf planes;                   // per-query state of k_planes: bounds, histograms, key counts
    bool done_zeroed = false;
    int64_t done_q = 0;
    // io: the query inputs and results too (a small call has its own, `call`)
    cudaError_t reserve(int64_t Q, int64_t items, int64_t units, int64_t sumk, bool io = true);
    // what a search with an index's planes needs beside; before reserve() and
    // view() (when it fails it may have freed the scratch)
    cudaError_t reserve_planes(int64_t Q, int64_t sumk, int64_t n_objects);
    void release();
    Work view(int64_t Q, bool scores) const;
};

// Calls whose inputs and results fit are packed into one upload and one
// download through pinned memory, which every index holds.  Below the limit
// packing gains all along (354 KB, 384 queries of 64 items: 149 us a call, 183
// unpacked; 118 KB 88 and 110); above it still some (472 KB 174 and 208, 944 KB
// 275 and 293), for which an index pins no more.
constexpr size_t kCallBytes = 384 << 10;
// The pinned words of an index (host_err).
cudaError_t alloc_host_words(genie_index *ix);

int validate_queries(const genie_queries *q, std::vector<int64_t> &out_off, int64_t &n_items);

// The device view of an index for a tuning: ix->dev plus the tile
// directories of the tuning's two tile sizes (built on first use).
DevIndex index_view(genie_index *ix, const Tuning &t);
// Called with every batch of queries before it is searched with a tuning:
// builds the cumulative planes of a byte-valued index (planes.cu) once the
// searches that may use them are worth it.
void note_search(genie_index *ix, const genie_queries *q, const Tuning &t);
// Whether the index's values allow planes, built or not.
bool may_have_planes(genie_index *ix);
// Frees the planes of the current device's indexes that are not in use; whether
// there were any.  Their searches go back to the lists, and earn planes anew.
bool give_back_planes();
// An index is destroyed.
void forget_planes(genie_index *ix);
// Held from an index's view to the launch of what uses it.
struct PlanesUse {
    genie_index *ix;
    explicit PlanesUse(genie_index *index);
    ~PlanesUse();
    PlanesUse(const PlanesUse &) = delete;
    PlanesUse &operator=(const PlanesUse &) = delete;
};
// How a batch is counted on an index with planes: the kernels to launch
// (LaunchNeed; a batch without planes needs kNeedLists) and the PlanesRoute that
// the plan kernel goes by.
struct PlanesPlan {
    uint32_t need, route;
};
PlanesPlan planes_plan(const genie_index *ix, const genie_queries *q);

// Asynchronous steps of one batch for the serving loop (batch.cu): stage,
// launch and download on the batch's own stream; poll; copy the results out.
int batch_submit_async(genie_batch *b, const genie_queries *q, bool scores);
int batch_ready(genie_batch *b);      // 1 done, 0 still running, < 0 a CUDA error
int batch_collect(genie_batch *b, uint32_t *ids, uint32_t *counts, float *scores);
int check_device_error(uint32_t err);
// Drop the fixed workspace's cached device address of a device (after a reset).
void noalloc_forget(int dev);
// Search of a subsequence index (subseq.cu), on ix->stream; waits when sync.
int subseq_search(genie_index *ix, const genie_queries *q, const std::vector<int64_t> &out_off, int64_t n_items,
                  uint32_t *out_ids, uint32_t *out_counts, float *out_scores, bool sync);
int64_t count_units(const HostIndex &h, const genie_queries *q);

}  // namespace gg

namespace gg {
// Device arrays and view of an index from its host mirror; with device_ids
// >= 0 the ids and key offsets are on the device already (device build).
int upload_index(genie_index *ix, int64_t device_ids = -1);
int finish_index_create(genie_index *ix, genie_index **out, int64_t device_ids = -1);
// Device build of a one-value-per-object index (build_index.cu); *used is
// false when a dim's value range needs the host builder.
int build_device_index(const int32_t *values, int64_t n, int32_t d, genie_index *ix, bool *used);
}  // namespace gg

struct genie_index {
    int device = 0;
    bool is_bag = false;
    int32_t sub_shift = -1;          // subsequence index: ids are rowID << sub_shift | offset (-1: not one)
    gg::HostIndex host;              // host mirror: bounds and key offsets (ids live on the device)
    int64_t n_ids = 0;
    int32_t codec = 0;
    int32_t max_seg = 0;
    int64_t n_words = 0;
    int64_t n_segs = 0;
    gg::DevBuf d_ids, d_key_off, d_key_base, d_dim_min, d_dim_max;
    gg::DevBuf d_words, d_key_seg, d_seg_word_off, d_seg_first, d_seg_len;
    gg::DevIndex dev{};
    gg::Tuning tuning{};
    // tile directories (tile_dir.cu), built on first use per tile size and
    // kept while the index lives
    std::mutex dir_mu;
    bool dir_rows_ready = false;
    int64_t dir_rows = -1;
    gg::DevBuf d_dir_slot, d_dir_row_key;
    bool bm_ready = false;
    int64_t bm_words = 0;
    uint32_t bm_zero = 0;
    gg::DevBuf d_bm_slot, d_bm_rows;
    std::vector<std::pair<int32_t, gg::DevBuf *>> dirs;
    std::atomic<int64_t> pl_bytes{-1};   // what the planes take (0: the index has none, -1: not looked at)
    std::atomic<int64_t> pl_touched{0};  // posting ids its searches have touched before they were built
    std::atomic<int64_t> pl_tiles{0};    // set once built
    std::atomic<int64_t> pl_built{0};    // how often they have been: a graph holds the pointers of one time
    int64_t pl_row_vec = 0;
    gg::DevBuf d_planes, d_pl_vals;
    std::mutex pl_mu;                // of the two below; held while the planes are freed
    int pl_users = 0;                // calls between the index's view and their launches
    bool pl_held = false;            // a caller captured launches that use the planes
    cudaStream_t stream = nullptr;
    std::mutex mu;                   // serialises searches on this handle's workspace
    gg::Workspace ws;
    uint32_t *host_err = nullptr;    // pinned: error word of the last search, then kCallBytes of a small call
    int64_t call_results = -1;       // small call in flight: result slots (-1: none), and where its
    size_t call_ctr = 0;             // counters and results start in the call's bytes
    int last_launches = 0;
    ~genie_index();
};
