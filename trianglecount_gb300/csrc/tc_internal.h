// tc_internal.h -- shared declarations of libtc's translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>

#include "tc.h"

namespace tc {

// ---- errors ------------------------------------------------------------------
// Records a message for tc_last_error() on the calling thread; returns status.
int set_error(int status, const char *fmt, ...) __attribute__((format(printf, 2, 3)));
int cuda_error(cudaError_t e, const char *what, const char *file, int line);

#define TC_CUDA(call)                                                                 \
    do {                                                                              \
        cudaError_t tc_e_ = (call);                                                   \
        if (tc_e_ != cudaSuccess) return ::tc::cuda_error(tc_e_, #call, __FILE__, __LINE__); \
    } while (0)

#define TC_TRY(call)                    \
    do {                                \
        int tc_s_ = (call);             \
        if (tc_s_ != TC_OK) return tc_s_; \
    } while (0)

// ---- device scratch ------------------------------------------------------------
// Stream-ordered allocation from the device's default memory pool (its release
// threshold is raised at context creation, so freed blocks stay cached and a
// steady-state call does not reach the driver allocator).
int dalloc(void **p, size_t bytes, cudaStream_t s);
void dfree(void *p, cudaStream_t s);

template <class T>
struct DBuf {
    T *p = nullptr;
    size_t n = 0;
    cudaStream_t s = nullptr;
    DBuf() = default;
    DBuf(const DBuf &) = delete;
    DBuf &operator=(const DBuf &) = delete;
    ~DBuf() { reset(); }
    int alloc(size_t count, cudaStream_t stream) {
        reset();
        s = stream;
        n = count;
        return dalloc((void **)&p, (count ? count : 1) * sizeof(T), stream);
    }
    void reset() {
        if (p) dfree(p, s);
        p = nullptr;
        n = 0;
    }
    T *release() {
        T *q = p;
        p = nullptr;
        n = 0;
        return q;
    }
};

// ---- counting kernels (tc_count.cu) ----------------------------------------------
struct GraphDesc {
    const int32_t *rp;
    const int32_t *col;
    int64_t n_rows;
    int64_t n_roots;
    int64_t chunk_base;           // exclusive prefix of 32-row chunks over graphs
    int64_t vbase;                // exclusive prefix of (n_rows + 1) over graphs
    int64_t ebase;                // exclusive prefix of nnz over graphs
    unsigned long long *per_root; // optional g_sum output (zeroed by the caller)
    int32_t mbits;                // mask bits of the packed rows' entries (pack_mask_bits)
};

struct HeavyEntry {
    int32_t g, u, unit_base, n_slices;  // units = ceil(d+(u) / tile) * n_slices
};

// The packed count's arrays (tc_pack.cu), pooled over a launch's graphs:
// V = sum (n_rows + 1), E = sum nnz.
struct PackScratch {
    uint32_t *code = nullptr;      // V, then 512 words per graph (popularity histogram and cursors)
    int4 *desc = nullptr;          // V
    uint4 *ent = nullptr;          // (E + 13 V) / 4 + 2
    uint32_t *mid_list = nullptr;  // E / 33 + 1
    uint2 *units = nullptr;        // E / 16 + 1
};

// Device arrays of one count launch, sized for its graphs (pooled over a batch):
// V = sum (n_rows + 1), C = sum ceil(n_rows / 32), E = sum nnz.
struct CountScratch {
    HeavyEntry *heavy = nullptr;  // heavy_cap entries
    int64_t heavy_cap = 0;
    uint32_t *light_list = nullptr;         // V: light tasks from entry 0 up, micro tasks from entry V - 1
                                            // down, as global rows chunk * 32 + lane
    int32_t *in_cnt = nullptr;              // V
    int32_t *in_off = nullptr;              // V + 1
    unsigned long long *in_work = nullptr;  // V
    unsigned long long *out_work = nullptr; // V
    int32_t *in_list = nullptr;             // E
    uint8_t *mid = nullptr;                 // E: edge done middle-centric
    PackScratch pk;                         // the packed count's arrays instead of the above
};
// Allocates the arrays of the packed or the plain-id count, where sc does not have them yet.
int scratch_alloc(CountScratch *sc, int64_t V, int64_t E, int64_t heavy_cap, int n_graphs, bool packed,
                  cudaStream_t s);
// The same, the plain-id count's (less per row) where the packed count's do not fit
// the memory; *packed then says so.
int scratch_alloc_either(CountScratch *sc, int64_t V, int64_t E, int64_t heavy_cap, int n_graphs, bool *packed,
                         cudaStream_t s);
void scratch_free(CountScratch *sc, cudaStream_t s);

// Per-launch device words, zeroed by one memset before each count.
struct CountWork {
    unsigned long long heavy_packed; // (entries << 32) | units, from the classifier
    unsigned int heavy_cursor;
    unsigned int small_cursor;       // light-task cursor
    unsigned int aux_cursor[2];      // chunk cursors of in_count, transpose/classify
    unsigned int self_loops;         // the packed count met a row that is its own member
    int error;                       // 1: heavy-unit list overflow; 2: a bulk-copy staging wait gave up
    unsigned long long total_work;   // sum over oriented edges of the cheaper side's length
    unsigned long long n_tasks;      // tasks listed by the classifier, one atomic per chunk for both
                                     // lists: light (low half, task list from the bottom) and micro
                                     // (high half, from the top)
};

struct Tuned {  // resolved tc_tuning with derived table geometry
    int warp_max;        // power of two
    int log_warp_slots;
    int light_max_work;
    int unit_work;
    int long_list;
    int probe_kicks;     // 0: linear-probing hash; > 0: cuckoo hash with this kick bound
    int heavy_bitmap;    // 1: heavy units on direct-address bitmaps when the ids fit
    int hash_pairs;      // 1: bucketed-pair hash tables (one 8-byte load per probe)
    int flat_max_deg;    // graphs whose rows are all this short count with flat_kernel (0: never)
    int intersect;       // 0: hash tables; 1: bulk-staged sorted lists; 2: per light task by its work
    int bitmap_bytes;    // shared memory the bitmap kernel may use (ids < 8 x this)
    int sm_count;
    int tile;            // block table entries per tile (a quarter of its slots)
    int log_block_slots;
    int threads;         // per block
    int blocks;          // persistent grid
    int pack_blocks;     // persistent grid of the packed count
    int aux_blocks;      // resident grid of the per-chunk auxiliary kernels
    size_t smem;         // dynamic shared memory bytes
};

int resolve_tuning(const tc_tuning &t, int sm_count, Tuned *out);

// ---- packed count (tc_pack.cu) ----------------------------------------------------
// The default tuning's count of skewed graphs (packed_graphs); the options that name a table form (linear
// probing, pair tables, id bitmaps, sorted lists) count on tc_count.cu's tables
// of plain ids.
inline bool packed_count(const Tuned &tn) {
    return tn.probe_kicks > 0 && !tn.hash_pairs && !tn.heavy_bitmap && tn.intersect == 0;
}
bool pack_fits(int64_t V, int64_t E);  // else the plain-id tables count it
int pack_mask_bits(int64_t n_rows);
size_t pack_scratch_bytes(int64_t V, int64_t E, int n_graphs);
int pack_scratch_alloc(PackScratch *ps, int64_t V, int64_t E, int n_graphs, cudaStream_t s);
void pack_scratch_free(PackScratch *ps, cudaStream_t s);
// The packed count's persistent grid, num / den of what fits (a grid kept below
// occupancy leaves the same share of an SM free as the plain-id count's).
int pack_blocks(int sm_count, int num, int den, int *out);
int launch_packed(const GraphDesc *d_desc, int n_graphs, int64_t total_chunks, int64_t total_vertices,
                  int64_t total_edges, const PackScratch &ps, CountWork *work, unsigned long long *results,
                  bool per_root, const Tuned &tn, cudaStream_t s, int *launches, cudaEvent_t *kev);
// Out-neighbours per block unit of the packed count: 32 to 512.
inline int pack_slice(const Tuned &tn) {
    const int s = tn.unit_work / 2048;
    return s < 32 ? 32 : s > 512 ? 512 : s;
}
// What a count of g launches under its context's tuning, as far as the tuning decides it.
struct CountRoute {
    enum Form { kFlat, kSingle, kPacked, kPlain } form;
    int warp_max, slice;  // of the packed count
    bool same(const CountRoute &o) const {  // (the plain-id count reads every threshold)
        return form == o.form && form != kPlain && warp_max == o.warp_max && slice == o.slice;
    }
};
CountRoute count_route(const tc_graph *g);
// One-kernel count of a graph of few edges, on its own ids.
int launch_single(const GraphDesc &d, CountWork *work, unsigned long long *result, const Tuned &tn, cudaStream_t s,
                  int *launches, cudaEvent_t *kev);
// Zeroes a launch's work words and its n results.
int zero_work(CountWork *work, unsigned long long *results, int n, cudaStream_t s);
// Records a kernel-timing event on s; inside a stream capture (the plain
// count's cached graph) as an external event node, so that every replay of
// the captured chain records it too.
int record_kernel_event(cudaEvent_t ev, cudaStream_t s);

// launch_count for callers that cannot allocate: the in-edge scan keeps its
// tile sums in scan_tmp (scan_tmp_cap values); nothing is allocated.
int launch_count_noalloc(const GraphDesc *d_desc, int64_t total_chunks, int64_t total_vertices,
                         const CountScratch &sc, int32_t *scan_tmp, int64_t scan_tmp_cap, CountWork *work,
                         unsigned long long *results, const Tuned &tn, cudaStream_t s);

// One-kernel count of a graph whose rows are all at most max_deg <= 8 long
// (one lane per root, lists in registers; loop_free: no row holds its own id, so a
// root with one member has no hit); fills the work words and result
// like launch_count.
int launch_flat(const int32_t *rp, const int32_t *col, int64_t n_roots, int max_deg, bool loop_free, CountWork *work,
                unsigned long long *result, unsigned long long *per_root, const Tuned &tn, cudaStream_t s,
                int *launches, cudaEvent_t *kev);

// Enqueues [degree -> in_count -> scan -> transpose/classify -> micro ->
// count] for n_graphs descriptors on stream s; results[n_graphs] receives the
// per-graph totals (zeroed here); total_vertices = sum (n_rows + 1), max_rows
// = the largest n_rows.  kev (optional, two events) is recorded around the
// counting kernels (heavy bitmap + persistent count).  halo_parts: some graph
// of the launch is a halo part (n_roots < n_rows); its heavy units then run
// the count kernel's instance for small units.
int launch_count(const GraphDesc *d_desc, int n_graphs, int64_t total_chunks, int64_t total_vertices,
                 int64_t total_edges, bool packed, int64_t max_rows, const CountScratch &sc, CountWork *work, unsigned long long *results, bool per_root,
                 const Tuned &tn, cudaStream_t s, int *launches, cudaEvent_t *kev = nullptr,
                 bool halo_parts = false);

// ---- scans and sort (tc_scan.cu, tc_sort.cu) ----------------------------------------
// Exclusive scan of n values into out[0..n] (out[n] = total).  out may alias in.
int scan_exclusive_i32(const int32_t *in, int32_t *out, int64_t n, cudaStream_t s);
int scan_exclusive_i64(const int64_t *in, int64_t *out, int64_t n, cudaStream_t s);
// Exclusive scan of 0/1 byte flags into int32 positions out[0..n].
int scan_flags_u8(const uint8_t *flags, int32_t *out, int64_t n, cudaStream_t s);
// scan_exclusive_i32 with its tile sums in caller memory (no allocation).
int scan_exclusive_i32_tmp(const int32_t *in, int32_t *out, int64_t n, int32_t *tmp, int64_t tmp_cap,
                           cudaStream_t s);
// The count's in-list offsets: in_off[0..n] = exclusive scan of the in-edge
// counts held in the high halves of in_work[0..n), and each in_work[i]'s high
// half becomes in_off[i] + count, the end of vertex i's in-list.  The tile
// sums go to tmp (tmp_cap values), or to a stream-ordered allocation when tmp
// is null.
int scan_in_slots(unsigned long long *in_work, int32_t *in_off, int64_t n, int32_t *tmp, int64_t tmp_cap,
                  cudaStream_t s);
// Local ids of a halo part's members: out[0..n] = exclusive scan of (part
// vertices) + (halo vertices left) << 32 (cd: class, degree; out[n]: both totals).
int scan_halo_ids(const int2 *cd, const uint8_t *removed, int64_t *out, int64_t n, cudaStream_t s);
// LSD radix sort of n 64-bit keys on bits [0, bits).  Result in *keys (the
// two buffers may be swapped).  tmp must hold n keys.
int radix_sort_u64(uint64_t **keys, uint64_t **tmp, int64_t n, int bits, cudaStream_t s);

int device_sm_count(int device);

// ---- row lengths (tc_api.cu) --------------------------------------------------------
// What the choice of a graph's count asks of its rows' lengths.
constexpr int64_t kSkew = 5;
struct RowStats {
    int32_t longest = -1;  // the longest row; -1: not known
    uint32_t skewed = 0;   // entries in rows longer than kSkew x the mean
    uint32_t far = 0;      // entries in rows that no degree orientation has (RowBounds)
    int32_t filled = 0;    // rows that have entries
};
// An orientation by degree has rows of at most sqrt(2 nnz) members, and in R-MAT
// and Chung-Lu graphs of at most a tenth of that.
struct RowBounds {
    int32_t skew, far;
};
inline RowBounds row_bounds(int64_t n_rows, int64_t nnz) {
    const int64_t b = n_rows > 0 ? kSkew * nnz / n_rows : 0;
    int64_t f = 512;
    while (16 * f * f < nnz) f += f / 8;  // about sqrt(nnz) / 4
    return {b < INT32_MAX ? (int32_t)b : INT32_MAX, (int32_t)f};
}
#ifdef __CUDACC__
// Appends x to list, *n entries long, with one atomic for the lanes that are here
// together (a frontier holds hundreds of thousands of vertices, and one atomic
// each on the one counter was most of the peeling).
__device__ __forceinline__ void push_together(int32_t *list, int32_t *n, int32_t x) {
    const unsigned here = __activemask();
    const int lane = threadIdx.x & 31, first = __ffs(here) - 1;
    int at = 0;
    if (lane == first) at = atomicAdd(n, __popc(here));
    at = __shfl_sync(here, at, first);
    list[at + __popc(here & ((1u << lane) - 1u))] = x;
}

// One thread's rows, then a block's added to the launch's: all its threads call add,
// once (one warp's sums at a time were 150 K atomics on one line for every part of a
// halo extraction, 30 us of its 1 ms).
struct RowTally {
    int longest = 0;
    unsigned skewed = 0, far = 0, filled = 0, of_roots = 0;
    __device__ __forceinline__ void row(int d, RowBounds b) {
        longest = max(longest, d);
        filled += (unsigned)(d > 0);
        if (d > b.skew) skewed += (unsigned)d;
        if (d > b.far) far += (unsigned)d;
    }
    __device__ __forceinline__ void add(RowStats *out, int32_t *root_nnz = nullptr) {
        __shared__ int s_longest;
        __shared__ unsigned s_sum[4];
        if (threadIdx.x < 4) s_sum[threadIdx.x] = 0;
        if (threadIdx.x == 0) s_longest = 0;
        __syncthreads();
        longest = __reduce_max_sync(0xffffffffu, longest);
        const unsigned sum[4] = {__reduce_add_sync(0xffffffffu, skewed), __reduce_add_sync(0xffffffffu, far),
                                 __reduce_add_sync(0xffffffffu, of_roots), __reduce_add_sync(0xffffffffu, filled)};
        if ((threadIdx.x & 31) == 0 && longest) {
            atomicMax(&s_longest, longest);
            for (int i = 0; i < 4; ++i)
                if (sum[i]) atomicAdd(&s_sum[i], sum[i]);
        }
        __syncthreads();
        if (threadIdx.x == 0 && s_longest) {
            atomicMax(&out->longest, s_longest);
            if (s_sum[0]) atomicAdd(&out->skewed, s_sum[0]);
            if (s_sum[1]) atomicAdd(&out->far, s_sum[1]);
            if (root_nnz && s_sum[2]) atomicAdd(root_nnz, (int)s_sum[2]);
            atomicAdd(&out->filled, (int)s_sum[3]);
        }
    }
};
#endif
// The row statistics of a device CSR into *d_out.
int row_stats(tc_ctx *ctx, const int32_t *rp, int64_t n_rows, int64_t nnz, RowStats *d_out);

// Counts n graphs (same device) with one batched launch on ctx's stream and
// waits up to timeout_ms for the results (TC_E_TIMEOUT after that; the
// launch is then still in flight).  Scratch comes from the stream-ordered pool.
int count_graphs_direct(tc_ctx *ctx, tc_graph *const *graphs, int n, uint64_t *outs, int64_t timeout_ms,
                        float *kernel_ms);
// Moves a graph to another context of the same device (reference counts follow).
int graph_rebind(tc_graph *g, tc_ctx *ctx);
// Device bytes of a graph: its CSR, and the scratch that it has or that its count takes.
size_t graph_device_bytes(const tc_graph *g);

// Context lifetime: every graph, ugraph and batch holds a reference to its
// context, so tc_ctx_destroy only drops the caller's reference and the
// context is freed when its last object is destroyed.
void ctx_retain(tc_ctx *c);
void ctx_release(tc_ctx *c);

}  // namespace tc

// ---- library object layouts ----------------------------------------------------------
struct tc_ctx {
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    int sm_count = 0;
    tc_tuning tuning{};
    tc::Tuned tuned{};
    unsigned long long tuning_epoch = 0;  // bumped by every tuning change (cached count graphs go stale)
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
    cudaEvent_t kev[2] = {nullptr, nullptr};  // around the last count kernel launch
    bool kev_recorded = false;
    unsigned long long *h_pinned = nullptr;  // small pinned read-back area
    // created on first use by tc_count_parts_csr_i32: a copy stream and a
    // high-priority validation stream, so uploads overlap the counts
    cudaStream_t aux[2] = {nullptr, nullptr};
    std::atomic<int> refs{1};                // the handle + one per live object
};

struct tc_graph {
    tc_ctx *ctx = nullptr;
    int32_t *rp = nullptr;
    int32_t *col = nullptr;
    int64_t n_rows = 0, nnz = 0, n_roots = 0;
    tc::RowStats rows;     // known for uploads and device-built graphs; of wrapped ones as look_at_rows saw them
    int64_t root_nnz = -1; // entries in the roots' rows; -1: not known
    bool owns = true;
    bool loop_free = false;  // no row holds its own id (device-built graphs)
    bool no_pack = false;    // the packed count's scratch did not fit the memory
    // per-graph count scratch, sized on first use
    tc::GraphDesc *d_desc = nullptr;
    tc::CountWork *d_work = nullptr;
    unsigned long long *d_result = nullptr;
    tc::CountScratch sc{};
    tc::GraphDesc desc_on_device{};  // what d_desc holds (skip re-uploads)
    bool desc_valid = false;
    // The count chain captured as a CUDA graph on the graph's second count and
    // replayed after that (one launch instead of ~10 stream operations), while
    // the results pointer and the context's tuning stay the same; a results
    // pointer is captured once two counts in a row used it.
    cudaGraphExec_t exec = nullptr;
    unsigned long long *exec_results = nullptr;
    unsigned long long *last_results = nullptr;  // results pointer of the previous chain count
    unsigned long long exec_epoch = 0;
    int exec_launches = 0;
    int chain_counts = 0;  // chain counts enqueued so far
};

struct tc_ugraph {
    tc_ctx *ctx = nullptr;
    int32_t *rp = nullptr;
    int32_t *col = nullptr;
    int32_t *deg = nullptr;    // degree used for orientation
    int32_t *rowid = nullptr;  // row of each entry (nnz)
    int64_t n_rows = 0, nnz = 0;
};
