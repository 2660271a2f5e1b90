// tc_pack.cu -- the default exact count: packed rows, root-centric.
//
// Quantity and citations as in tc_count.cu: for each root u, the sum over v in
// N+(u) of |N+(u) n N+(v)| (ShareKernelTCV62_update_v1.cu:43-191).  That size
// depends only on which ids are equal, so any renumbering of the ids gives the
// same count.  Here every count renumbers the vertices by popularity (how many
// root lists hold them, most popular first) and packs each row into 32-bit
// entries of the renumbered ids: entry = (block << mbits) | mask, bit i of the
// mask standing for id block * mbits + i.  Popular ids are in most lists and
// sit together, so a list's many popular ids share few entries (R-MAT 20:
// 0.81 entries per id over all rows, but 0.37 x the ids along the lists that
// the count streams), and the blocks that a probe looks for are mostly small
// numbers: 99 % of R-MAT 20's streamed entries are of the first 2048 blocks
// (kLow).  So
//   * a root's row is a table addressed by the block itself for blocks < kLow
//     (one 16-bit shared load per probe; a list's blocks ascend there, so a
//     warp's 32 loads fall in neighbouring words), with a small linear-probing
//     hash for the rest;
//   * a probe is one AND and half a popcount for up to 15 ids.
// Every root streams the lists of all its out-neighbours through its own table
// (W+ ids in the reference's terms).  Compared with choosing the shorter side
// per edge that is 1.0-2.4 x the entries, but there is no transpose of the
// edges (one atomic per edge, a scan, in-lists), a table is built once per
// root and none for the halo rows of a part, and a root's hits are one sum.
//
// Launch sequence (one CUDA-graph-capturable chain, plain or batched):
//   pop      in-degree of every vertex over the root rows (a sample of the edges
//            of large launches: only the order matters, and only roughly)
//   hist     per graph, a histogram of the popularities in 256 buckets
//            (exact below 16, then eight per octave)
//   assign   new id = bucket start + order of arrival; written as the entry of
//            that single id (block, one mask bit).  Lists the roots by length:
//            up to kRowMax entries are found by their chunk, longer ones up to
//            warp_max are listed, longer ones become block units
//   pack     rows to entries: gather the members' single-id entries and OR
//            those of one block together
//   count    persistent grid: block units, then listed rows one per warp, then
//            32-row chunks whose short rows are counted several at a time
//
// A graph of few edges skips the renumbering: single_kernel counts it in one
// launch on its own ids (entry = (id << 1) | 1).
#include <algorithm>

#include "tc_internal.h"

namespace tc {
namespace {

constexpr int kWarp = 32;
constexpr unsigned kFull = 0xffffffffu;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / kWarp;
constexpr int kRowMax = 32;         // roots of at most this out-degree are counted several per warp
constexpr int kBuckets = 256;       // popularity buckets
constexpr int kPopTile = 4096;      // edges per block of pop
constexpr int64_t kSampleEdges = 1 << 18;  // (R-MAT 16 125 us with 2^21, where it is not sampled, 116 so)
constexpr int kPopItems = kPopTile / kThreads;
constexpr uint32_t kHashMul = 0x9E3779B1u;

// The first kLow x 15 ids make the low blocks: entry (block << 16) | 15-bit mask,
// so that e >> 15 is the byte offset of the block's 16-bit mask in a table.  The
// other ids make the high blocks: entry ((id / mbits + 2^(27 - mbits)) << mbits) |
// mask with as many mask bits as the ids leave (pack_mask_bits), above every low
// entry.  Tables: the low blocks' masks, then a hash of whole high entries.
constexpr int kLow = 2048;                          // 4 KB of masks, 30,720 ids
constexpr int kLowBits = 15;
constexpr uint32_t kLowEnd = (uint32_t)kLow << 16;  // low entries are below it, high ones not
static_assert(kLowEnd == 1u << 27, "pack_mask_bits and assign_kernel place the high entries at 2^27");
constexpr int kLogWarpH = 8, kLogBlockH = 11;       // words of the hash, per warp and per block
constexpr int kWarpTile = 96, kBlockTile = 768;     // high entries of a root looked up at a time (filter_put)
constexpr int kWarpWords = kLow / 2 + (1 << kLogWarpH);
constexpr int kBlockWords = kLow / 2 + (1 << kLogBlockH);
static_assert(kBlockWords <= kWarps * kWarpWords, "the block table lies in the warps' tables");
constexpr int kPiece = 128, kSmallScan = 512;       // see pack_kernel

// Where a row's entries lie: quads of four entries (16 bytes, zero-padded), the
// high blocks' first, then the low blocks' in pairs of quads (octets).  Row x of
// a graph starts at quad (ebase + rp[x] + 13 (vbase + x) + 3) / 4, which leaves
// its d members and both paddings room: the high entries and their padding take
// at most (h + 3) / 4 quads, the low ones (l + 7) / 4, and consecutive starts
// differ by at least (d + 10) / 4.
//   The n low entries, ascending, are dealt to the row's octets like cards:
// octet j holds entries j, j + octets, j + 2 octets ..., so that the lanes of a
// warp, which take consecutive octets, look up consecutive entries (neighbouring
// words of the table: few bank conflicts) with each load of theirs.  The octets'
// first quads lie together, and so do their second ones: a warp's loads cover
// whole lines (octets of 32 bytes in place: twice the L1 wavefronts, R-MAT 21's
// streaming 3.3 ms instead of 2.6).
constexpr int kRowPad = 13;
__device__ __forceinline__ int64_t row_quad(int64_t e, int64_t v) { return (e + kRowPad * v + 3) >> 2; }

// Word of low entry i < 2048 + 8 among `octets` octets (octets <= 256: the
// quotient by a 20-bit reciprocal is exact, as i x its error < 2^20).
struct Deal {
    int octets;
    uint32_t inv;
    __device__ __forceinline__ explicit Deal(int n) : octets((n + 7) >> 3), inv(0) {
        if (octets) inv = ((1u << 20) + octets - 1) / (uint32_t)octets;
    }
    __device__ __forceinline__ int operator()(int i) const {
        const int k = (int)(((uint32_t)i * inv) >> 20);
        return 4 * ((k >> 2) * octets + i - k * octets) + (k & 3);
    }
};

struct PackParams {
    const GraphDesc *gd;
    int n_graphs;
    int64_t total_chunks, total_edges;
    CountWork *work;
    unsigned long long *results;
    uint32_t *code;      // per vertex (pooled): popularity, then the single-id entry
    uint32_t *hist;      // per graph: kBuckets counts, then kBuckets cursors
    uint4 *ent;          // the rows' entries, in quads at row_quad
    int4 *desc;          // per vertex (pooled): (first quad, quads of high blocks, octets of low blocks, entries)
    uint32_t *mid_list;  // roots for one warp each, as global rows chunk * 32 + lane
    uint2 *units;        // block units: (global row, slice)
    int zero_quad;       // a quad of ent past the rows', set to zeros
    int warp_max, slice;
    int rank_chunks;  // 32-row chunks per block of hist and assign
    int pack_rows;    // rows per warp of pack, and per grab of the short roots: a power of two, at most 32
};

__device__ __forceinline__ unsigned long long sum_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

__device__ __forceinline__ int warp_excl_scan(int v, int lane, int *total) {
    int x = v;
#pragma unroll
    for (int o = 1; o < kWarp; o <<= 1) {
        const int t = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += t;
    }
    *total = __shfl_sync(kFull, x, kWarp - 1);
    return x - v;
}

__device__ __forceinline__ int graph_of_chunk(const GraphDesc *gd, int n, int64_t chunk) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (gd[mid].chunk_base <= chunk) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ int graph_of_edge(const GraphDesc *gd, int n, int64_t e) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (gd[mid].ebase <= e) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Most popular first: bucket 255 - q, q exact below 16, then eight per octave.
__device__ __forceinline__ int pop_bucket(uint32_t pop) {
    if (pop < 16) return kBuckets - 1 - (int)pop;
    const int lg = 31 - __clz(pop);
    return kBuckets - 1 - (16 + (lg - 4) * 8 + (int)((pop >> (lg - 3)) & 7u));
}

// In-degrees over the root rows.  One block per tile of pooled edges; of a graph
// of at least kSampleEdges edges every fourth tile.
__global__ void __launch_bounds__(kThreads) pop_kernel(PackParams P) {
    int64_t t0 = (int64_t)blockIdx.x * kPopTile;
    const int64_t t1 = min(t0 + kPopTile, P.total_edges);
    while (t0 < t1) {
        const int g = graph_of_edge(P.gd, P.n_graphs, t0);
        const GraphDesc &G = P.gd[g];
        const int64_t next = g + 1 < P.n_graphs ? P.gd[g + 1].ebase : P.total_edges;
        const bool skip = next - G.ebase >= kSampleEdges && (blockIdx.x & 3) != 0;
        const int64_t n_root_edges = skip ? 0 : (int64_t)__ldg(G.rp + G.n_roots);
        const int64_t a = t0 - G.ebase, b = min(t1 - G.ebase, n_root_edges);
        const int32_t *__restrict__ col = G.col;
        uint32_t *pop = P.code + G.vbase;
        int v[kPopItems];
#pragma unroll
        for (int i = 0; i < kPopItems; ++i) {
            const int64_t j = a + i * kThreads + threadIdx.x;
            v[i] = j < b ? __ldg(col + j) : -1;
        }
#pragma unroll
        for (int i = 0; i < kPopItems; ++i)
            if (v[i] >= 0) atomicAdd(pop + v[i], 1u);
        t0 = next;  // past t0: a graph without edges is never found
    }
}

// The rows of one graph among a block's chunks [c, c_end).
struct RowSpan {
    int g;
    int64_t x0, x1, next;
};
__device__ __forceinline__ RowSpan row_span(const PackParams &P, int64_t c, int64_t c_end) {
    RowSpan s;
    s.g = graph_of_chunk(P.gd, P.n_graphs, c);
    const GraphDesc &G = P.gd[s.g];
    s.next = min(c_end, G.chunk_base + (G.n_rows + kWarp - 1) / kWarp);
    s.x0 = (c - G.chunk_base) * kWarp;
    s.x1 = min(G.n_rows, (s.next - G.chunk_base) * kWarp);
    return s;
}

__global__ void __launch_bounds__(kThreads) hist_kernel(PackParams P) {
    __shared__ uint32_t cnt[kBuckets];
    int64_t c = (int64_t)blockIdx.x * P.rank_chunks;
    const int64_t c_end = min(c + P.rank_chunks, P.total_chunks);
    while (c < c_end) {
        const RowSpan s = row_span(P, c, c_end);
        cnt[threadIdx.x] = 0;
        __syncthreads();
        const uint32_t *pop = P.code + P.gd[s.g].vbase;
        for (int64_t x = s.x0 + threadIdx.x; x < s.x1; x += kThreads) atomicAdd(&cnt[pop_bucket(pop[x])], 1u);
        __syncthreads();
        if (cnt[threadIdx.x]) atomicAdd(P.hist + (int64_t)s.g * 2 * kBuckets + threadIdx.x, cnt[threadIdx.x]);
        c = s.next;
    }
}

__global__ void __launch_bounds__(kThreads) assign_kernel(PackParams P) {
    __shared__ uint32_t cnt[kBuckets];
    __shared__ int wsum[kWarps];
    __shared__ unsigned s_mid, s_unit;
    const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
    int64_t c = (int64_t)blockIdx.x * P.rank_chunks;
    const int64_t c_end = min(c + P.rank_chunks, P.total_chunks);
    while (c < c_end) {
        const RowSpan s = row_span(P, c, c_end);
        const GraphDesc &G = P.gd[s.g];
        const int mb = G.mbits;
        uint32_t *code = P.code + G.vbase;
        const int32_t *__restrict__ rp = G.rp;
        cnt[threadIdx.x] = 0;
        if (threadIdx.x == 0) s_mid = s_unit = 0;
        __syncthreads();
        for (int64_t x = s.x0 + threadIdx.x; x < s.x1; x += kThreads) {
            atomicAdd(&cnt[pop_bucket(code[x])], 1u);
            const int d = x < G.n_roots ? __ldg(rp + x + 1) - __ldg(rp + x) : 0;
            if (d > P.warp_max) atomicAdd(&s_unit, (unsigned)((d + P.slice - 1) / P.slice));
            else if (d > kRowMax) atomicAdd(&s_mid, 1u);
        }
        // bucket starts: an exclusive scan of the graph's histogram, one bucket per thread
        uint32_t *hist = P.hist + (int64_t)s.g * 2 * kBuckets;
        const int h = (int)hist[threadIdx.x];
        int tot;
        int start = warp_excl_scan(h, lane, &tot);
        if (lane == 0) wsum[warp] = tot;
        __syncthreads();
        for (int w = 0; w < warp; ++w) start += wsum[w];
        const uint32_t mine = cnt[threadIdx.x];
        const uint32_t base = mine ? atomicAdd(hist + kBuckets + threadIdx.x, mine) : 0;
        cnt[threadIdx.x] = (uint32_t)start + base;
        if (threadIdx.x == 0) {
            if (s_mid) s_mid = (unsigned)atomicAdd(&P.work->n_tasks, (unsigned long long)s_mid);
            if (s_unit) s_unit = (unsigned)atomicAdd(&P.work->heavy_packed, (unsigned long long)s_unit);
        }
        __syncthreads();
        for (int64_t x = s.x0 + threadIdx.x; x < s.x1; x += kThreads) {
            const uint32_t id = atomicAdd(&cnt[pop_bucket(code[x])], 1u);
            const bool low = id < (uint32_t)(kLow * kLowBits);
            const uint32_t bits = low ? (uint32_t)kLowBits : (uint32_t)mb;
            const uint32_t blk = id / bits, bit = 1u << (id - blk * bits);
            code[x] = low ? (blk << 16) | bit : kLowEnd + (blk << mb) + bit;
            const int d = x < G.n_roots ? __ldg(rp + x + 1) - __ldg(rp + x) : 0;
            const uint32_t row = (uint32_t)(G.chunk_base * kWarp + x);
            if (d > P.warp_max) {
                const int n = (d + P.slice - 1) / P.slice;
                const unsigned o = atomicAdd(&s_unit, (unsigned)n);
                for (int i = 0; i < n; ++i) P.units[o + i] = make_uint2(row, (uint32_t)i);
            } else if (d > kRowMax) {
                P.mid_list[atomicAdd(&s_mid, 1u)] = row;
            }
        }
        __syncthreads();  // cnt and the counters are reused by the next graph's rows
        c = s.next;
    }
}

// Rows to entries, a warp for pack_rows rows.  Rows of at most 32 members: whole
// rows are laid side by side in windows of at most 32 members, one lane each,
// and the lanes of one row with one block merge their bits (__match_any_sync).
// Longer rows, kPiece members at a time: the low blocks' bits are ORed into masks
// by block, the high ones go out as they are (their blocks, without hubs, seldom
// meet: hashing them to merge their bits cost more than the whole row's other
// work, R-MAT 23's eight parts 10.1 ms of packing, 6.4 without).  Then the masks
// are scanned in order and the non-empty ones dealt out, so that the entries
// ascend; a row of at most kPiece members scans the first kSmallScan blocks and
// lists the others as it meets them, since scanning 2048 blocks for 100 members
// would be most of its work.
__global__ void __launch_bounds__(kThreads, 5) pack_kernel(PackParams P) {
    __shared__ __align__(16) uint32_t s_dir[kWarps][kLow / 2];
    __shared__ uint16_t s_list[kWarps][kPiece];
    __shared__ int4 s_row[kWarps][kWarp];
    const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
    uint32_t *dir = s_dir[warp];
    for (int i = lane; i < kLow / 2; i += kWarp) dir[i] = 0;
    __syncwarp();
    if (blockIdx.x == 0 && threadIdx.x == 0) P.ent[(uint32_t)P.zero_quad] = make_uint4(0, 0, 0, 0);
    const uint32_t le = kFull >> (31 - lane), lt = le >> 1;
    const int per = kWarp / P.pack_rows;  // grabs per 32-row chunk
    for (;;) {
        unsigned grab = 0;
        if (lane == 0) grab = atomicAdd(&P.work->aux_cursor[1], 1u);
        const int64_t i0 = (int64_t)__shfl_sync(kFull, grab, 0);
        if (i0 >= P.total_chunks * per) break;
        const int64_t c = i0 / per;
        const GraphDesc &G = P.gd[graph_of_chunk(P.gd, P.n_graphs, c)];
        const int32_t *__restrict__ col = G.col;
        const uint32_t *__restrict__ code = P.code + G.vbase;
        const int mb = G.mbits;
        const int64_t x = (c - G.chunk_base) * kWarp + (i0 - c * per) * P.pack_rows + lane;
        const bool row = lane < P.pack_rows && x < G.n_rows;
        int rs = 0, d = 0;
        int64_t q0 = 0;
        if (row) {
            rs = __ldg(G.rp + x);
            d = __ldg(G.rp + x + 1) - rs;
            q0 = row_quad(G.ebase + rs, G.vbase + x);
        }
        int4 *desc = P.desc + G.vbase + x;
        const bool shrt = mb >= 5 && d <= kWarp;  // with fewer bits a row and a block do not fit the match's key
        const int sd = shrt ? d : 0;
        int total;
        const int excl = warp_excl_scan(sd, lane, &total);
        if (row && d == 0) *desc = make_int4((int)q0, 0, 0, 0);
        for (int pos = 0; pos < total;) {
            const int off = excl - pos;
            const bool in = sd > 0 && off >= 0 && off + sd <= kWarp;
            const uint32_t starts = __reduce_or_sync(kFull, in ? 1u << off : 0u);
            const int wlen = __reduce_max_sync(kFull, in ? off + sd : 0);
            if (in) s_row[warp][off] = make_int4(rs - off, (int)q0, (int)x, 0);
            __syncwarp();
            uint32_t e = 0;
            int ss = 0;
            int4 r = make_int4(0, 0, 0, 0);
            if (lane < wlen) {
                ss = 31 - __clz(starts & le);
                r = s_row[warp][ss];
                const int v = __ldg(col + r.x + lane);
                if (v == r.z) P.work->self_loops = 1;
                e = __ldg(code + v);
            }
            const bool low = e < kLowEnd;
            // lanes of one row and one block (a high block's number is at least 2^(27 - mb) >= kLow)
            const uint32_t key = ((uint32_t)ss << (32 - mb)) | (low ? e >> 16 : e >> mb);
            const uint32_t peers = __match_any_sync(kFull, lane < wlen ? key : 0xffffffffu - (uint32_t)lane);
            const bool lead = lane < wlen && (peers & lt) == 0;
            uint32_t rest = peers & ~(1u << lane);
            const int more = __reduce_max_sync(kFull, lane < wlen ? __popc(rest) : 0);
            uint32_t m = e;
            for (int i = 0; i < more; ++i) {
                const int src = rest ? __ffs(rest) - 1 : lane;
                m |= __shfl_sync(kFull, e, src);
                rest &= rest - 1u;
            }
            const uint32_t lows = __ballot_sync(kFull, lead && low), highs = __ballot_sync(kFull, lead && !low);
            if (lead) {
                const uint32_t before = lt & ~((1u << ss) - 1u);
                const uint32_t later = starts & ~le;  // the next row's first lane ends this one
                const uint32_t mine = ~((1u << ss) - 1u) & (later ? (later & (0u - later)) - 1u : kFull);
                const int at = low ? ((__popc(highs & mine) + 3) & ~3) + Deal(__popc(lows & mine))(__popc(lows & before))
                                   : __popc(highs & before);
                reinterpret_cast<uint32_t *>(P.ent + (uint32_t)r.y)[at] = m;
            }
            if (in) {
                const uint32_t seg = (sd == kWarp ? kFull : (1u << sd) - 1u) << off;
                const int nh = __popc(highs & seg), nl = __popc(lows & seg);
                const int hq = (nh + 3) >> 2;
                const Deal deal(nl);
                uint32_t *out = reinterpret_cast<uint32_t *>(P.ent + q0);
                for (int i = nh; i < 4 * hq; ++i) out[i] = 0;
                for (int i = nl; i < 8 * deal.octets; ++i) out[4 * hq + deal(i)] = 0;
                *desc = make_int4((int)q0, hq, deal.octets, nh + nl);
            }
            __syncwarp();  // s_row is rewritten
            pos += wlen;
        }
        for (unsigned todo = __ballot_sync(kFull, d > 0 && !shrt); todo; todo &= todo - 1u) {
            const int k = __ffs(todo) - 1;
            const int rrs = __shfl_sync(kFull, rs, k), rd = __shfl_sync(kFull, d, k);
            const int64_t rq = __shfl_sync(kFull, q0, k);
            const uint32_t rx = (uint32_t)__shfl_sync(kFull, (int)x, k);
            uint32_t *out = reinterpret_cast<uint32_t *>(P.ent + rq);
            const bool small = rd <= kPiece;
            const int dn = small ? kSmallScan : kLow;  // blocks scanned in order; a small row lists its others
            int o = 0, nl = 0, n_list = 0;  // high entries written; low blocks of this lane; blocks listed
            for (int p0 = 0; p0 < rd; p0 += kPiece) {
                const int p1 = min(rd, p0 + kPiece);
                uint32_t e[kPiece / kWarp];
#pragma unroll
                for (int q = 0; q < kPiece / kWarp; ++q) {
                    const int i = p0 + q * kWarp + lane;
                    e[q] = i < p1 ? (uint32_t)__ldg(col + rrs + i) : kFull;
                }
#pragma unroll
                for (int q = 0; q < kPiece / kWarp; ++q) {
                    if (e[q] == rx) P.work->self_loops = 1;
                    e[q] = e[q] != kFull ? __ldg(code + e[q]) : 0u;
                }
#pragma unroll
                for (int q = 0; q < kPiece / kWarp; ++q) {
                    if (p0 + q * kWarp >= rd) break;  // warp-uniform
                    const uint32_t blk = e[q] >> 16;
                    const bool high = e[q] >= kLowEnd;
                    bool list = false;
                    if (e[q] && !high) {
                        const int half = (int)(blk & 1u) * 16;
                        const uint32_t old = atomicOr(dir + (blk >> 1), (e[q] & 0xffffu) << half);
                        const bool fresh = ((old >> half) & 0xffffu) == 0;
                        nl += (int)fresh;
                        list = fresh && blk >= (uint32_t)dn;
                    }
                    const uint32_t bh = __ballot_sync(kFull, high);
                    if (high) out[o + __popc(bh & lt)] = e[q];
                    o += __popc(bh);
                    if (small) {
                        const uint32_t b = __ballot_sync(kFull, list);
                        if (list) s_list[warp][n_list + __popc(b & lt)] = (uint16_t)blk;
                        n_list += __popc(b);
                    }
                }
            }
            __syncwarp();
            const int hq = (o + 3) >> 2;
            if (lane < 4 * hq - o) out[o + lane] = 0;
            // the low entries, ascending, eight blocks per lane at a time
            nl = __reduce_add_sync(kFull, nl);
            const Deal deal(nl);
            uint32_t *lrow = out + 4 * hq;
            int at = 0;
            for (int w0 = 0; w0 < dn / 8; w0 += kWarp) {
                const int w = w0 + lane;
                uint4 *d4 = reinterpret_cast<uint4 *>(dir) + w;
                uint4 v = make_uint4(0, 0, 0, 0);
                if (w < dn / 8) v = *d4;
                uint32_t f = 0;  // bit i: block 8 w + i is there (a mask's top bit is 0: no carry between the halves)
                const uint32_t vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t t = vs[i] + 0x7fff7fffu;
                    f |= (((t >> 15) & 1u) | ((t >> 30) & 2u)) << (2 * i);
                }
                int tot;
                int i = at + warp_excl_scan(__popc(f), lane, &tot);
                at += tot;
                if (tot == 0) continue;
                const bool any = f != 0;
                for (; f; f &= f - 1u) {
                    const int b = 8 * w + __ffs(f) - 1;
                    lrow[deal(i++)] = ((uint32_t)b << 16) | reinterpret_cast<const uint16_t *>(dir)[b];
                }
                asm volatile("" ::: "memory");  // halves are read, whole words cleared: not to be taken for others
                if (any) *d4 = make_uint4(0, 0, 0, 0);
            }
            for (int w = lane; w < n_list; w += kWarp) {
                const int b = s_list[warp][w];
                uint16_t *m = reinterpret_cast<uint16_t *>(dir) + b;
                lrow[deal(at + w)] = ((uint32_t)b << 16) | *m;
                *m = 0;
            }
            if (lane < 8 * deal.octets - nl) lrow[deal(nl + lane)] = 0;
            if (lane == k) *desc = make_int4((int)rq, hq, deal.octets, o + nl);
            __syncwarp();
        }
    }
}

// ---- counting ------------------------------------------------------------------
// Where rows and entries of the graph at hand lie.  Packed: quads in ent, places
// in desc.  Raw (no renumbering): entry (id << 1) | 1 made from col, a row's
// members all taken as high blocks.
template <bool kRaw>
struct Rows {
    const int32_t *__restrict__ rp;
    const int32_t *__restrict__ col;
    const int4 *__restrict__ desc;
    const uint4 *__restrict__ ent;
    int mb, zero;  // zero: a quad of zeros
    __device__ __forceinline__ int4 row(int v) const {  // as desc; raw: the first member instead of the quad
        if (kRaw) {
            const int s = __ldg(rp + v), n = __ldg(rp + v + 1) - s;
            return make_int4(s, (n + 3) >> 2, 0, n);
        }
        return __ldg(desc + v);
    }
    // Quad i from `first` on; raw: of the members below `end`.
    __device__ __forceinline__ uint4 quad(int first, int i, int end) const {
        if (kRaw) {
            uint32_t e[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int j = first + 4 * i + q;
                e[q] = j < end ? ((uint32_t)__ldg(col + j) << 1) | 1u : 0u;
            }
            return make_uint4(e[0], e[1], e[2], e[3]);
        }
        return __ldg(ent + ((uint32_t)first + (uint32_t)i));  // offsets wrap in 32 bits
    }
    __device__ __forceinline__ uint4 at(int quad) const { return __ldg(ent + (uint32_t)quad); }
    __device__ __forceinline__ int bits() const { return kRaw ? 1 : mb; }
};

template <bool kRaw>
__device__ __forceinline__ Rows<kRaw> rows_of(const PackParams &P, const GraphDesc &G) {
    Rows<kRaw> R;
    R.rp = G.rp;
    R.col = G.col;
    R.desc = P.desc + G.vbase;
    R.ent = P.ent;
    R.mb = G.mbits;
    R.zero = P.zero_quad;
    return R;
}

template <class F>
__device__ __forceinline__ void each4(uint4 q, F f) {
    f(q.x);
    f(q.y);
    f(q.z);
    f(q.w);
}

// e (0: none) into a linear-probing hash of mask + 1 places, not all of them
// taken, from place p on.  All lanes of the warp call it, and they probe in step,
// as in the look-ups below: after loops of their own the lanes went on in two
// groups through all the code behind, every instruction issued twice (R-MAT 21's
// listed roots 2.25 instead of 1.2 ms).
__device__ __forceinline__ void place(uint32_t *tab, uint32_t mask, uint32_t p, int mb, uint32_t e) {
    bool open = e != 0u;
    // (the bound is the largest hash's, the same for all lanes: their hashes may differ in size)
    for (int left = 1 << kLogBlockH; left && __any_sync(kFull, open); --left) {
        if (open) {
            const uint32_t old = atomicCAS(tab + p, 0u, e);
            const bool same = ((old ^ e) >> mb) == 0;
            if (same) atomicOr(tab + p, e);
            open = old != 0u && !same;
            p = (p + 1u) & mask;
        }
    }
}

// ... of 2^lg places by the top bits of the block's hash.
__device__ __forceinline__ void hash_put(uint32_t *hs, int lg, int mb, uint32_t e) {
    place(hs, (1u << lg) - 1u, ((e >> mb) * kHashMul) >> (32 - lg), mb, e);
}

// A row's low blocks are all different (pack_kernel), so plain stores put them.
__device__ __forceinline__ void low_put(uint32_t *words, uint32_t e, bool in = true) {
    if (e) reinterpret_cast<uint16_t *>(words)[e >> 16] = in ? (uint16_t)e : (uint16_t)0;
}

// Members that a quad's entries share with such a hash.  (An absent entry looks
// nowhere: it may come without a table.)
__device__ __forceinline__ uint32_t hash_hits(const uint32_t *hs, int lg, int mb, uint4 q) {
    const uint32_t e[4] = {q.x, q.y, q.z, q.w};
    const uint32_t mask = (1u << lg) - 1u;
    uint32_t n = 0, left = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t m = e[i] ? hs[((e[i] >> mb) * kHashMul) >> (32 - lg)] : 0u;
        if (((m ^ e[i]) >> mb) == 0) n += __popc(m & e[i] & ((1u << mb) - 1u));
        else if (m) left |= 1u << i;
    }
    uint32_t step = 1;  // places past the first one
    while (__any_sync(kFull, left != 0)) {
        if (left) {
            const int i = __ffs(left) - 1;
            const uint32_t x = i == 0 ? e[0] : i == 1 ? e[1] : i == 2 ? e[2] : e[3];
            const uint32_t m = hs[((((x >> mb) * kHashMul) >> (32 - lg)) + step) & mask];
            const bool match = ((m ^ x) >> mb) == 0;
            if (match) n += __popc(m & x & ((1u << mb) - 1u));
            ++step;
            if (match || m == 0u || step > mask) {
                left &= left - 1u;
                step = 1;
            }
        }
    }
    return n;
}

// A longer root's high entries: a filter of 2^lg words, one bit per block by its
// hash, and behind it a hash of 2^lg places, at most three quarters of them
// taken.  Most streamed entries' blocks are not there, and the filter says so
// with one load and no loop; the few others are looked up.
__device__ __forceinline__ void filter_put(uint32_t *hs, int lg, int mb, uint32_t e) {
    const uint32_t h = (e >> mb) * kHashMul, mask = (1u << lg) - 1u;
    if (e) atomicOr(hs + (h >> (32 - lg)), 1u << ((h >> (27 - lg)) & 31u));
    place(hs + (1 << lg), mask, (h >> 5) & mask, mb, e);
}
__device__ __forceinline__ uint32_t filter_hits(const uint32_t *hs, int lg, int mb, uint4 q) {
    const uint32_t e[4] = {q.x, q.y, q.z, q.w};
    uint32_t n = 0, there = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t h = (e[i] >> mb) * kHashMul;
        const uint32_t w = hs[h >> (32 - lg)];
        there |= (e[i] ? (w >> ((h >> (27 - lg)) & 31u)) & 1u : 0u) << i;
    }
    const uint32_t *tab = hs + (1 << lg);
    const uint32_t mask = (1u << lg) - 1u;
    uint32_t step = 0;
    while (__any_sync(kFull, there != 0)) {  // in step, as above
        if (there) {
            const int i = __ffs(there) - 1;
            const uint32_t x = i == 0 ? e[0] : i == 1 ? e[1] : i == 2 ? e[2] : e[3];
            const uint32_t m = tab[((((x >> mb) * kHashMul) >> 5) + step) & mask];
            const bool match = ((m ^ x) >> mb) == 0;
            if (match) n += __popc(m & x & ((1u << mb) - 1u));
            ++step;
            if (match || m == 0u || step > mask) {
                there &= there - 1u;
                step = 0;
            }
        }
    }
    return n;
}

// Members that a quad's entries, all of low blocks, share with the masks.
__device__ __forceinline__ uint32_t low_mask(const uint32_t *words, uint32_t e) {
    return *reinterpret_cast<const uint16_t *>(reinterpret_cast<const char *>(words) + (e >> 15)) & e;
}
__device__ __forceinline__ uint32_t low_hits(const uint32_t *words, uint4 q) {
    return __popc(low_mask(words, q.x) | (low_mask(words, q.y) << 16)) +
           __popc(low_mask(words, q.z) | (low_mask(words, q.w) << 16));
}

// Up to 32 lists (one per lane: n steps, of one quad each from quad `first` on,
// or of an octet's two, n quads apart; raw: of members below `end`) laid end to
// end.  ListAt, per warp and list that is not empty: its first quad less its
// place, and the octets or the caller's word.
template <bool kRaw>
struct alignas(8) ListAt {
    int off, x;
};
template <>
struct alignas(4) ListAt<true> {
    int off, x, end;
};
struct ListSpan {
    int excl, total;  // the lane's list's place (out of reach when it has none); steps in all
    unsigned have;    // lanes with a list
};
constexpr int kNoList = 0x7fffffff;
template <bool kRaw>
__device__ __forceinline__ ListSpan span_lists(int n, int first, int end, int x, int lane, ListAt<kRaw> *s_at) {
    ListSpan s;
    s.excl = warp_excl_scan(n, lane, &s.total);
    s.have = __ballot_sync(kFull, n > 0);
    if (n > 0) {
        ListAt<kRaw> a;
        a.off = first - (kRaw ? 4 : 1) * s.excl;
        a.x = x;
        if constexpr (kRaw) a.end = end;
        s_at[__popc(s.have & ((1u << lane) - 1u))] = a;
    }
    return s;
}

// Walks a span's steps, one per lane at a time.  load(b, b1) loads the steps
// [b, min(b1, b + 32)): the lists' first steps mark a bit each, and a lane's
// list is k + the number of marks up to it (k: lists begun before b, less one).
// Rounds come in order and end at lists' ends or at full warps, so k moves on by
// the marks below b1.
template <bool kRaw, int kStep, bool kWord = false>
struct ListWalk {
    const Rows<kRaw> &R;
    const ListAt<kRaw> *s_at;
    int lane, mark, k;  // mark: the lane's list's place, kNoList without one
    __device__ __forceinline__ ListWalk(const Rows<kRaw> &R, const ListSpan &s, int lane, const ListAt<kRaw> *s_at)
        : R(R), s_at(s_at), lane(lane), mark((s.have >> lane) & 1u ? s.excl : kNoList), k(-1) {}
    __device__ __forceinline__ void load(int b, int b1, uint4 (&q)[kStep], int &w) {
        const int o = mark - b;
        const uint32_t starts =
            __reduce_or_sync(kFull, (unsigned)o < (unsigned)min(kWarp, b1 - b) ? 1u << o : 0u);
        const int t = b + lane;
        const int at = k + __popc(starts & (kFull >> (31 - lane)));
        if constexpr (kRaw) {
            q[0] = make_uint4(0, 0, 0, 0);
            if (t < b1) {
                const ListAt<true> a = s_at[at];
                if constexpr (kWord) w = a.x;
                q[0] = R.quad(a.off, t, a.end);
            }
        } else {
            // (a lane past b1 has the last list's place and loads the quad of zeros)
            const ListAt<false> a = s_at[at];
            if constexpr (kWord) w = a.x;
            const bool in = t < b1;
            q[0] = R.at(in ? a.off + t : R.zero);
            if constexpr (kStep == 2) q[1] = R.at(in ? a.off + t + a.x : R.zero);
        }
        k += __popc(starts);
    }
    // The steps [b0, b1); f gets their quads.  The next round's loads go out
    // before this round's look-ups.
    template <class F>
    __device__ __forceinline__ void run(int b0, int b1, F f) {
        if (b0 >= b1) return;
        uint4 p[kStep], q[kStep];
        int pw = 0, qw = 0;
        auto use = [&](uint4 (&c)[kStep], int w) {
#pragma unroll
            for (int i = 0; i < kStep; ++i) {
                if constexpr (kWord) f(c[i], w);
                else f(c[i]);
            }
        };
        load(b0, b1, p, pw);
        for (int b = b0;;) {
            b += kWarp;
            if (b < b1) load(b, b1, q, qw);
            use(p, pw);
            if (b >= b1) break;
            b += kWarp;
            if (b < b1) load(b, b1, p, pw);
            use(q, qw);
            if (b >= b1) break;
        }
    }
};

template <bool kRaw, int kStep, class F>
__device__ __forceinline__ void flat_lists(const Rows<kRaw> &R, int first, int n, int end, int lane,
                                           ListAt<kRaw> *s_at, F f) {
    const ListSpan s = span_lists<kRaw>(n, first, end, n, lane, s_at);
    __syncwarp();
    ListWalk<kRaw, kStep> W(R, s, lane, s_at);
    W.run(0, s.total, f);
    __syncwarp();  // s_at is rewritten by the next call
}

// Streams the lists of up to 32 partners (one per lane, id p or -1) through a
// table (words: kLow / 2 words of masks; hs: a filter and hash of 2^lg words each), the low
// blocks' and the high blocks' quads apart.
template <bool kRaw>
__device__ __forceinline__ uint32_t stream_lists(const Rows<kRaw> &R, int p, const uint32_t *words, const uint32_t *hs, int lg, bool low,
                                                 bool high, int lane, ListAt<kRaw> *s_at) {
    uint32_t hits = 0;
    const int mb = R.bits();
    int4 l = make_int4(0, 0, 0, 0);
    if (p >= 0) l = R.row(p);
    if (high)
        flat_lists<kRaw, 1>(R, l.x, l.y, l.x + l.w, lane, s_at,
                            [&](uint4 q) { hits += kRaw ? hash_hits(hs, lg + 1, mb, q) : filter_hits(hs, lg, mb, q); });
    if (!kRaw && low)
        flat_lists<kRaw, 2>(R, l.x + l.y, l.z, 0, lane, s_at, [&](uint4 q) { hits += low_hits(words, q); });
    return hits;
}

// One root x of out-degree d > kRowMax on one warp; its high blocks' entries in
// hashes of at most kWarpTile of them at a time.
template <bool kRaw>
__device__ __forceinline__ uint32_t warp_row(const Rows<kRaw> &R, int x, int rs, int d, int lane, uint32_t *words,
                                             uint32_t *hs, ListAt<kRaw> *s_at) {
    const int4 l = R.row(x);
    const int mb = R.bits();
    uint32_t hits = 0;
    int t0 = 0;
    do {
        if (!kRaw && t0 == 0)
            for (int i = lane; i < kLow / 8; i += kWarp) reinterpret_cast<uint4 *>(words)[i] = make_uint4(0, 0, 0, 0);
        for (int i = lane; i < (1 << kLogWarpH) / 4; i += kWarp)
            reinterpret_cast<uint4 *>(hs)[i] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        const int t1 = min(l.y, t0 + kWarpTile / 4);
        for (int i0 = t0; i0 < t1; i0 += kWarp) {
            const int i = i0 + lane;
            each4(i < t1 ? R.quad(l.x, i, l.x + l.w) : make_uint4(0, 0, 0, 0),
                  [&](uint32_t e) {
                      if (kRaw) hash_put(hs, kLogWarpH, mb, e);
                      else filter_put(hs, kLogWarpH - 1, mb, e);
                  });
        }
        if (!kRaw && t0 == 0)
            for (int i = lane; i < 2 * l.z; i += kWarp)
                each4(R.quad(l.x, l.y + i, 0), [&](uint32_t e) { low_put(words, e); });
        __syncwarp();
        for (int j = 0; j < d; j += kWarp)
            hits += stream_lists<kRaw>(R, j + lane < d ? __ldg(R.col + rs + j + lane) : -1, words, hs, kLogWarpH - 1, t0 == 0,
                                       t1 > t0, lane, s_at);
        __syncwarp();
        t0 = t1;
    } while (t0 < l.y);
    return hits;
}

// The short roots (out-degree at most kRowMax) among up to 32 consecutive rows,
// one per lane (out-degree d at rs, 0 when it has none to count).  Whole roots
// are laid side by side in windows of at most 32 out-neighbours, one lane per
// out-neighbour, so that one round of loads brings the places of all their
// lists.  The high blocks of the window's roots go into a small hash per root in
// the warp's hs, and all their lists' high quads are streamed end to end, each
// against its root's hash.  The low blocks' lists are streamed root by root, each
// through the warp's masks, which hold only that root's entries (put before and
// taken out after it: few, where clearing the masks would write 4 KB).
template <bool kRaw>
struct alignas(16) ShortState {
    // per root of the window: rs - its first lane; row().x; row().w; low octets | high quads << 8 | its row's
    // lane << 16.  Raw roots may have one member, packed ones have at least two.
    int4 row[kRaw ? kWarp : kWarp / 2];
    int tab[kRaw ? kWarp : kWarp / 2];  // its hash: first place | log2 places << 16 | the root's number << 24
    int cnt[kRaw ? kWarp : kWarp / 2];  // its hits among the high blocks (per-root counts)
};
template <bool kRaw, bool kPerRoot>
__device__ __forceinline__ uint32_t short_rows(const Rows<kRaw> &R, int64_t x, int rs, int d, int lane,
                                               uint32_t *words, uint32_t *hs, ShortState<kRaw> &S,
                                               ListAt<kRaw> *s_low,
                                               ListAt<kRaw> *s_high, unsigned long long *per_root) {
    uint32_t acc = 0;
    const int mb = R.bits();
    const uint32_t le = kFull >> (31 - lane);
    int total;
    const int excl = warp_excl_scan(d, lane, &total);
    int4 l = make_int4(0, 0, 0, 0);
    if (d > 0) l = R.row((int)x);
    for (int pos = 0; pos < total;) {
        const int off = excl - pos;
        const bool in = d > 0 && off >= 0 && off + d <= kWarp;
        const uint32_t starts = __reduce_or_sync(kFull, in ? 1u << off : 0u);
        const int wlen = __reduce_max_sync(kFull, in ? off + d : 0);
        // the roots' hashes: four places per high entry, rounded up to a power of two (fewer than 8 per member:
        // at most 256 in all)
        const int lg = in && l.y > 0 ? 32 - __clz(4 * min(4 * l.y, l.w) - 1) : 0;
        int places;
        const int tb = warp_excl_scan(lg ? 1 << lg : 0, lane, &places);
        if (in) {
            const int i = __popc(starts & ((1u << off) - 1u));
            S.row[i] = make_int4(rs - off, l.x, l.w, l.z | (l.y << 8) | (lane << 16));
            S.tab[i] = tb | (lg << 16) | (i << 24);
            if (kPerRoot) S.cnt[i] = 0;
        }
        __syncwarp();
        int4 pl = make_int4(0, 0, 0, 0);
        uint4 mine = make_uint4(0, 0, 0, 0);  // a quad of the low blocks of this lane's root (it has no more than lanes)
        uint4 high = make_uint4(0, 0, 0, 0);  // ... and of the high ones
        int tab = 0, low0 = 0;
        if (lane < wlen) {
            const int i_root = __popc(starts & le) - 1;
            const int4 r = S.row[i_root];
            tab = S.tab[i_root];
            const int i = lane - (31 - __clz(starts & le)), lq = r.w & 0xff, hq = (r.w >> 8) & 0xff;
            const int p = __ldg(R.col + r.x + lane);
            if (i < 2 * lq) mine = R.quad(r.y + hq, i, 0);
            if (i < hq) high = R.quad(r.y, i, r.y + r.z);
            pl = R.row(p);
            low0 = pl.x + pl.y;
            if (lq == 0) pl.z = 0;  // nothing to find there
            if (hq == 0) pl.y = 0;
        }
        const ListSpan lo = span_lists<kRaw>(kRaw ? 0 : pl.z, low0, 0, pl.z, lane, s_low);
        const ListSpan hi = span_lists<kRaw>(pl.y, pl.x, pl.x + pl.w, tab, lane, s_high);
        __syncwarp();
        if (hi.total > 0) {
            for (int i = lane; i < places; i += kWarp) hs[i] = 0;
            __syncwarp();
            each4(high, [&](uint32_t e) { hash_put(hs + (tab & 0xffff), (tab >> 16) & 31, mb, e); });
            __syncwarp();
            ListWalk<kRaw, 1, true> H(R, hi, lane, s_high);
            H.run(0, hi.total, [&](uint4 q, int w) {
                const uint32_t hit = hash_hits(hs + (w & 0xffff), (w >> 16) & 31, mb, q);
                acc += hit;
                if (kPerRoot && hit) atomicAdd(&S.cnt[w >> 24], (int)hit);
            });
            __syncwarp();
        }
        // The next root's first round of loads goes out before the last look-ups of the root before.
        ListWalk<kRaw, kRaw ? 1 : 2> W(R, lo, lane, s_low);
        uint4 q[kRaw ? 1 : 2];
        int word = 0;
        if constexpr (!kRaw) {
            const uint32_t rest = starts & (starts - 1u);
            const int end = rest ? __shfl_sync(kFull, lo.excl, __ffs(rest) - 1) : lo.total;
            if (end > 0) W.load(0, end, q, word);
        }
        int i_root = 0;
        for (uint32_t todo = kPerRoot || lo.total > 0 ? starts : 0u; todo; ++i_root) {
            const int a = __ffs(todo) - 1;  // the root's lanes [a, b), the next one's [b, b2)
            todo &= todo - 1u;
            const int b = todo ? __ffs(todo) - 1 : wlen;
            const uint32_t todo2 = todo & (todo - 1u);
            const int b2 = todo2 ? __ffs(todo2) - 1 : wlen;
            uint32_t hits = 0;
            if constexpr (!kRaw) {
                const int lo0 = __shfl_sync(kFull, lo.excl, a);
                const int lo1 = b < kWarp ? __shfl_sync(kFull, lo.excl, b & 31) : lo.total;
                const int lo2 = b2 < kWarp ? __shfl_sync(kFull, lo.excl, b2 & 31) : lo.total;
                if (lo1 > lo0) {
                    const bool own = lane >= a && lane < b;
                    if (own) each4(mine, [&](uint32_t e) { low_put(words, e); });
                    __syncwarp();
                    for (int q0 = lo0; q0 < lo1; q0 += kWarp) {
                        const uint4 c0 = q[0], c1 = q[1];
                        if (q0 + kWarp < lo1) W.load(q0 + kWarp, lo1, q, word);
                        else if (lo2 > lo1) W.load(lo1, lo2, q, word);
                        hits += low_hits(words, c0) + low_hits(words, c1);
                    }
                    __syncwarp();
                    if (own) each4(mine, [&](uint32_t e) { low_put(words, e, false); });
                    __syncwarp();  // the next root's entries go in
                } else if (lo2 > lo1) {
                    W.load(lo1, lo2, q, word);  // no round of this root did it
                }
            }
            const int4 r = S.row[i_root];
            if (kPerRoot) {
                const unsigned s = __reduce_add_sync(kFull, hits);
                const unsigned t = s + (unsigned)S.cnt[i_root];
                if (lane == (r.w >> 16) && t) per_root[x] = t;
            }
            acc += hits;
        }
        __syncwarp();  // S and the lists are rewritten
        pos += wlen;
    }
    return acc;
}

// Whether v is a member of its own row (0 or 1).
__device__ __noinline__ uint32_t self_member(const Rows<false> &R, int v, const uint32_t *__restrict__ code) {
    const int4 l = R.row(v);
    const uint32_t e = __ldg(code + v);
    const int sh = e < kLowEnd ? 16 : R.mb;
    uint32_t n = 0;
    for (int i = 0; i < l.y + 2 * l.z; ++i)
        each4(R.quad(l.x, i, 0), [&](uint32_t q) {
            if ((q < kLowEnd) == (e < kLowEnd) && ((q ^ e) >> sh) == 0) n |= (uint32_t)((q & e & ((1u << sh) - 1u)) != 0);
        });
    return n;
}

// The count: one persistent grid takes the block units, then the listed roots
// (one warp each), then the short roots, each from its cursor, so that blocks
// that find no more of one kind fill the others' tail.  Bound by the L1 / shared
// pipe and by issue: a warp's round is two 16-byte loads of entries per lane and
// eight look-ups, about 100 instructions per 256 entries.  R-MAT 21, whole:
// 11.3 G W+ probes are 4.4 G entries; 2.45 ms against 5.98 for the plain-id tables
// (6.68 -> 2.88 ms per count with the passes before): the pipe 88 % busy, 61 % of
// the issue slots, 8.6 TB/s from L2.  4 blocks per SM (64 registers): with 5 (48)
// the next round's loads did not fit beside this round's, 4.3 instead of the 3.8 ms
// that it took then.
constexpr int kPackedMinBlocks = 4;
template <bool kPerRoot>
__global__ void __launch_bounds__(kThreads, kPackedMinBlocks) packed_kernel(PackParams P) {
    __shared__ __align__(16) uint32_t s_words[kWarps][kWarpWords];
    __shared__ ListAt<false> s_lists[kWarps][kWarp], s_high[kWarps][kWarp];
    __shared__ ShortState<false> s_short[kWarps];
    __shared__ unsigned s_unit;
    __shared__ int s_chunk;
    const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
    ListAt<false> *s_at = s_lists[warp];
    unsigned long long acc = 0;  // this lane's hits for graph cur_g
    int cur_g = -1;
    auto flush = [&](int g) {
        const unsigned long long s = sum_u64(acc);
        if (lane == 0 && cur_g >= 0 && s) atomicAdd(P.results + cur_g, s);
        acc = 0;
        cur_g = g;
    };
    {  // block units
        const unsigned n_units = (unsigned)P.work->heavy_packed;
        uint32_t *words = s_words[0];
        uint32_t *hs = words + kLow / 2;
        for (;;) {
            if (threadIdx.x == 0) s_unit = atomicAdd(&P.work->heavy_cursor, 1u);
            __syncthreads();
            const unsigned unit = s_unit;
            if (unit >= n_units) break;
            const uint2 un = P.units[unit];
            const int g = graph_of_chunk(P.gd, P.n_graphs, (int64_t)(un.x / kWarp));
            const GraphDesc &G = P.gd[g];
            const Rows<false> R = rows_of<false>(P, G);
            const int x = (int)(un.x - (uint32_t)(G.chunk_base * kWarp));
            const int rs = __ldg(G.rp + x), d = __ldg(G.rp + x + 1) - rs;
            const int4 l = R.row(x);
            const int j0 = (int)un.y * P.slice, j1 = min(d, j0 + P.slice);
            const int step = max(1, min(kWarp, (j1 - j0 + kWarps - 1) / kWarps));
            uint32_t hits = 0;
            int t0 = 0;
            do {  // the low blocks once; the high blocks' entries a tile at a time
                for (int i = threadIdx.x + (t0 ? kLow / 8 : 0); i < kBlockWords / 4; i += kThreads)
                    reinterpret_cast<uint4 *>(words)[i] = make_uint4(0, 0, 0, 0);
                if (threadIdx.x == 0) s_chunk = 0;
                __syncthreads();
                const int t1 = min(l.y, t0 + kBlockTile / 4);
                for (int i0 = t0 + warp * kWarp; i0 < t1; i0 += kThreads) {
                    const int i = i0 + lane;
                    each4(i < t1 ? R.quad(l.x, i, 0) : make_uint4(0, 0, 0, 0),
                          [&](uint32_t e) { filter_put(hs, kLogBlockH - 1, R.mb, e); });
                }
                if (t0 == 0)
                    for (int i = threadIdx.x; i < 2 * l.z; i += kThreads)
                        each4(R.quad(l.x, l.y + i, 0), [&](uint32_t e) { low_put(words, e); });
                __syncthreads();
                for (;;) {
                    int q = 0;
                    if (lane == 0) q = atomicAdd(&s_chunk, 1);
                    const int j = j0 + __shfl_sync(kFull, q, 0) * step;
                    if (j >= j1) break;
                    hits += stream_lists<false>(R, lane < step && j + lane < j1 ? __ldg(G.col + rs + j + lane) : -1,
                                                words, hs, kLogBlockH - 1, t0 == 0, t1 > t0, lane, s_at);
                }
                __syncthreads();
                t0 = t1;
            } while (t0 < l.y);
            if (kPerRoot) {
                const unsigned long long s = sum_u64(hits);
                if (lane == 0 && s) atomicAdd(G.per_root + x, s);
            }
            if (g != cur_g) flush(g);
            acc += hits;
            __syncthreads();
        }
        __syncthreads();
    }
    {  // listed roots
        const unsigned n_mid = (unsigned)P.work->n_tasks;
        for (;;) {
            unsigned t = 0;
            if (lane == 0) t = atomicAdd(&P.work->small_cursor, 1u);
            t = __shfl_sync(kFull, t, 0);
            if (t >= n_mid) break;
            const uint32_t row = P.mid_list[t];
            const int g = graph_of_chunk(P.gd, P.n_graphs, (int64_t)(row / kWarp));
            const GraphDesc &G = P.gd[g];
            const int x = (int)(row - (uint32_t)(G.chunk_base * kWarp));
            const int rs = __ldg(G.rp + x), d = __ldg(G.rp + x + 1) - rs;
            const uint32_t hits = warp_row<false>(rows_of<false>(P, G), x, rs, d, lane, s_words[warp],
                                                  s_words[warp] + kLow / 2, s_at);
            if (kPerRoot) {
                const unsigned s = __reduce_add_sync(kFull, hits);
                if (lane == 0) G.per_root[x] = s;
            }
            if (g != cur_g) flush(g);
            acc += hits;
        }
    }
    {  // short roots
        const bool self_loops = P.work->self_loops != 0;
        const int per = kWarp / P.pack_rows;  // grabs per 32-row chunk
        for (int i = lane; i < kLow / 8; i += kWarp) reinterpret_cast<uint4 *>(s_words[warp])[i] = make_uint4(0, 0, 0, 0);
        __syncwarp();
        for (;;) {
            unsigned i = 0;
            if (lane == 0) i = atomicAdd(&P.work->aux_cursor[0], 1u);
            i = __shfl_sync(kFull, i, 0);
            const int64_t c = (int64_t)(i / (unsigned)per);
            if (c >= P.total_chunks) break;
            const int g = graph_of_chunk(P.gd, P.n_graphs, c);
            const GraphDesc &G = P.gd[g];
            const int64_t x = (c - G.chunk_base) * kWarp + (int64_t)(i % (unsigned)per) * P.pack_rows + lane;
            int rs = 0, d = 0;
            if (lane < P.pack_rows && x < G.n_roots) {
                rs = __ldg(G.rp + x);
                d = __ldg(G.rp + x + 1) - rs;
            }
            if (g != cur_g) flush(g);
            // a root with one member v has a hit only if v is its own member: looked for where there are such rows
            if (self_loops && d == 1) {
                const uint32_t hit = self_member(rows_of<false>(P, G), __ldg(G.col + rs), P.code + G.vbase);
                acc += hit;
                if (kPerRoot && hit) G.per_root[x] = hit;
            }
            if (d < 2 || d > kRowMax) d = 0;
            acc += short_rows<false, kPerRoot>(rows_of<false>(P, G), x, rs, d, lane, s_words[warp],
                                               s_words[warp] + kLow / 2, s_short[warp], s_at, s_high[warp],
                                               G.per_root);
        }
    }
    flush(-1);
}

// One graph of few edges in one launch, on its own ids: a warp takes `rows`
// consecutive rows (few, so that a small graph fills many warps), the short
// ones together and the longer ones one after the other.
template <bool kPerRoot>
__global__ void __launch_bounds__(kThreads) single_kernel(GraphDesc G, int rows, unsigned long long *result) {
    // raw rows have no low blocks: only a hash
    __shared__ __align__(16) uint32_t s_hash[kWarps][1 << kLogWarpH];
    __shared__ ListAt<true> s_lists[kWarps][kWarp], s_high[kWarps][kWarp];
    __shared__ ShortState<true> s_short[kWarps];
    const int lane = threadIdx.x & (kWarp - 1), warp = threadIdx.x / kWarp;
    Rows<true> R;
    R.rp = G.rp;
    R.col = G.col;
    R.desc = nullptr;
    R.ent = nullptr;
    R.mb = 1;
    R.zero = 0;
    const int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kWarp;
    const int64_t nw = (int64_t)gridDim.x * kWarps;
    unsigned long long acc = 0;
    for (int64_t x0 = w0 * rows; x0 < G.n_roots; x0 += nw * rows) {
        const int64_t x = x0 + lane;
        int rs = 0, d = 0;
        if (lane < rows && x < G.n_roots) {
            rs = __ldg(G.rp + x);
            d = __ldg(G.rp + x + 1) - rs;
        }
        acc += short_rows<true, kPerRoot>(R, x, rs, d > kRowMax ? 0 : d, lane, nullptr, s_hash[warp], s_short[warp], s_lists[warp],
                                          s_high[warp], G.per_root);
        for (unsigned todo = __ballot_sync(kFull, d > kRowMax); todo; todo &= todo - 1u) {
            const int k = __ffs(todo) - 1;
            const int rrs = __shfl_sync(kFull, rs, k), rd = __shfl_sync(kFull, d, k);
            const uint32_t hits = warp_row<true>(R, (int)(x0 + k), rrs, rd, lane, nullptr, s_hash[warp],
                                                 s_lists[warp]);
            acc += hits;
            if (kPerRoot) {
                const unsigned s = __reduce_add_sync(kFull, hits);
                if (lane == 0) G.per_root[x0 + k] = s;
            }
        }
    }
    acc = sum_u64(acc);
    if (lane == 0 && acc) atomicAdd(result, acc);
}

}  // namespace

int pack_mask_bits(int64_t n_rows) {
    int mb = 16;
    while (mb > 1 && (n_rows + mb - 1) / mb > (int64_t)31 << (27 - mb)) --mb;
    return mb;
}

bool pack_fits(int64_t V, int64_t E) { return E + kRowPad * V + 8 < ((int64_t)1 << 34); }  // quads numbered in 32 bits

size_t pack_scratch_bytes(int64_t V, int64_t E, int n_graphs) {
    const size_t v = (size_t)std::max<int64_t>(V, 1), e = (size_t)std::max<int64_t>(E, 1);
    return sizeof(uint32_t) * (v + (size_t)n_graphs * 2 * kBuckets) + sizeof(int4) * v +
           sizeof(uint32_t) * (e + kRowPad * v + 8) + sizeof(uint32_t) * (e / (kRowMax + 1) + 1) +
           sizeof(uint2) * (e / (kRowMax / 2) + 1);
}

int pack_scratch_alloc(PackScratch *ps, int64_t V, int64_t E, int n_graphs, cudaStream_t s) {
    const size_t v = (size_t)std::max<int64_t>(V, 1), e = (size_t)std::max<int64_t>(E, 1);
    int st = dalloc((void **)&ps->code, sizeof(uint32_t) * (v + (size_t)n_graphs * 2 * kBuckets), s);
    if (st == TC_OK) st = dalloc((void **)&ps->desc, sizeof(int4) * v, s);
    if (st == TC_OK) st = dalloc((void **)&ps->ent, sizeof(uint32_t) * (e + kRowPad * v + 8), s);  // see row_quad
    if (st == TC_OK) st = dalloc((void **)&ps->mid_list, sizeof(uint32_t) * (e / (kRowMax + 1) + 1), s);
    // a row of more than 32 has at most one unit per 32 of its members, and one more
    if (st == TC_OK) st = dalloc((void **)&ps->units, sizeof(uint2) * (e / (kRowMax / 2) + 1), s);
    if (st != TC_OK) pack_scratch_free(ps, s);
    return st;
}

void pack_scratch_free(PackScratch *ps, cudaStream_t s) {
    dfree(ps->code, s);
    dfree(ps->desc, s);
    dfree(ps->ent, s);
    dfree(ps->mid_list, s);
    dfree(ps->units, s);
    *ps = PackScratch();
}

int launch_packed(const GraphDesc *d_desc, int n_graphs, int64_t total_chunks, int64_t total_vertices,
                  int64_t total_edges, const PackScratch &ps, CountWork *work, unsigned long long *results,
                  bool per_root, const Tuned &tn, cudaStream_t s, int *launches, cudaEvent_t *kev) {
    if (total_chunks * kWarp >= ((int64_t)1 << 32))
        return set_error(TC_E_RANGE, "a count of more than 2^32 rows in one launch is not supported");
    TC_TRY(zero_work(work, results, n_graphs, s));
    int nl = 0;
    if (total_chunks > 0) {
        PackParams P;
        P.gd = d_desc;
        P.n_graphs = n_graphs;
        P.total_chunks = total_chunks;
        P.total_edges = total_edges;
        P.work = work;
        P.results = results;
        P.code = ps.code;
        P.hist = ps.code + total_vertices;
        P.ent = ps.ent;
        P.desc = ps.desc;
        P.mid_list = ps.mid_list;
        P.units = ps.units;
        P.zero_quad = (int)(uint32_t)((total_edges + kRowPad * total_vertices + 4) >> 2);  // see row_quad, pack_scratch_alloc
        // Rows of up to 512 (twice the tuning's bound) on one warp: a block's eight warps wait for one another around
        // every unit's table (R-MAT 21 3.16 ms with 256, 3.00 with 512, 2.97 with no bound, whose last rows could be
        // a warp's millisecond).  Units of 512 out-neighbours (unit_work / 2048): with 128 a row's table was built
        // four times as often (3.37 ms; R-MAT 23's eight parts 32.9, 30.6 with 512).
        P.warp_max = 2 * tn.warp_max;
        P.slice = pack_slice(tn);
        TC_CUDA(cudaMemsetAsync(ps.code, 0,
                                sizeof(uint32_t) * ((size_t)total_vertices + (size_t)n_graphs * 2 * kBuckets), s));
        const int64_t tiles = (total_edges + kPopTile - 1) / kPopTile;
        if (tiles > 0) {
            pop_kernel<<<(unsigned)tiles, kThreads, 0, s>>>(P);
            TC_CUDA(cudaGetLastError());
            ++nl;
        }
        // few rows per block and warp while they do not fill the GPU
        P.rank_chunks = (int)std::min<int64_t>(64, std::max<int64_t>(8, total_chunks / ((int64_t)tn.sm_count * 8)));
        P.pack_rows = kWarp;
        while (P.pack_rows > 4 && total_chunks * kWarp / P.pack_rows < (int64_t)tn.sm_count * 40) P.pack_rows /= 2;
        const unsigned rank_blocks = (unsigned)((total_chunks + P.rank_chunks - 1) / P.rank_chunks);
        hist_kernel<<<rank_blocks, kThreads, 0, s>>>(P);
        TC_CUDA(cudaGetLastError());
        assign_kernel<<<rank_blocks, kThreads, 0, s>>>(P);
        TC_CUDA(cudaGetLastError());
        const int64_t want = (total_chunks * (kWarp / P.pack_rows) + kWarps - 1) / kWarps;
        // five blocks fit an SM, or the share of them that the tuning leaves the packed grid
        pack_kernel<<<(unsigned)std::min<int64_t>(want, (int64_t)tn.pack_blocks * 5 / kPackedMinBlocks), kThreads, 0, s>>>(P);
        TC_CUDA(cudaGetLastError());
        if (kev) TC_TRY(record_kernel_event(kev[0], s));
        if (per_root) packed_kernel<true><<<tn.pack_blocks, kThreads, 0, s>>>(P);
        else packed_kernel<false><<<tn.pack_blocks, kThreads, 0, s>>>(P);
        TC_CUDA(cudaGetLastError());
        if (kev) TC_TRY(record_kernel_event(kev[1], s));
        nl += 4;
    }
    if (launches) *launches = nl;
    return TC_OK;
}

int launch_single(const GraphDesc &d, CountWork *work, unsigned long long *result, const Tuned &tn, cudaStream_t s,
                  int *launches, cudaEvent_t *kev) {
    TC_TRY(zero_work(work, result, 1, s));
    if (kev) TC_TRY(record_kernel_event(kev[0], s));
    if (d.n_roots > 0) {
        // few rows per warp while the warps do not fill the GPU
        const int64_t warps = (int64_t)tn.sm_count * 32;
        int rows = 2;
        while (rows < kWarp && (d.n_roots + rows - 1) / rows > warps) rows *= 2;
        const int64_t want = ((d.n_roots + rows - 1) / rows + kWarps - 1) / kWarps;
        const unsigned blocks = (unsigned)std::min<int64_t>(want, (int64_t)tn.sm_count * 16);
        if (d.per_root) single_kernel<true><<<blocks, kThreads, 0, s>>>(d, rows, result);
        else single_kernel<false><<<blocks, kThreads, 0, s>>>(d, rows, result);
        TC_CUDA(cudaGetLastError());
    }
    if (kev) TC_TRY(record_kernel_event(kev[1], s));
    if (launches) *launches = d.n_roots > 0 ? 1 : 0;
    return TC_OK;
}

int pack_blocks(int sm_count, int num, int den, int *out) {
    int occ = 0;
    TC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, packed_kernel<false>, kThreads, 0));
    if (occ < 1) return set_error(TC_E_INVALID, "the packed count kernel does not fit on an SM");
    *out = sm_count * std::max(1, occ * num / den);
    return TC_OK;
}

}  // namespace tc
