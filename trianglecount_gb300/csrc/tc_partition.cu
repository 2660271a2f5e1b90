// tc_partition.cu -- balanced label-propagation partitioning of an undirected
// CSR on the device, the stand-in for the reference's METIS assignment
// (dgl.metis_partition_assignment(G, k), Halo_creation_preprocess.py:304, 341,
// 378; METIS itself is a third-party library that is not part of the
// reference tree).
//
// Like METIS it looks for parts of near-equal size with few cut edges, so a
// part's 1-hop halo stays small.  The method is label propagation with
// capacity-limited migration (in the manner of Spinner, Martella et al.,
// ICDE 2017), synchronous and integer-only, so a seed gives the same
// assignment on every GPU and host:
//   init     vertex v -> part floor(v k / n) (balanced contiguous ranges)
//   choose   per vertex, the label most common among its neighbours (ties:
//            stay, else a seeded hash decides); a vertex whose best label
//            beats its own becomes a candidate for that label
//   migrate  a candidate for label b moves with probability R_b / W_b (R_b:
//            room left under the cap ceil(1.03 n / k) plus the candidates
//            expected to leave b, W_b: candidates for b), decided by a seeded
//            hash; part sizes are recounted
// until fewer than 0.1% of the vertices move or the iteration budget is spent
// (looked at from the host after two iterations, then after every eight).
// Measured cut fractions at k = 8 (random parts: 0.875): Chung-Lu 0.71,
// R-MAT 0.81 (its hubs touch every part), a road grid 0.002; largest part
// 1.03 x the mean.
#include <algorithm>
#include <vector>

#include "tc_internal.h"

namespace tc {
namespace {

constexpr int kMaxParts = 64;
constexpr int kPT = 256;  // threads per block
constexpr int kLpFlight = 4;  // neighbours per lane and round (two: 1.37 instead of 1.31 ms then)
constexpr int kGroupDeg = 255, kAloneDeg = 64, kWarpDeg = 1024;  // see lp_choose_kernel
constexpr unsigned kFull = 0xffffffffu;

// splitmix64 finaliser (Steele, Lea, Flood, "Fast splittable pseudorandom
// number generators", OOPSLA 2014) over the packed inputs.
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

__device__ __forceinline__ uint32_t hash_vl(uint64_t seed, int it, int64_t v, int l) {
    return (uint32_t)(mix64(seed ^ mix64(((uint64_t)it << 40) ^ ((uint64_t)v << 8) ^ (uint64_t)l)) >> 32);
}

// The vertices of long rows, listed once: a warp takes one of mid at a time and a
// block one of big, each spread over the whole grid, so that long rows that lie
// together (ids in order of degree) are not one warp's work.
struct LpLong {
    int32_t *mid, *big;
    int32_t *n;  // vertices in mid, in big
};

// Labels and wishes are bytes on the device (at most 64 parts): the choose
// pass gathers one label per neighbour, and 4 x smaller arrays hit closer
// caches.
__global__ void lp_init_kernel(uint8_t *label, const int32_t *__restrict__ rp, int64_t n, int k, int32_t *size,
                               int mid_deg, LpLong rows) {
    __shared__ int32_t s[kMaxParts];
    for (int i = threadIdx.x; i < k; i += blockDim.x) s[i] = 0;
    __syncthreads();
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int l = (int)(v * k / n), d = rp[v + 1] - rp[v];
        label[v] = (uint8_t)l;
        atomicAdd(&s[l], 1);
        if (d > kWarpDeg) push_together(rows.big, rows.n + 1, (int32_t)v);
        else if (d > mid_deg) push_together(rows.mid, rows.n, (int32_t)v);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < k; i += blockDim.x)
        if (s[i]) atomicAdd(&size[i], s[i]);
}

// The words of one iteration, zeroed together.  The iterations of one batch
// are enqueued without a look from the host: an iteration whose predecessor in
// the batch moved fewer than 0.1 % of the vertices (or was itself left out: it
// moved none) does nothing.
struct LpIter {
    int32_t size[kMaxParts];              // part sizes before the iteration
    int32_t flow[kMaxParts * kMaxParts];  // candidates from part a to part b at [a * k + b]
    int32_t moved;
};
__device__ __forceinline__ bool lp_stopped(const LpIter *batch, int i, int64_t n) {
    return i > 0 && (int64_t)batch[i - 1].moved * 1000 < n;
}

// Best label by (count, tie hash) from its key's parts, the current label
// winning ties on count; -1 when that is the current one or there is none.
__device__ __forceinline__ unsigned long long lp_key(int count, uint64_t seed, int it, int64_t v, int l, int cur) {
    if (count <= 0) return 0ull;
    const uint32_t tie = l == cur ? 0xffffffffu : (hash_vl(seed, it, v, l) >> 1);
    return ((unsigned long long)(uint32_t)count << 32) | tie;
}

// One warp picks from a finished histogram h of k counts.
__device__ __forceinline__ int lp_pick(const int32_t *h, int k, uint64_t seed, int it, int64_t v, int cur, int lane) {
    unsigned long long best = 0, own[kMaxParts / 32] = {0, 0};
#pragma unroll
    for (int q = 0; q < kMaxParts / 32; ++q) {
        const int l = lane + 32 * q;
        if (l < k) own[q] = lp_key(h[l], seed, it, v, l, cur);
        best = own[q] > best ? own[q] : best;
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(kFull, best, o);
        best = t > best ? t : best;
    }
    if (best == 0 || (uint32_t)best == 0xffffffffu) return -1;
    const int bl = own[1] == best ? lane + 32 : own[0] == best ? lane : -1;
    return __shfl_sync(kFull, bl, __ffs(__ballot_sync(kFull, bl >= 0)) - 1);
}

// Per vertex, the label most common among its neighbours.  With at most 16 parts,
// vertices of degree <= 255 (kGroupDeg) are counted by eight lanes each, four at a
// time: the counts are bytes packed in kWords 64-bit registers per lane and are
// summed over the lanes with shuffles -- no histogram in memory, and the warp
// waits for four vertices' gathers at once.  (One warp per vertex with a shared
// histogram left most lanes idle on most rows: Chung-Lu n = 500 K, mean degree
// 16, k = 8, 20 iterations 3.87 ms the whole call, 1.26 ms so.)  With more parts
// vertices of degree <= 64 (kAloneDeg) are counted one at a time in the warp's
// histogram.  A warp takes per_warp consecutive vertices of these: 32, or fewer
// while that many would leave SMs without a block (lp_per_warp).  The others come
// from the lists (LpLong): up to degree kWarpDeg a warp each, larger ones the whole
// block, so that a hub's row is not one warp's chain of gathers.  (With each left
// to the warp or block that its neighbours in id belong to, graphs whose ids go by degree took
// 3 to 5 x a warp per vertex: R-MAT 20, k = 8, 7.9 instead of 1.5 ms.)
// Counts the labels of the row [a, a + d) into h, `step` lanes (or threads) of rank
// `at` together, four gathers in flight each.
__device__ __forceinline__ void lp_tally(const int32_t *__restrict__ col, const uint8_t *__restrict__ label, int a, int d,
                                         int at, int step, int32_t *h) {
    for (int j = at; j < d; j += 4 * step) {
        int p[4], q[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) p[i] = j + step * i < d ? __ldg(col + a + j + step * i) : -1;
#pragma unroll
        for (int i = 0; i < 4; ++i) q[i] = p[i] >= 0 ? __ldg(label + p[i]) : -1;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (q[i] >= 0) atomicAdd(&h[q[i]], 1);
    }
}

template <int kWords>
__global__ void __launch_bounds__(kPT) lp_choose_kernel(const int32_t *__restrict__ rp, const int32_t *__restrict__ col,
                                                        const uint8_t *__restrict__ label, int64_t n, int k,
                                                        int per_warp, LpLong rows, uint64_t seed, int it, int i_batch,
                                                        LpIter *batch, int8_t *__restrict__ desired) {
    constexpr int kMidDeg = kWords > 0 ? kGroupDeg : kAloneDeg;
    __shared__ int32_t hist[kPT / 32][kMaxParts];
    __shared__ int32_t s_flow[kMaxParts * kMaxParts];  // candidates from part a to part b at [a * k + b]
    if (lp_stopped(batch, i_batch, n)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < k * k; i += blockDim.x) s_flow[i] = 0;
    __syncthreads();
    int32_t *h = hist[warp];
    const int n_mid = rows.n[0], n_big = rows.n[1];
    // one warp: its finished histogram's pick for vertex v
    auto decide = [&](const int32_t *counts, int64_t v, int cl) {
        const int pick = lp_pick(counts, k, seed, it, v, cl, lane);
        if (lane == 0) {
            desired[v] = (int8_t)pick;
            if (pick >= 0) atomicAdd(&s_flow[cl * k + pick], 1);
        }
    };
    for (int b = blockIdx.x; b < n_big; b += gridDim.x) {
        const int64_t v = rows.big[b];
        for (int i = lane; i < k; i += 32) h[i] = 0;
        __syncwarp();
        const int a = rp[v];
        lp_tally(col, label, a, rp[v + 1] - a, threadIdx.x, kPT, h);
        __syncthreads();
        if (warp == 0) {
            for (int i = lane; i < k; i += 32) {
                int t = 0;
#pragma unroll
                for (int w = 0; w < kPT / 32; ++w) t += hist[w][i];
                hist[0][i] = t;
            }
            __syncwarp();
            decide(hist[0], v, label[v]);
        }
        __syncthreads();
    }
    auto alone = [&](int64_t v, int a, int d, int cl) {  // one vertex by the whole warp
        for (int i = lane; i < k; i += 32) h[i] = 0;
        __syncwarp();
        lp_tally(col, label, a, d, lane, 32, h);
        __syncwarp();
        decide(h, v, cl);
        __syncwarp();
    };
    for (int b = blockIdx.x + gridDim.x * warp; b < n_mid; b += gridDim.x * (kPT / 32)) {
        const int64_t v = rows.mid[b];
        const int a = rp[v];
        alone(v, a, rp[v + 1] - a, label[v]);
    }
    const int per_block = per_warp * (kPT / 32);
    for (int64_t v0 = (int64_t)blockIdx.x * per_block; v0 < n; v0 += (int64_t)gridDim.x * per_block) {
        const int64_t first = v0 + warp * per_warp, mine = first + lane;
        int rs = 0, d = 0, cur = 0;
        bool has = lane < per_warp && mine < n;
        if (has) {
            rs = rp[mine];
            d = rp[mine + 1] - rs;
            cur = label[mine];
            has = d <= kMidDeg;  // the others are listed
        }
        const int mine_d = has ? d : 0;
        if (kWords == 0) {
            if (has && d == 0) desired[mine] = -1;
            for (unsigned todo = __ballot_sync(kFull, mine_d > 0); todo; todo &= todo - 1u) {
                const int src = __ffs(todo) - 1;
                alone(first + src, __shfl_sync(kFull, rs, src), __shfl_sync(kFull, mine_d, src),
                      __shfl_sync(kFull, cur, src));
            }
        } else {
            int choice = -1;  // of this lane's vertex
            const int g = lane >> 3, l8 = lane & 7;
            for (int r = 0; r < per_warp; r += 4) {
                const int src = r + g;  // the group's vertex: lane src's
                const int a = __shfl_sync(kFull, rs, src);
                const int dd = __shfl_sync(kFull, mine_d, src), cl = __shfl_sync(kFull, cur, src);
                unsigned long long c[kWords > 0 ? kWords : 1];
#pragma unroll
                for (int w = 0; w < kWords; ++w) c[w] = 0;
                for (int j = l8; j < dd; j += 8 * kLpFlight) {  // so many gathers in flight per lane
                    int p[kLpFlight], q[kLpFlight];
#pragma unroll
                    for (int i = 0; i < kLpFlight; ++i) p[i] = j + 8 * i < dd ? __ldg(col + a + j + 8 * i) : -1;
#pragma unroll
                    for (int i = 0; i < kLpFlight; ++i) q[i] = p[i] >= 0 ? (int)__ldg(label + p[i]) : 8 * kWords;
#pragma unroll
                    for (int i = 0; i < kLpFlight; ++i)
#pragma unroll
                        for (int w = 0; w < kWords; ++w)
                            if (q[i] >> 3 == w) c[w] += 1ull << (8 * (q[i] & 7));
                }
                int best = 0, count[kWords > 0 ? kWords : 1];
#pragma unroll
                for (int w = 0; w < kWords; ++w) {
#pragma unroll
                    for (int o = 4; o >= 1; o >>= 1) c[w] += __shfl_xor_sync(kFull, c[w], o);
                    count[w] = (int)((c[w] >> (8 * l8)) & 255u);  // of label 8 w + l8
                    best = max(best, count[w]);
                }
#pragma unroll
                for (int o = 4; o >= 1; o >>= 1) best = max(best, __shfl_xor_sync(kFull, best, o));
                int of_cur = (int)((c[0] >> (8 * (cl & 7))) & 255u);
                if (kWords > 1 && cl >= 8) of_cur = (int)((c[kWords - 1] >> (8 * (cl & 7))) & 255u);
                int pick = -1;
                const bool leave = best > 0 && of_cur < best;
                if (__any_sync(kFull, leave)) {
                    // the largest (tie, lowest label first) among the labels of the best count
                    unsigned long long key = 0;
                    if (leave) {
#pragma unroll
                        for (int w = 0; w < kWords; ++w)
                            if (count[w] == best) {
                                const int l = 8 * w + l8;
                                const unsigned long long t =
                                    ((unsigned long long)(hash_vl(seed, it, first + src, l) >> 1) << 8) |
                                    (unsigned long long)(255 - l);
                                key = t > key ? t : key;
                            }
                    }
#pragma unroll
                    for (int o = 4; o >= 1; o >>= 1) {
                        const unsigned long long t = __shfl_xor_sync(kFull, key, o);
                        key = t > key ? t : key;
                    }
                    if (leave) pick = 255 - (int)(key & 255u);
                }
                // lanes r .. r + 3 own the four vertices: group g's pick
                const int got = __shfl_sync(kFull, pick, ((lane - r) & 3) << 3);
                if (lane >= r && lane < r + 4) choice = got;
            }
            if (has) {
                desired[mine] = (int8_t)choice;
                if (choice >= 0) atomicAdd(&s_flow[cur * k + choice], 1);
            }
        }
    }
    __syncthreads();
    int32_t *flow = batch[i_batch].flow;
    for (int i = threadIdx.x; i < k * k; i += blockDim.x)
        if (s_flow[i]) atomicAdd(&flow[i], s_flow[i]);
}

// A candidate for part b moves with probability room_b / want_b: it moves
// when its hash h (32 bits) satisfies h * want_b < room_b * 2^32.  room_b is
// the space left under the cap plus the candidates expected to leave b: those
// wanting part t, times t's acceptance rate before that credit
// (min(1, (cap - size_t) / want_t)), which under-counts the departures.  The
// parts' sizes after the moves are counted on the way.
__global__ void lp_migrate_kernel(const uint8_t *__restrict__ label, const int8_t *__restrict__ desired, int64_t n,
                                  int k, int32_t cap, uint64_t seed, int it, int i_batch, LpIter *batch,
                                  uint8_t *__restrict__ out) {
    __shared__ int64_t s_room0[kMaxParts], s_want[kMaxParts], s_room[kMaxParts];
    __shared__ int32_t s_moved, s_size[kMaxParts];
    if (lp_stopped(batch, i_batch, n)) return;
    const int32_t *size = batch[i_batch].size, *flow = batch[i_batch].flow;
    for (int t = threadIdx.x; t < k; t += blockDim.x) {
        int64_t w = 0;
        for (int a = 0; a < k; ++a) w += flow[a * k + t];
        s_want[t] = w;
        s_room0[t] = max((int64_t)0, (int64_t)cap - size[t]);
        s_size[t] = 0;
    }
    if (threadIdx.x == 0) s_moved = 0;
    __syncthreads();
    for (int b = threadIdx.x; b < k; b += blockDim.x) {
        int64_t leave = 0;
        for (int t = 0; t < k; ++t) {
            const int64_t f = flow[b * k + t];
            if (f) leave += s_room0[t] >= s_want[t] ? f : f * s_room0[t] / s_want[t];
        }
        s_room[b] = s_room0[b] + leave;
    }
    __syncthreads();
    int my_moves = 0;
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
        const int b = desired[v];
        int l = label[v];
        if (b >= 0) {
            const uint64_t h = hash_vl(seed ^ 0x5A5A5A5Aull, it, v, b);
            if (h * (uint64_t)s_want[b] < ((uint64_t)s_room[b] << 32)) {
                l = b;
                ++my_moves;
            }
        }
        out[v] = (uint8_t)l;
        atomicAdd(&s_size[l], 1);
    }
    if (my_moves) atomicAdd(&s_moved, my_moves);
    __syncthreads();
    if (threadIdx.x == 0 && s_moved) atomicAdd(&batch[i_batch].moved, s_moved);
    for (int t = threadIdx.x; t < k; t += blockDim.x)
        if (s_size[t]) atomicAdd(&batch[i_batch + 1].size[t], s_size[t]);
}

__global__ void lp_widen_kernel(const uint8_t *label, int64_t n, int32_t *out) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        out[v] = label[v];
}

// Vertices per warp of the choose pass, at least four where a warp counts four at a
// time.
int lp_per_warp(int64_t n, int k, const tc_ctx *ctx) {
    int w = 32;
    while (w > (k <= 16 ? 4 : 1) && n / (w * (kPT / 32)) < (int64_t)ctx->sm_count * 4) w /= 2;
    return w;
}

int pgrid(int64_t n, const tc_ctx *ctx) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + kPT - 1) / kPT, (int64_t)ctx->sm_count * 16));
}

}  // namespace
}  // namespace tc

using namespace tc;

extern "C" {

int tc_gen_parts_lp(tc_ctx *ctx, const tc_ugraph *ug, int k, uint64_t seed, int iterations, int32_t *part) {
    if (!ug || !part || k < 1 || k > kMaxParts || iterations < 0)
        return set_error(TC_E_INVALID, "bad label-propagation arguments (1 <= k <= %d, iterations >= 0)", kMaxParts);
    if (!ctx) ctx = ug->ctx;
    const int64_t n = ug->n_rows;
    if (n == 0) return TC_OK;
    cudaStream_t s = ctx->stream;
    // Iterations enqueued per look at the moves: two (a graph whose contiguous parts
    // are good moves little and stops: a road grid of 90 K vertices 120 us with
    // eight, of which seven did nothing, 82 with one), then eight.
    constexpr int kBatch = 8, kFirst = 2;
    DBuf<uint8_t> la, lb;
    DBuf<int8_t> desired;
    DBuf<int32_t> wide, lists;
    DBuf<LpIter> batch;  // the one after a batch's last holds the next batch's first sizes; behind all, the lists' lengths
    TC_TRY(la.alloc((size_t)n, s));
    TC_TRY(lb.alloc((size_t)n, s));
    TC_TRY(desired.alloc((size_t)n, s));
    TC_TRY(wide.alloc((size_t)n, s));
    TC_TRY(batch.alloc(kBatch + 2, s));
    const int mid_deg = k <= 16 ? kGroupDeg : kAloneDeg;
    const size_t most_mid = (size_t)(ug->nnz / (mid_deg + 1)), most_big = (size_t)(ug->nnz / (kWarpDeg + 1));
    TC_TRY(lists.alloc(most_mid + most_big, s));
    const LpLong rows{lists.p, lists.p + most_mid, batch.p[kBatch + 1].size};
    const int32_t cap = (int32_t)std::min<int64_t>(INT32_MAX, (n * 103 + 100LL * k - 1) / (100LL * k));
    const int gv = pgrid(n, ctx);
    const int pw = lp_per_warp(n, k, ctx), per_block = pw * (kPT / 32);
    const int gc = (int)std::min<int64_t>((n + per_block - 1) / per_block, (int64_t)ctx->sm_count * 64);
    TC_CUDA(cudaMemsetAsync(batch.p, 0, sizeof(LpIter) * (kBatch + 2), s));
    lp_init_kernel<<<gv, kPT, 0, s>>>(la.p, ug->rp, n, k, batch.p[0].size, mid_deg, rows);
    TC_CUDA(cudaGetLastError());
    bool more = k > 1;
    for (int it0 = 0, m = 0; it0 < iterations && more; it0 += m) {
        if (it0 > 0) {  // the last batch's end is this one's start
            TC_CUDA(cudaMemcpyAsync(batch.p[0].size, batch.p[m].size, sizeof(LpIter().size), cudaMemcpyDeviceToDevice, s));
            TC_CUDA(cudaMemsetAsync(batch.p[0].flow, 0, sizeof(LpIter) * (kBatch + 1) - sizeof(LpIter().size), s));
        }
        m = std::min(it0 > 0 ? kBatch : kFirst, iterations - it0);
        uint8_t *from = la.p, *to = lb.p;
        for (int i = 0; i < m; ++i) {
            const int it = it0 + i;
            if (k <= 8)
                lp_choose_kernel<1><<<gc, kPT, 0, s>>>(ug->rp, ug->col, from, n, k, pw, rows, seed, it, i, batch.p,
                                                    desired.p);
            else if (k <= 16)
                lp_choose_kernel<2><<<gc, kPT, 0, s>>>(ug->rp, ug->col, from, n, k, pw, rows, seed, it, i, batch.p,
                                                    desired.p);
            else
                lp_choose_kernel<0><<<gc, kPT, 0, s>>>(ug->rp, ug->col, from, n, k, pw, rows, seed, it, i, batch.p,
                                                    desired.p);
            lp_migrate_kernel<<<gv, kPT, 0, s>>>(from, desired.p, n, k, cap, seed, it, i, batch.p, to);
            TC_CUDA(cudaGetLastError());
            std::swap(from, to);
        }
        int32_t moved[kBatch];
        TC_CUDA(cudaMemcpy2DAsync(moved, sizeof(int32_t), &batch.p[0].moved, sizeof(LpIter), sizeof(int32_t), (size_t)m,
                                  cudaMemcpyDeviceToHost, s));
        TC_CUDA(cudaStreamSynchronize(s));
        int done = 0;  // iterations of the batch that ran
        while (done < m && more) more = (int64_t)moved[done++] * 1000 >= n;  // else fewer than 0.1% of the vertices moved
        if (done & 1) std::swap(la.p, lb.p);  // la: the labels after them
    }
    lp_widen_kernel<<<gv, kPT, 0, s>>>(la.p, n, wide.p);
    TC_CUDA(cudaGetLastError());
    TC_CUDA(cudaMemcpyAsync(part, wide.p, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToHost, s));
    TC_CUDA(cudaStreamSynchronize(s));
    return TC_OK;
}

}  // extern "C"
