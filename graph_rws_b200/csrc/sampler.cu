// GPU neighbour sampling, dedup / reindex, and the column reindex of sampled blocks.
//
// Replaces the sampling half of the reference's extension.  The reference samples per 16-row
// window and keeps the top-K columns by edge weight (core/include/sampling.cuh:65-448, driven by
// core/wrapper/sampling_wrapper.cu:58-438); it has no random generator.  Here a hop is
//   1. sample_hop          a group of 4 to 32 lanes per frontier node (a warp above fan-out 32):
//                          uniform sampling without replacement on a counter-based Philox4x32-10
//                          stream keyed by (seed, node, hop), so a node's list does not depend on
//                          batch composition, launch shape or GPU count (Floyd's subset algorithm;
//                          degree <= fanout takes every neighbour in CSR order);
//   2. dedup / reindex     a global-memory hash set of the nodes: the source list of the hop is the
//                          destination nodes followed by the new nodes in ascending id order, and
//                          every sampled edge gets the position of its endpoint in that list.  All
//                          hops of a batch share one table, and a bitmap of the node ids gives the
//                          order; single hops, graphs of unknown size and small batches of very
//                          large graphs have a table per hop and a radix sort;
//   3. block               the device BCSR builder (bcsr_build.cu) takes the fixed-stride lists as
//                          they are, or, of a single hop, compacted to a local CSR.
// reindex_and_prune_kernel (core/include/reindex.cuh:33-102) is kept as well, with the same
// integer arithmetic, for graphs that carry the reference's window-level `active_windows`.
#include <cub/cub.cuh>

#include "grws_common.cuh"

namespace grws {

constexpr int MAX_FANOUT = 256;          // the reference's dispatch stops at 256 too (core/helper/macros.h:60-71)
constexpr int SAMPLE_WARPS = 8;

// ---------------------------------------------------------------------------------------------
// Philox4x32-10 (Salmon et al., SC'11)
// ---------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ void philox4x32_10(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3,
                                                       uint32_t k0, uint32_t k1, uint32_t (&out)[4]) {
#pragma unroll
    for (int r = 0; r < 10; ++r) {
        const uint64_t p0 = (uint64_t)0xD2511F53u * c0;
        const uint64_t p1 = (uint64_t)0xCD9E8D57u * c2;
        const uint32_t n0 = (uint32_t)(p1 >> 32) ^ c1 ^ k0;
        const uint32_t n1 = (uint32_t)p1;
        const uint32_t n2 = (uint32_t)(p0 >> 32) ^ c3 ^ k1;
        const uint32_t n3 = (uint32_t)p0;
        c0 = n0; c1 = n1; c2 = n2; c3 = n3;
        k0 += 0x9E3779B9u; k1 += 0xBB67AE85u;
    }
    out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// j-th 64-bit draw of the stream (seed, node, hop): counter {node, hop, j >> 1, 0}, key = seed;
// words (2*(j&1)+1 : 2*(j&1)) of the block
__device__ __forceinline__ uint64_t sample_draw64(uint64_t seed, uint32_t node, uint32_t hop, uint32_t j) {
    uint32_t o[4];
    philox4x32_10(node, hop, j >> 1, 0u, (uint32_t)seed, (uint32_t)(seed >> 32), o);
    const uint32_t lo = (j & 1) ? o[2] : o[0], hi = (j & 1) ? o[3] : o[1];
    return ((uint64_t)hi << 32) | lo;
}

// Fan-outs up to 32: a group of G lanes per frontier node (G the power of two that holds the fan-out), one pick per
// lane.  The duplicate resolution is the same sequential rule as below, on registers: pick j is compared with
// the resolved picks before it by one ballot of the group.  A warp serves 32 / G nodes.  The three hops of a batch of
// 1,024 seeds, fan-out 15-10-5: 84 us with a warp per node and picks in shared memory, 28 us like this.
template <int G>
__global__ void __launch_bounds__(SAMPLE_WARPS * 32)
sample_hop_group_kernel(const int64_t *__restrict__ row_ptr, const int32_t *__restrict__ col_idx,
                        const float *__restrict__ values, const int32_t *__restrict__ nodes, int64_t n,
                        int fanout, uint64_t seed, const uint64_t *__restrict__ seed_dev, uint32_t hop,
                        int32_t *__restrict__ out_nbr, float *__restrict__ out_w, int32_t *__restrict__ out_cnt) {
    if (seed_dev) seed = *seed_dev;          // a seed that changes between replays of one captured launch
    const int lane = threadIdx.x & 31, j = lane & (G - 1), first = lane - j;
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    const int32_t v = i < n ? nodes[i] : -1;
    int64_t e0 = 0, d = 0;
    if (v >= 0) {
        e0 = __ldg(row_ptr + v);
        d = __ldg(row_ptr + v + 1) - e0;
    }
    int64_t pick = j;                        // degree <= fanout: every neighbour in CSR order
    if (d > fanout && j < fanout)
        pick = (int64_t)__umul64hi(sample_draw64(seed, (uint32_t)v, hop, (uint32_t)j), (uint64_t)(d - fanout + j + 1));
    if (__any_sync(0xffffffffu, d > fanout)) {
        const unsigned group = (G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u) << first;
        for (int t = 1; t < fanout; ++t) {
            const int64_t p = __shfl_sync(0xffffffffu, pick, first + t);
            const unsigned same = __ballot_sync(0xffffffffu, j < t && pick == p) & group;
            if (j == t && same && d > fanout) pick = d - fanout + t;
        }
    }
    if (i >= n || j >= fanout) return;
    const bool in = j < d;
    out_nbr[i * fanout + j] = in ? __ldg(col_idx + e0 + pick) : -1;
    out_w[i * fanout + j] = in ? (values ? __ldg(values + e0 + pick) : 1.0f) : 0.0f;
    if (j == 0 && out_cnt) out_cnt[i] = (int32_t)(d < fanout ? d : fanout);
}

// Wider fan-outs, one warp per frontier node.  Output slots have a fixed stride of `fanout`; unused slots hold
// -1 / 0.  For degree d > fanout f, pick j is floor(draw_j * (d - f + j + 1) / 2^64) unless an
// earlier pick has that value, in which case it is d - f + j (Floyd); picks are emitted in j order.
__global__ void __launch_bounds__(SAMPLE_WARPS * 32)
sample_hop_kernel(const int64_t *__restrict__ row_ptr, const int32_t *__restrict__ col_idx,
                  const float *__restrict__ values, const int32_t *__restrict__ nodes, int64_t n,
                  int fanout, uint64_t seed, const uint64_t *__restrict__ seed_dev, uint32_t hop,
                  int32_t *__restrict__ out_nbr, float *__restrict__ out_w, int32_t *__restrict__ out_cnt) {
    __shared__ int64_t picks[SAMPLE_WARPS][MAX_FANOUT];
    if (seed_dev) seed = *seed_dev;          // a seed that changes between replays of one captured launch
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * SAMPLE_WARPS + warp;
    if (i >= n) return;
    const int32_t v = nodes[i];
    int32_t *nb = out_nbr + i * fanout;
    float *ww = out_w + i * fanout;
    int64_t e0 = 0, d = 0;
    if (v >= 0) {
        e0 = __ldg(row_ptr + v);
        d = __ldg(row_ptr + v + 1) - e0;
    }
    if (d <= fanout) {
        for (int j = lane; j < fanout; j += 32) {
            const bool in = j < d;
            nb[j] = in ? __ldg(col_idx + e0 + j) : -1;
            ww[j] = in ? (values ? __ldg(values + e0 + j) : 1.0f) : 0.0f;
        }
        if (lane == 0 && out_cnt) out_cnt[i] = (int32_t)d;
        return;
    }
    int64_t *pk = picks[warp];
    // all draws first (independent), then the sequential duplicate resolution
    for (int j = lane; j < fanout; j += 32)
        pk[j] = (int64_t)__umul64hi(sample_draw64(seed, (uint32_t)v, hop, (uint32_t)j), (uint64_t)(d - fanout + j + 1));
    __syncwarp();
    for (int j = 1; j < fanout; ++j) {
        const int64_t t = pk[j];
        bool dup = false;
        for (int q = lane; q < j; q += 32) dup |= (pk[q] == t);
        if (__any_sync(0xffffffffu, dup)) {
            if (lane == 0) pk[j] = d - fanout + j;
        }
        __syncwarp();
    }
    for (int j = lane; j < fanout; j += 32) {
        const int64_t e = e0 + pk[j];
        nb[j] = __ldg(col_idx + e);
        ww[j] = values ? __ldg(values + e) : 1.0f;
    }
    if (lane == 0 && out_cnt) out_cnt[i] = fanout;
}

// ---------------------------------------------------------------------------------------------
// dedup / reindex
// ---------------------------------------------------------------------------------------------
constexpr int32_t EMPTY_KEY = -1;
constexpr int32_t NEW_NODE = 0x7fffffff;     // value of a neighbour that is not a destination node (rank not yet known)

__device__ __forceinline__ uint32_t hash_node(int32_t k) {
    uint32_t x = (uint32_t)k * 0x9E3779B1u;
    return x ^ (x >> 15);
}

// inserts `key`; returns the slot.  `fresh` tells whether this call created the entry.
__device__ __forceinline__ uint32_t table_insert(int32_t *keys, uint32_t mask, int32_t key, bool &fresh) {
    uint32_t h = hash_node(key) & mask;
    for (;;) {
        // a plain read first: a slot that already holds this key (a hub sampled from many rows) or
        // another one needs no atomic
        const int32_t cur = *reinterpret_cast<const volatile int32_t *>(keys + h);
        if (cur == key) { fresh = false; return h; }
        if (cur == EMPTY_KEY) {
            const int32_t prev = atomicCAS(keys + h, EMPTY_KEY, key);
            if (prev == EMPTY_KEY) { fresh = true; return h; }
            if (prev == key) { fresh = false; return h; }
        }
        h = (h + 1) & mask;
    }
}

__device__ __forceinline__ int32_t table_lookup(const int32_t *keys, const int32_t *vals, uint32_t mask, int32_t key) {
    uint32_t h = hash_node(key) & mask;
    for (;;) {
        const int32_t k = keys[h];
        if (k == key) return vals[h];
        if (k == EMPTY_KEY) return -1;
        h = (h + 1) & mask;
    }
}

__global__ void insert_dst_kernel(const int32_t *__restrict__ dst, int64_t n_dst, int32_t *keys, int32_t *vals,
                                  uint32_t mask, int32_t *__restrict__ out_src) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_dst) return;
    const int32_t v = dst[i];
    out_src[i] = v;
    if (v < 0) return;
    bool fresh;
    const uint32_t h = table_insert(keys, mask, v, fresh);
    atomicMin(vals + h, (int32_t)i);             // a repeated destination node keeps its first position
}

__global__ void insert_nbr_kernel(const int32_t *__restrict__ nbr, int64_t n_edges, int32_t *keys, int32_t *vals,
                                  uint32_t mask, int32_t *__restrict__ cand, int32_t *__restrict__ n_new) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int32_t u = e < n_edges ? nbr[e] : -1;
    bool fresh = false;
    if (u >= 0) table_insert(keys, mask, u, fresh);
    // one atomic on the shared counter per warp, not per new node (the order of `cand` does not
    // matter: it is sorted before the ranks are given out); vals[h] stays NEW_NODE until then
    const unsigned m = __ballot_sync(0xffffffffu, fresh);
    if (m) {
        const int lane = threadIdx.x & 31, leader = __ffs(m) - 1;
        int base = 0;
        if (lane == leader) base = atomicAdd(n_new, __popc(m));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (fresh) cand[base + __popc(m & ((1u << lane) - 1u))] = u;
    }
}

__global__ void rank_new_kernel(const int32_t *__restrict__ cand_sorted, const int32_t *__restrict__ n_new,
                                int64_t n_dst, const int32_t *keys, int32_t *vals, uint32_t mask,
                                int32_t *__restrict__ out_src) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *n_new) return;
    const int32_t u = cand_sorted[i];
    out_src[n_dst + i] = u;
    uint32_t h = hash_node(u) & mask;
    while (keys[h] != u) h = (h + 1) & mask;
    vals[h] = (int32_t)(n_dst + i);
}

// local ids of the sampled neighbours, and the number of valid entries of every destination row
__global__ void localize_kernel(const int32_t *__restrict__ nbr, int64_t n_dst, int fanout, const int32_t *keys,
                                const int32_t *vals, uint32_t mask, int32_t *__restrict__ out_local,
                                int64_t *__restrict__ row_cnt) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;   // one thread per destination row
    if (i >= n_dst) return;
    int cnt = 0;
    for (int j = 0; j < fanout; ++j) {
        const int32_t u = nbr[i * fanout + j];
        int32_t l = -1;
        if (u >= 0) { l = table_lookup(keys, vals, mask, u); ++cnt; }
        out_local[i * fanout + j] = l;
    }
    row_cnt[i + 1] = cnt;
    if (i == 0) row_cnt[0] = 0;
}

__global__ void finish_counts_kernel(const int32_t *__restrict__ n_new, int64_t n_dst, const int64_t *__restrict__ row_ptr,
                                     int64_t *__restrict__ out_counts) {
    out_counts[0] = n_dst + *n_new;      // number of source nodes
    out_counts[1] = row_ptr[n_dst];      // number of sampled edges
}

__global__ void compact_kernel(const int32_t *__restrict__ local, const float *__restrict__ w, int64_t n_dst, int fanout,
                               const int64_t *__restrict__ row_ptr, int32_t *__restrict__ out_col, float *__restrict__ out_val) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_dst) return;
    int64_t o = row_ptr[i];
    for (int j = 0; j < fanout; ++j) {
        const int32_t l = local[i * fanout + j];
        if (l >= 0) { out_col[o] = l; out_val[o] = w[i * fanout + j]; ++o; }
    }
}

__global__ void fill_i32(int32_t *p, int64_t n, int32_t v) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) p[i] = v;
}

// same integer arithmetic as reindex_and_prune_kernel (core/include/reindex.cuh:33-102): the window
// of a column is col / tile_rows with C division, so a -1 padding id is looked up as window 0
template <typename T>
__global__ void reindex_kernel(const int32_t *__restrict__ in_cols, T *__restrict__ values,
                               const int32_t *__restrict__ active_windows, int64_t num_indices, int num_active,
                               int tile_rows, int tile_cols, int32_t *__restrict__ out_cols) {
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= num_indices) return;
    const int g = in_cols[idx];
    const int target = g / tile_rows;
    int left = 0, right = num_active - 1, found = -1;
    while (left <= right) {
        const int mid = (left + right) / 2;
        const int win = __ldg(active_windows + mid);
        if (win == target) { found = mid; break; }
        if (win < target) left = mid + 1; else right = mid - 1;
    }
    if (found != -1) {
        out_cols[idx] = found * tile_rows + (g % tile_rows);
    } else {
        out_cols[idx] = 0;
        const int64_t base = (idx / tile_cols) * tile_rows * tile_cols;
        const int cit = (int)(idx % tile_cols);
        for (int r = 0; r < tile_rows; ++r) values[base + r * tile_cols + cit] = T(0.0f);
    }
}

// column ids through a table: out[i] = map[cols[i]], negative ids as they are (an id past the table: -1, and *ok
// becomes 0)
__global__ void relabel_columns_kernel(const int32_t *__restrict__ cols, int64_t n, const int32_t *__restrict__ map, int64_t n_map,
                                       int32_t *__restrict__ out, int32_t *__restrict__ ok) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t c = cols[i];
    if (c >= n_map && ok) *ok = 0;
    out[i] = c < 0 ? c : c < n_map ? __ldg(map + c) : -1;
}

// Column slots that name no row of the operand (-1 padding, ids of num_cols or more) become slots of row 0 with
// zero values.  Only such slots' values are written: eight neighbouring threads cover 16-byte rows of a tile.  (A
// masked fill reads and writes all values: 45 us for the 33 MB of a sampled step's first block, and 60 us with the
// comparisons around it; 9.5 us like this, caches cold.)
template <typename T>
__global__ void sanitize_columns_kernel(int32_t *__restrict__ cols, T *__restrict__ vals, int64_t n, int64_t num_cols) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t c = cols[i];
    if (c != -1 && c < num_cols) return;
    cols[i] = 0;
    T *v = vals + i / TILE_COLS * TILE_ELEMS + i % TILE_COLS;
#pragma unroll
    for (int r = 0; r < TILE_ROWS; ++r) v[r * TILE_COLS] = T(0.0f);
}

// one launch instead of four fills: empty hash table, candidate list of sentinels, zero counter,
// and the part of the source list behind the destination nodes set to -1
__global__ void dedup_init_kernel(int32_t *keys, int32_t *vals, int64_t slots, int32_t *cand, int64_t n_cand,
                                  int32_t *n_new, int32_t *src_tail, int64_t n_tail) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t i = i0; i < slots; i += stride) { keys[i] = EMPTY_KEY; vals[i] = NEW_NODE; }
    for (int64_t i = i0; i < n_cand; i += stride) cand[i] = NEW_NODE;
    for (int64_t i = i0; i < n_tail; i += stride) src_tail[i] = -1;
    if (i0 == 0) *n_new = 0;
}

// local id of every sampled neighbour (one thread per list slot)
__global__ void localize_flat_kernel(const int32_t *__restrict__ nbr, int64_t n_entries, const int32_t *keys,
                                     const int32_t *vals, uint32_t mask, int32_t *__restrict__ out_local) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_entries) return;
    const int32_t u = nbr[e];
    out_local[e] = u >= 0 ? table_lookup(keys, vals, mask, u) : -1;
}

// ---------------------------------------------------------------------------------------------
// dedup of a whole mini-batch over a graph whose node count is known: one hash table for all hops
// (a hop's destination nodes are the previous hop's source list, so they are in it already), and a
// bitmap of the node ids per hop instead of a sort of the new ids: a prefix sum of its bit counts
// gives every new node its place in ascending order.  Ids at or above the node count (a last hop may
// name some) go to a list of their own and rank behind the others.  The list is sorted in runs, the runs are merged in
// groups, and an id's rank is the sum of its places in the groups; all three in CTAs and threads of launches that
// the hop has anyway, so that a hop without such ids does not pay for them.
// ---------------------------------------------------------------------------------------------
constexpr int RANK_THREADS = 256;                // bitmap words per CTA
constexpr int OVER_RUN = 8192;                   // ids past the bitmap that one CTA sorts (shared memory: 32 KB)

struct HopRank {
    uint32_t *bits;                              // [words] new nodes of this hop
    int32_t *prefix;                             // [words] new nodes in the words before, of the same CTA
    int32_t *sums;                               // [CTAs] new nodes of a CTA's words, then of all earlier CTAs
    int32_t *over;                               // ids past the bitmap, then in runs of OVER_RUN ascending ids
    int32_t *merged;                             // the same in groups of over_group() ascending ids
    int32_t *counters;                           // {new nodes, ids in `over`, CTAs that have counted}
    int64_t words, num_nodes;
};

__global__ void layers_init_kernel(int32_t *keys, int32_t *vals, int64_t slots, uint32_t *bits, int64_t n_bits, int32_t *counters, int n_counters) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x, i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint4 none = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu), fresh = make_uint4(NEW_NODE, NEW_NODE, NEW_NODE, NEW_NODE);
    for (int64_t i = i0; i < slots / 4; i += stride) {          // slots is a power of two, 64 or more
        reinterpret_cast<uint4 *>(keys)[i] = none;              // EMPTY_KEY
        reinterpret_cast<uint4 *>(vals)[i] = fresh;
    }
    for (int64_t i = i0; i < n_bits; i += stride) bits[i] = 0;
    if (i0 < n_counters) counters[i0] = 0;
}

__global__ void insert_seeds_kernel(const int32_t *__restrict__ seeds, int64_t n, int32_t *keys, int32_t *vals, uint32_t mask) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || seeds[i] < 0) return;
    bool fresh;
    const uint32_t h = table_insert(keys, mask, seeds[i], fresh);
    atomicMin(vals + h, (int32_t)i);             // a repeated seed keeps its first position
}

__global__ void insert_marked_kernel(const int32_t *__restrict__ nbr, int64_t n_entries, int32_t *keys, uint32_t mask, const HopRank r) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int32_t u = e < n_entries ? nbr[e] : -1;
    if (u < 0) return;
    bool fresh;
    table_insert(keys, mask, u, fresh);
    if (!fresh) return;
    if (u < r.num_nodes) atomicOr(r.bits + (u >> 5), 1u << (u & 31));
    else r.over[atomicAdd(r.counters + 1, 1)] = u;
}

__device__ __forceinline__ int block_exclusive(int v, int *warp_part, int *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    __syncthreads();                             // the previous use of warp_part is over
    if (lane == 31) warp_part[warp] = incl;
    __syncthreads();
    int ahead = 0, all = 0;
#pragma unroll
    for (int i = 0; i < RANK_THREADS / 32; ++i) {
        all += warp_part[i];
        if (i < warp) ahead += warp_part[i];
    }
    *total = all;
    return ahead + incl - v;
}

// Counts the new nodes of every CTA's words; the CTA that counts last turns the counts into prefixes.  CTAs from
// rank_blocks on sort the runs of the ids past the bitmap: there are as many as the hop's list slots could need, and
// they return at once where it has no such ids.  A last hop of 8,192 rows, fan-out 15, that names 120 k ids of 5 M
// columns: 229 us with all its kernels (12.3 ms with a scan of the list for every id, 265 us with a radix sort); 980 k
// such ids: 618 us (497 us with a radix sort, which num_nodes = 0 asks for; a bitmap of all columns costs less than either).
__global__ void __launch_bounds__(RANK_THREADS)
rank_sums_kernel(const HopRank r, int rank_blocks) {
    __shared__ int warp_part[RANK_THREADS / 32];
    __shared__ bool last;
    __shared__ uint32_t ids[OVER_RUN];
    if ((int)blockIdx.x >= rank_blocks) {
        const int64_t i0 = (int64_t)((int)blockIdx.x - rank_blocks) * OVER_RUN;
        const int n = (int)min((long long)(r.counters[1] - i0), (long long)OVER_RUN);
        if (n <= 0) return;
        int padded = 2;
        while (padded < n) padded <<= 1;
        for (int j = threadIdx.x; j < padded; j += RANK_THREADS) ids[j] = j < n ? (uint32_t)r.over[i0 + j] : 0xffffffffu;
        block_sort(ids, padded);
        for (int j = threadIdx.x; j < n; j += RANK_THREADS) r.over[i0 + j] = (int32_t)ids[j];
        return;
    }
    const int64_t i = (int64_t)blockIdx.x * RANK_THREADS + threadIdx.x;
    int total;
    const int mine = i < r.words ? __popc(r.bits[i]) : 0;
    const int before = block_exclusive(mine, warp_part, &total);
    if (i < r.words) r.prefix[i] = before;
    if (threadIdx.x == 0) {
        r.sums[blockIdx.x] = total;
        __threadfence();
        last = atomicAdd(r.counters + 2, 1) == rank_blocks - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    int done = 0;
    for (int b0 = 0; b0 < rank_blocks; b0 += RANK_THREADS) {
        const int b = b0 + (int)threadIdx.x;
        const int v = b < rank_blocks ? *reinterpret_cast<const volatile int32_t *>(r.sums + b) : 0;
        const int ahead = block_exclusive(v, warp_part, &total);
        if (b < rank_blocks) r.sums[b] = done + ahead;
        done += total;
    }
    if (threadIdx.x == 0) r.counters[0] = done + r.counters[1];
}

// ids of a group of about as many runs as there are groups
__device__ __forceinline__ int64_t over_group(int64_t n_over) {
    int64_t fan = 1;
    while (fan * fan * OVER_RUN < n_over) fan <<= 1;
    return fan * OVER_RUN;
}

// number of ids below u in ids[first, end), which holds ascending runs of `run` ids
__device__ __forceinline__ int64_t count_below(const int32_t *ids, int64_t first, int64_t end, int64_t run, int32_t u) {
    int64_t k = 0;
    for (int64_t b = first; b < end; b += run) k += lower_bound(ids + b, (int)(end - b < run ? end - b : run), u);
    return k;
}

// place of a new node among the hop's new nodes in ascending order
__device__ __forceinline__ int32_t rank_of(const HopRank &r, int32_t u) {
    if (u < r.num_nodes) {
        const int64_t i = u >> 5;
        return r.sums[i / RANK_THREADS] + r.prefix[i] + __popc(r.bits[i] & ((1u << (u & 31)) - 1u));
    }
    const int64_t n_over = r.counters[1];
    return r.counters[0] - (int32_t)n_over + (int32_t)count_below(r.merged, 0, n_over, over_group(n_over), u);
}

// source list of the hop: destination nodes ++ new nodes in ascending order ++ -1 (ids past the bitmap are merged here
// and written by the next kernel)
__global__ void __launch_bounds__(RANK_THREADS)
emit_sources_kernel(const HopRank r, const int32_t *__restrict__ dst, int64_t n_dst, int64_t n_src, int32_t *__restrict__ out_src) {
    const int64_t i = (int64_t)blockIdx.x * RANK_THREADS + threadIdx.x, stride = (int64_t)gridDim.x * RANK_THREADS;
    if (i < r.words) {
        uint32_t b = r.bits[i];
        int32_t *o = out_src + n_dst + r.sums[i / RANK_THREADS] + r.prefix[i];
        for (; b; b &= b - 1) *o++ = (int32_t)(i * 32) + __ffs(b) - 1;
    }
    const int64_t n_over = r.counters[1], group = over_group(n_over);
    for (int64_t j = i; j < n_over; j += stride) {
        const int64_t g0 = j / group * group, g1 = g0 + group < n_over ? g0 + group : n_over;
        r.merged[g0 + count_below(r.over, g0, g1, OVER_RUN, r.over[j])] = r.over[j];
    }
    for (int64_t j = i; j < n_dst; j += stride) out_src[j] = dst[j];
    for (int64_t j = n_dst + r.counters[0] + i; j < n_src; j += stride) out_src[j] = -1;
}

// local id of every sampled neighbour; the table learns the ids of the nodes that are new in this hop
// (every thread that meets a new node writes the same value), and the source list the ids past the bitmap
__global__ void localize_ranked_kernel(const int32_t *__restrict__ nbr, int64_t n_entries, int64_t n_dst, const int32_t *keys, int32_t *vals,
                                       uint32_t mask, const HopRank r, int32_t *__restrict__ out_local, int32_t *__restrict__ out_src) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= n_entries) return;
    if (e < r.counters[1]) out_src[n_dst + rank_of(r, r.merged[e])] = r.merged[e];
    const int32_t u = nbr[e];
    int32_t l = -1;
    if (u >= 0) {
        uint32_t h = hash_node(u) & mask;
        while (keys[h] != u) h = (h + 1) & mask;             // every neighbour has been inserted
        l = *reinterpret_cast<const volatile int32_t *>(vals + h);
        if (l == NEW_NODE) {
            l = (int32_t)n_dst + rank_of(r, u);
            *reinterpret_cast<volatile int32_t *>(vals + h) = l;
        }
    }
    out_local[e] = l;
}

// per-hop figures for the caller: {source nodes (padded destinations + new nodes), sampled edges,
// tiles of the block, real (non-padding) frontier nodes}
__global__ void hop_counts_kernel(const int32_t *__restrict__ n_new, const int32_t *__restrict__ dst, int64_t n_dst,
                                  const int32_t *__restrict__ cnt, const int64_t *__restrict__ window_offset, int64_t W,
                                  int64_t *__restrict__ out) {
    __shared__ unsigned long long s_edges, s_real;
    if (threadIdx.x == 0) { s_edges = 0; s_real = 0; }
    __syncthreads();
    unsigned long long e = 0, r = 0;
    for (int64_t i = threadIdx.x; i < n_dst; i += blockDim.x) { e += (unsigned long long)cnt[i]; r += dst[i] >= 0 ? 1 : 0; }
    atomicAdd(&s_edges, e);
    atomicAdd(&s_real, r);
    __syncthreads();
    if (threadIdx.x == 0) {
        out[0] = n_dst + *n_new;
        out[1] = (int64_t)s_edges;
        out[2] = window_offset[W];
        out[3] = (int64_t)s_real;
    }
}

// bcsr_build.cu
int block_build_fill(int64_t n_dst, int fanout, const int64_t *window_offset, int64_t num_tiles, int32_t *out_cols, void *out_vals,
                     int val_dtype, void *scratch, size_t scratch_bytes, cudaStream_t st);

static inline size_t up256(size_t x) { return (x + 255) / 256 * 256; }
static inline unsigned nblocks(int64_t n, int t) { int64_t b = (n + t - 1) / t; return (unsigned)(b < 1 ? 1 : b); }

static int launch_sample_hop(const int64_t *row_ptr, const int32_t *col_idx, const float *values, const int32_t *nodes, int64_t n, int fanout,
                             uint64_t seed, const uint64_t *seed_dev, uint32_t hop, int32_t *nbr, float *w, int32_t *cnt, cudaStream_t st) {
    const int T = SAMPLE_WARPS * 32;
    if (fanout <= 4) sample_hop_group_kernel<4><<<nblocks(n * 4, T), T, 0, st>>>(row_ptr, col_idx, values, nodes, n, fanout, seed, seed_dev, hop, nbr, w, cnt);
    else if (fanout <= 8) sample_hop_group_kernel<8><<<nblocks(n * 8, T), T, 0, st>>>(row_ptr, col_idx, values, nodes, n, fanout, seed, seed_dev, hop, nbr, w, cnt);
    else if (fanout <= 16) sample_hop_group_kernel<16><<<nblocks(n * 16, T), T, 0, st>>>(row_ptr, col_idx, values, nodes, n, fanout, seed, seed_dev, hop, nbr, w, cnt);
    else if (fanout <= 32) sample_hop_group_kernel<32><<<nblocks(n * 32, T), T, 0, st>>>(row_ptr, col_idx, values, nodes, n, fanout, seed, seed_dev, hop, nbr, w, cnt);
    else sample_hop_kernel<<<nblocks(n, SAMPLE_WARPS), T, 0, st>>>(row_ptr, col_idx, values, nodes, n, fanout, seed, seed_dev, hop, nbr, w, cnt);
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

struct DedupScratch {
    int32_t *keys, *vals, *cand, *cand_sorted, *n_new;
    void *cub_tmp;
    size_t cub_bytes, total;
    uint32_t slots;
};

static DedupScratch carve_dedup(void *base, int64_t n_dst, int fanout) {
    DedupScratch s;
    const int64_t n_edges = n_dst * fanout;
    uint64_t want = 2ull * (uint64_t)(n_dst + n_edges) + 16, slots = 64;
    while (slots < want) slots <<= 1;
    s.slots = (uint32_t)slots;
    char *p = static_cast<char *>(base);
    size_t off = 0;
    auto take = [&](size_t bytes) { char *q = p ? p + off : nullptr; off += up256(bytes); return (void *)q; };
    s.keys = (int32_t *)take(slots * 4);
    s.vals = (int32_t *)take(slots * 4);
    s.cand = (int32_t *)take((size_t)(n_edges + 1) * 4);
    s.cand_sorted = (int32_t *)take((size_t)(n_edges + 1) * 4);
    s.n_new = (int32_t *)take(256);
    size_t c1 = 0, c2 = 0;
    cub::DeviceRadixSort::SortKeys(nullptr, c1, (const int32_t *)nullptr, (int32_t *)nullptr, (int)(n_edges > 0 ? n_edges : 1));
    cub::DeviceScan::InclusiveSum(nullptr, c2, (const int64_t *)nullptr, (int64_t *)nullptr, (int)(n_dst + 1));
    s.cub_bytes = c1 > c2 ? c1 : c2;
    s.cub_tmp = take(s.cub_bytes);
    s.total = off;
    return s;
}

}  // namespace grws

using namespace grws;

extern "C" {

__attribute__((visibility("default")))
int grws_sample_hop(const int64_t *row_ptr, const int32_t *col_idx, const float *values, const int32_t *nodes,
                    int64_t num_nodes, int fanout, uint64_t seed, uint32_t hop, int32_t *out_nbr, float *out_w,
                    int32_t *out_cnt, void *stream) {
    GRWS_REQUIRE(num_nodes >= 0, "negative size");
    GRWS_REQUIRE(fanout > 0 && fanout <= MAX_FANOUT, "fanout %d outside [1, %d]", fanout, MAX_FANOUT);
    if (num_nodes == 0) return GRWS_OK;
    GRWS_REQUIRE(row_ptr && col_idx && nodes && out_nbr && out_w, "null pointer");
    return launch_sample_hop(row_ptr, col_idx, values, nodes, num_nodes, fanout, seed, nullptr, hop, out_nbr, out_w, out_cnt,
                             static_cast<cudaStream_t>(stream));
}

__attribute__((visibility("default")))
size_t grws_dedup_scratch_bytes(int64_t n_dst, int fanout) {
    if (n_dst < 0 || fanout <= 0) return 0;
    return carve_dedup(nullptr, n_dst, fanout).total;
}

__attribute__((visibility("default")))
int grws_dedup_reindex(const int32_t *dst, int64_t n_dst, const int32_t *nbr, int fanout, int32_t *out_src,
                       int32_t *out_local, int64_t *out_row_ptr, int64_t *out_counts, void *scratch,
                       size_t scratch_bytes, void *stream) {
    GRWS_REQUIRE(n_dst >= 0 && fanout > 0, "bad size");
    GRWS_REQUIRE(n_dst * (int64_t)fanout < 0x7fffffffLL, "hop too large");
    GRWS_REQUIRE(out_src && out_local && out_row_ptr && out_counts && scratch, "null pointer");
    DedupScratch s = carve_dedup(scratch, n_dst, fanout);
    if (scratch_bytes < s.total) return fail(GRWS_ERR_SCRATCH, "dedup scratch too small: %zu < %zu", scratch_bytes, s.total);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t n_edges = n_dst * fanout;
    const uint32_t mask = s.slots - 1;
    GRWS_CUDA_TRY(cudaMemsetAsync(s.keys, 0xff, (size_t)s.slots * 4, st));                 // EMPTY_KEY
    fill_i32<<<nblocks(s.slots, 256) > 2048 ? 2048 : nblocks(s.slots, 256), 256, 0, st>>>(s.vals, s.slots, NEW_NODE);
    fill_i32<<<nblocks(n_edges + 1, 256) > 2048 ? 2048 : nblocks(n_edges + 1, 256), 256, 0, st>>>(s.cand, n_edges + 1, NEW_NODE);
    GRWS_CUDA_TRY(cudaMemsetAsync(s.n_new, 0, 256, st));
    if (n_dst > 0) {
        GRWS_REQUIRE(dst && nbr, "null pointer");
        insert_dst_kernel<<<nblocks(n_dst, 256), 256, 0, st>>>(dst, n_dst, s.keys, s.vals, mask, out_src);
        insert_nbr_kernel<<<nblocks(n_edges, 256), 256, 0, st>>>(nbr, n_edges, s.keys, s.vals, mask, s.cand, s.n_new);
        size_t tmp = s.cub_bytes;
        GRWS_CUDA_TRY(cub::DeviceRadixSort::SortKeys(s.cub_tmp, tmp, s.cand, s.cand_sorted, (int)n_edges, 0, 32, st));
        rank_new_kernel<<<nblocks(n_edges, 256), 256, 0, st>>>(s.cand_sorted, s.n_new, n_dst, s.keys, s.vals, mask, out_src);
        localize_kernel<<<nblocks(n_dst, 128), 128, 0, st>>>(nbr, n_dst, fanout, s.keys, s.vals, mask, out_local, out_row_ptr);
        tmp = s.cub_bytes;
        GRWS_CUDA_TRY(cub::DeviceScan::InclusiveSum(s.cub_tmp, tmp, out_row_ptr, out_row_ptr, (int)(n_dst + 1), st));
    } else {
        GRWS_CUDA_TRY(cudaMemsetAsync(out_row_ptr, 0, 8, st));
    }
    finish_counts_kernel<<<1, 1, 0, st>>>(s.n_new, n_dst, out_row_ptr, out_counts);
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

__attribute__((visibility("default")))
int grws_block_compact(const int32_t *local, const float *w, int64_t n_dst, int fanout, const int64_t *row_ptr,
                       int32_t *out_col, float *out_val, void *stream) {
    GRWS_REQUIRE(n_dst >= 0 && fanout > 0, "bad size");
    if (n_dst == 0) return GRWS_OK;
    GRWS_REQUIRE(local && w && row_ptr, "null pointer");
    compact_kernel<<<nblocks(n_dst, 128), 128, 0, static_cast<cudaStream_t>(stream)>>>(local, w, n_dst, fanout, row_ptr, out_col, out_val);
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

__attribute__((visibility("default")))
int grws_reindex_bcsr(const int32_t *in_cols, void *values, int val_dtype, const int32_t *active_windows,
                      int64_t num_indices, int64_t num_active, int tile_rows, int tile_cols, int32_t *out_cols,
                      void *stream) {
    GRWS_REQUIRE(num_indices >= 0 && num_active >= 0 && tile_rows > 0 && tile_cols > 0, "bad size");
    GRWS_REQUIRE(num_active < 0x7fffffffLL, "too many active windows");
    if (num_indices == 0) return GRWS_OK;
    GRWS_REQUIRE(in_cols && values && out_cols && (num_active == 0 || active_windows), "null pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned nb = nblocks(num_indices, 256);
    if (val_dtype == GRWS_F32)
        reindex_kernel<float><<<nb, 256, 0, st>>>(in_cols, (float *)values, active_windows, num_indices, (int)num_active, tile_rows, tile_cols, out_cols);
    else if (val_dtype == GRWS_F16)
        reindex_kernel<__half><<<nb, 256, 0, st>>>(in_cols, (__half *)values, active_windows, num_indices, (int)num_active, tile_rows, tile_cols, out_cols);
    else if (val_dtype == GRWS_BF16)
        reindex_kernel<__nv_bfloat16><<<nb, 256, 0, st>>>(in_cols, (__nv_bfloat16 *)values, active_windows, num_indices, (int)num_active, tile_rows, tile_cols, out_cols);
    else
        return fail(GRWS_ERR_UNSUPPORTED, "bad value dtype %d", val_dtype);
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

static int relabel_columns(const int32_t *cols, int64_t n, const int32_t *map, int64_t n_map, int32_t *out, int32_t *ok, void *stream) {
    GRWS_REQUIRE(n >= 0 && n_map >= 0, "negative size");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (ok) GRWS_CUDA_TRY(cudaMemsetAsync(ok, 1, sizeof(*ok), st));
    if (n == 0) return GRWS_OK;
    GRWS_REQUIRE(cols && out && (n_map == 0 || map), "null pointer");
    relabel_columns_kernel<<<nblocks(n, 256), 256, 0, st>>>(cols, n, map, n_map, out, ok);
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

__attribute__((visibility("default")))
int grws_relabel_columns(const int32_t *cols, int64_t n, const int32_t *map, int64_t n_map, int32_t *out, void *stream) {
    return relabel_columns(cols, n, map, n_map, out, nullptr, stream);
}

__attribute__((visibility("default")))
int grws_relabel_columns_checked(const int32_t *cols, int64_t n, const int32_t *map, int64_t n_map, int32_t *out, int32_t *ok,
                                 void *stream) {
    GRWS_REQUIRE(ok, "null pointer");
    return relabel_columns(cols, n, map, n_map, out, ok, stream);
}

__attribute__((visibility("default")))
int grws_sanitize_columns(int32_t *cols, void *vals, int val_dtype, int64_t num_tiles, int64_t num_cols, void *stream) {
    GRWS_REQUIRE(num_tiles >= 0 && num_cols >= 0, "negative size");
    if (num_tiles == 0) return GRWS_OK;
    GRWS_REQUIRE(cols && vals, "null pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t n = num_tiles * TILE_COLS;
    switch (val_dtype) {
        case GRWS_F32: sanitize_columns_kernel<float><<<nblocks(n, 256), 256, 0, st>>>(cols, (float *)vals, n, num_cols); break;
        case GRWS_F16: sanitize_columns_kernel<__half><<<nblocks(n, 256), 256, 0, st>>>(cols, (__half *)vals, n, num_cols); break;
        case GRWS_BF16: sanitize_columns_kernel<__nv_bfloat16><<<nblocks(n, 256), 256, 0, st>>>(cols, (__nv_bfloat16 *)vals, n, num_cols); break;
        default: return fail(GRWS_ERR_UNSUPPORTED, "bad value dtype %d", val_dtype);
    }
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

// ---------------------------------------------------------------------------------------------
// All hops of one mini-batch in one call: sample, dedup / reindex, block build, per hop, with
// every buffer sized by a bound that the host knows from (num_seeds, fanouts) alone, so nothing
// is read back between the hops.
// ---------------------------------------------------------------------------------------------
__attribute__((visibility("default")))
int grws_sample_layers_sizes(int64_t num_seeds, const int *fanouts, int num_hops, int64_t pad_to,
                             int64_t *n_dst, int64_t *n_src, int64_t *tiles_bound) {
    GRWS_REQUIRE(num_seeds >= 0 && num_hops >= 1 && num_hops <= 16 && fanouts && pad_to >= 0, "bad argument");
    int64_t d = num_seeds;
    for (int h = 0; h < num_hops; ++h) {
        GRWS_REQUIRE(fanouts[h] > 0 && fanouts[h] <= MAX_FANOUT, "fanout %d outside [1, %d]", fanouts[h], MAX_FANOUT);
        int64_t s = d * (1 + (int64_t)fanouts[h]);
        if (pad_to > 1) s = ceil_div(s, pad_to) * pad_to;
        GRWS_REQUIRE(s < 0x7fffffffLL, "hop %d too large", h);
        if (n_dst) n_dst[h] = d;
        if (n_src) n_src[h] = s;
        if (tiles_bound) tiles_bound[h] = d * fanouts[h] / TILE_COLS + ceil_div(d, TILE_ROWS);
        d = s;
    }
    return GRWS_OK;
}

// builder scratch, defined in bcsr_build.cu
size_t grws_csr_to_bcsr_scratch_bytes(int64_t num_rows, int64_t nnz);
int grws_block_build_count(const int32_t *local, const float *w, int64_t n_dst, int fanout, int64_t num_cols_bound,
                           int64_t *window_offset, void *scratch, size_t scratch_bytes, void *stream);

struct LayersScratch {
    int32_t *nbr, *local, *cnt;
    float *w;
    void *dedup, *build;
    size_t dedup_bytes, build_bytes, total;
    // where the new nodes are ranked by a bitmap (instead of `dedup`)
    bool bitmap;
    int32_t *keys, *vals, *counters;
    uint32_t *bits;                                  // [num_hops * words]
    HopRank rank;
    int64_t slots;
};

// The bitmap is cleared, counted and walked as a whole in every hop, so it is for graphs that are not too large for the
// batch: a sort of a few thousand new ids is one launch, one of more takes 40 us and up.  A mini-batch with the bitmap /
// with sorts, us, by its seeds and fan-outs (list slots of all hops: 1.3 k, 31 k, 39 k, 1.1 M):
//   nodes      37, 5-5     256, 10-10   37, 15-10-5   1024, 15-10-5
//   2.4 M     148 / 170     160 / 237     204 / 335      312 / 543
//    20 M     179 / 165     175 / 227     226 / 326      308 / 490
//    50 M     238 / 163     204 / 220     270 / 327      342 / 476
//   111 M     357 / 172     262 / 224     357 / 326      440 / 472
static bool ranks_by_bitmap(int64_t num_nodes, const int64_t *n_dst, const int *fanouts, int num_hops) {
    int64_t slots = 0;
    for (int h = 0; h < num_hops; ++h) slots += n_dst[h] * fanouts[h];
    return num_nodes > 0 && ceil_div(num_nodes, 32) <= 450000 + 60 * (slots < 40000 ? slots : 40000) + slots;
}

static int carve_layers(void *base, int64_t num_nodes, int64_t num_seeds, const int *fanouts, int num_hops, int64_t pad_to, LayersScratch *out) {
    int64_t n_dst[16], n_src[16];
    if (int st = grws_sample_layers_sizes(num_seeds, fanouts, num_hops, pad_to, n_dst, n_src, nullptr)) return st;
    const bool bitmap = ranks_by_bitmap(num_nodes, n_dst, fanouts, num_hops);
    size_t entries = 1, rows = 1, dedup = 0, build = 0;
    int64_t nodes = 1;
    for (int h = 0; h < num_hops; ++h) {
        const size_t e = (size_t)n_dst[h] * fanouts[h];
        if (e > entries) entries = e;
        if ((size_t)n_dst[h] > rows) rows = (size_t)n_dst[h];
        if (n_src[h] > nodes) nodes = n_src[h];
        const size_t d = bitmap ? 0 : carve_dedup(nullptr, n_dst[h], fanouts[h]).total;
        const size_t b = grws_csr_to_bcsr_scratch_bytes(n_dst[h], (int64_t)e);
        if (d > dedup) dedup = d;
        if (b > build) build = b;
    }
    // the buffers start on 256-byte boundaries (the table is cleared in 16-byte pieces), wherever the caller's scratch does
    char *p = reinterpret_cast<char *>(up256(reinterpret_cast<uintptr_t>(base)));
    size_t off = 0;
    auto take = [&](size_t bytes) { char *q = p ? p + off : nullptr; off += up256(bytes); return (void *)q; };
    out->nbr = (int32_t *)take(entries * 4);
    out->w = (float *)take(entries * 4);
    out->local = (int32_t *)take(entries * 4);
    out->cnt = (int32_t *)take(rows * 4);
    out->dedup = take(dedup);
    out->build = take(build);
    out->dedup_bytes = dedup;
    out->build_bytes = build;
    out->bitmap = bitmap;
    if (bitmap) {
        int64_t slots = 64;
        while (slots < 2 * nodes + 16) slots <<= 1;  // every node of the batch: the last source list holds them all
        const int64_t words = ceil_div(num_nodes, 32);
        out->slots = slots;
        out->rank.words = words;
        out->rank.num_nodes = num_nodes;
        out->keys = (int32_t *)take((size_t)slots * 4);
        out->vals = (int32_t *)take((size_t)slots * 4);
        out->bits = (uint32_t *)take((size_t)words * num_hops * 4);
        out->counters = (int32_t *)take((size_t)num_hops * 16);
        out->rank.prefix = (int32_t *)take((size_t)words * 4);
        out->rank.sums = (int32_t *)take((size_t)ceil_div(words, RANK_THREADS) * 4);
        out->rank.over = (int32_t *)take(entries * 4);
        out->rank.merged = (int32_t *)take(entries * 4);
    }
    out->total = off + 255;
    return GRWS_OK;
}

__attribute__((visibility("default")))
size_t grws_sample_layers_scratch_bytes(int64_t num_seeds, const int *fanouts, int num_hops, int64_t pad_to) {
    return grws_sample_layers_sized_scratch_bytes(0, num_seeds, fanouts, num_hops, pad_to);
}

__attribute__((visibility("default")))
size_t grws_sample_layers_sized_scratch_bytes(int64_t num_nodes, int64_t num_seeds, const int *fanouts, int num_hops, int64_t pad_to) {
    LayersScratch s = {};
    if (num_nodes < 0 || carve_layers(nullptr, num_nodes, num_seeds, fanouts, num_hops, pad_to, &s) != GRWS_OK) return 0;
    return s.total;
}

__attribute__((visibility("default")))
int grws_sample_layers(const int64_t *row_ptr, const int32_t *col_idx, const float *values, const int32_t *seeds,
                       int64_t num_seeds, const int *fanouts, int num_hops, uint64_t seed, const uint64_t *seed_dev,
                       int64_t pad_to, int val_dtype, int32_t *const *out_src, int64_t *const *out_window_offset,
                       int32_t *const *out_cols, void *const *out_vals, int64_t *out_counts, void *scratch,
                       size_t scratch_bytes, void *stream) {
    return grws_sample_layers_sized(row_ptr, 0, col_idx, values, seeds, num_seeds, fanouts, num_hops, seed, seed_dev, pad_to, val_dtype,
                                    out_src, out_window_offset, out_cols, out_vals, out_counts, scratch, scratch_bytes, stream);
}

__attribute__((visibility("default")))
int grws_sample_layers_sized(const int64_t *row_ptr, int64_t num_nodes, const int32_t *col_idx, const float *values,
                             const int32_t *seeds, int64_t num_seeds, const int *fanouts, int num_hops, uint64_t seed,
                             const uint64_t *seed_dev, int64_t pad_to, int val_dtype, int32_t *const *out_src,
                             int64_t *const *out_window_offset, int32_t *const *out_cols, void *const *out_vals, int64_t *out_counts,
                             void *scratch, size_t scratch_bytes, void *stream) {
    GRWS_REQUIRE(num_nodes >= 0 && num_nodes < 0x7fffffffLL, "node count outside [0, 2^31)");
    GRWS_REQUIRE(row_ptr && col_idx && (seeds || num_seeds == 0) && out_src && out_window_offset && out_cols && out_vals && scratch,
                 "null pointer");
    GRWS_REQUIRE(val_dtype >= GRWS_F32 && val_dtype <= GRWS_BF16, "bad value dtype %d", val_dtype);
    int64_t n_dst[16], n_src[16], tiles[16];
    if (int st = grws_sample_layers_sizes(num_seeds, fanouts, num_hops, pad_to, n_dst, n_src, tiles)) return st;
    LayersScratch s = {};
    if (int st = carve_layers(scratch, num_nodes, num_seeds, fanouts, num_hops, pad_to, &s)) return st;
    if (scratch_bytes < s.total) return fail(GRWS_ERR_SCRATCH, "sample_layers scratch too small: %zu < %zu", scratch_bytes, s.total);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int32_t *dst = seeds;
    const uint32_t table_mask = (uint32_t)(s.slots - 1);
    const unsigned rank_blocks = (unsigned)ceil_div(s.rank.words, RANK_THREADS);
    if (s.bitmap && num_seeds > 0) {
        const unsigned nb = nblocks(s.slots / 4, 256);
        layers_init_kernel<<<nb > 1184 ? 1184 : nb, 256, 0, st>>>(s.keys, s.vals, s.slots, s.bits, s.rank.words * num_hops, s.counters, 4 * num_hops);
        insert_seeds_kernel<<<nblocks(num_seeds, 256), 256, 0, st>>>(seeds, num_seeds, s.keys, s.vals, table_mask);
    }
    for (int h = 0; h < num_hops; ++h) {
        const int64_t nd = n_dst[h], f = fanouts[h], n_entries = nd * f, W = ceil_div(nd, (int64_t)TILE_ROWS);
        GRWS_REQUIRE(out_src[h] && out_window_offset[h] && (tiles[h] == 0 || (out_cols[h] && out_vals[h])), "null output of hop %d", h);
        if (nd == 0) {
            GRWS_CUDA_TRY(cudaMemsetAsync(out_window_offset[h], 0, 8, st));
            if (n_src[h] > 0) GRWS_CUDA_TRY(cudaMemsetAsync(out_src[h], 0xff, (size_t)n_src[h] * 4, st));
            if (out_counts) GRWS_CUDA_TRY(cudaMemsetAsync(out_counts + 4 * h, 0, 32, st));
            dst = out_src[h];
            continue;
        }
        // 1. neighbours of every frontier node (padding entries of the frontier, -1, get empty lists)
        if (int e = launch_sample_hop(row_ptr, col_idx, values, dst, nd, (int)f, seed, seed_dev, (uint32_t)h, s.nbr, s.w, s.cnt, st)) return e;
        // 2. source list = frontier ++ ascending new nodes ++ -1 padding; local id of every neighbour
        const int32_t *n_new;
        if (s.bitmap) {
            HopRank r = s.rank;
            r.bits = s.bits + s.rank.words * h;
            r.counters = s.counters + 4 * h;
            insert_marked_kernel<<<nblocks(n_entries, 256), 256, 0, st>>>(s.nbr, n_entries, s.keys, table_mask, r);
            const unsigned run_blocks = (unsigned)ceil_div(n_entries, (int64_t)OVER_RUN);
            rank_sums_kernel<<<rank_blocks + run_blocks, RANK_THREADS, 0, st>>>(r, (int)rank_blocks);
            const unsigned emit_blocks = nblocks(n_src[h], 4 * RANK_THREADS);
            emit_sources_kernel<<<emit_blocks > rank_blocks ? emit_blocks : rank_blocks, RANK_THREADS, 0, st>>>(r, dst, nd, n_src[h], out_src[h]);
            localize_ranked_kernel<<<nblocks(n_entries, 256), 256, 0, st>>>(s.nbr, n_entries, nd, s.keys, s.vals, table_mask, r, s.local, out_src[h]);
            n_new = r.counters;
        } else {
            const DedupScratch d = carve_dedup(s.dedup, nd, (int)f);
            const uint32_t mask = d.slots - 1;
            const int64_t init_n = (int64_t)d.slots > n_src[h] ? (int64_t)d.slots : n_src[h];
            dedup_init_kernel<<<nblocks(init_n, 256) > 1184 ? 1184 : nblocks(init_n, 256), 256, 0, st>>>(
                d.keys, d.vals, d.slots, d.cand, n_entries + 1, d.n_new, out_src[h] + nd, n_src[h] - nd);
            insert_dst_kernel<<<nblocks(nd, 256), 256, 0, st>>>(dst, nd, d.keys, d.vals, mask, out_src[h]);
            insert_nbr_kernel<<<nblocks(n_entries, 256), 256, 0, st>>>(s.nbr, n_entries, d.keys, d.vals, mask, d.cand, d.n_new);
            size_t tmp = d.cub_bytes;
            GRWS_CUDA_TRY(cub::DeviceRadixSort::SortKeys(d.cub_tmp, tmp, d.cand, d.cand_sorted, (int)n_entries, 0, 32, st));
            rank_new_kernel<<<nblocks(n_entries, 256), 256, 0, st>>>(d.cand_sorted, d.n_new, nd, d.keys, d.vals, mask, out_src[h]);
            localize_flat_kernel<<<nblocks(n_entries, 256), 256, 0, st>>>(s.nbr, n_entries, d.keys, d.vals, mask, s.local);
            n_new = d.n_new;
        }
        // 3. the hop's BCSR block straight from the fixed-stride lists
        if (int e = grws_block_build_count(s.local, s.w, nd, (int)f, n_src[h], out_window_offset[h], s.build, s.build_bytes, stream)) return e;
        if (int e = block_build_fill(nd, (int)f, out_window_offset[h], tiles[h], out_cols[h], out_vals[h], val_dtype, s.build,
                                     s.build_bytes, st)) return e;
        if (out_counts)
            hop_counts_kernel<<<1, 1024, 0, st>>>(n_new, dst, nd, s.cnt, out_window_offset[h], W, out_counts + 4 * h);
        GRWS_CUDA_TRY(cudaGetLastError());
        dst = out_src[h];
    }
    return GRWS_OK;
}

}  // extern "C"
