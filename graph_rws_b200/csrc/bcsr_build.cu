// Device-side BCSR construction.
//
//   CSR -> BCSR: the layout contract of csr_to_bcsr_cpu (core/wrapper/convert_wrapper.cpp:27-180).
//   The entries of a 16-row window are one contiguous range of the CSR arrays, so a window is
//   built by itself: its entries are ordered by (column, row), equal columns become one column
//   slot, slot / 8 is the tile, and the last duplicate of a (row, column) pair wins
//   (convert_wrapper.cpp:174).  A window of up to 512 entries is read once per phase, a larger one four
//   to six times by its CTA when it is counted, whatever its columns span.
//
//   BCSR -> transposed CSR: extracts the non-zero entries of the tiles as (column, row, value)
//   so that the transposed adjacency can be built once, cached and multiplied with the forward
//   kernel; this replaces the per-call atomic scatter of spmm_bcsr_transpose_atomic_kernel
//   (core/include/spmm_tc.cuh:211-270).
//
// cub::DeviceScan (CUDA toolkit) does the prefix sums over windows and columns.
#include <cub/cub.cuh>

#include "grws_common.cuh"

namespace grws {

// A window of up to SMALL_ENTRIES entries is sorted by one warp in registers (16 keys a lane); a larger
// one is ranked by a CTA through a bitmap of its columns, or by a sort where they span more than that.
// 512 covers every block of a sampled step up to fan-out 32, and all but the hub windows of a power-law
// graph of up to about 25 entries a row; 32 keys a lane would spill.
constexpr int SMALL_ENTRIES = 512;
constexpr int COUNT_WARPS = 8;
constexpr int LARGE_THREADS = 1024;
constexpr int BITMAP_WORDS = 16384;                // columns of a bitmap / 32
constexpr uint32_t BITMAP_COLS = BITMAP_WORDS * 32u;
constexpr int SORT_ENTRIES = 8 * LARGE_THREADS;    // entries of a large window that are sorted at a time where its columns span more than a bitmap
constexpr int PART_BINS = 2048;                    // column ranges that such a window's entries are divided into first, if they are more
constexpr int LARGE_SMEM = BITMAP_WORDS * 4 + BITMAP_WORDS / 2 * 4;   // bits + one prefix per word pair: two CTAs per SM
constexpr int LARGE_PLAIN = 1 << 30;               // flags in BuildScratch::large (there are fewer than 2^28 windows)
constexpr int LARGE_WIDE = 1 << 29, LARGE_MIXED = 1 << 28;      // within count_large_kernel: still to be numbered; in no order
constexpr int FILL_WARPS = 8;
constexpr int FILL_BYTES = 4096;                   // tiles a warp assembles in shared memory at a time
constexpr int FILL_LARGE_THREADS = 512;            // one warp per row of a window
constexpr int FILL_AHEAD = 8;                      // times 32 entries of a row in flight where their order is kept (a hub's row has thousands)

static inline size_t align_up(size_t x, size_t a = 256) { return (x + a - 1) / a * a; }

// The entries of a matrix by rows: a CSR (row_ptr set), or fixed-stride lists of `fanout` slots per row
// whose empty slots hold a negative id.
struct EntrySource {
    const int64_t *row_ptr;
    const int32_t *col;
    const float *val;
    int64_t num_rows;
    int fanout;
    bool unique;            // the caller knows that no (row, column) pair occurs twice
    __device__ __forceinline__ int64_t row_start(int64_t r) const {
        r = r < num_rows ? r : num_rows;
        return row_ptr ? row_ptr[r] : r * fanout;
    }
    // lists: a negative id is an empty slot; CSR ids are taken as they are (ordered as unsigned)
    __device__ __forceinline__ bool empty(int32_t c) const { return row_ptr == nullptr && c < 0; }
};

// Scratch shared by the count and fill phases.
//   rec, of a window of at most SMALL_ENTRIES entries (ordered by column slot):
//         column << 32 | slot << 5 | row in window << 1 | 1 if the entry is not written (an empty list
//         slot, or an earlier duplicate of the same row and column)
//   rec, of a larger window (in the order of the source): column << 32 | slot, all ones for an empty slot or an entry
//         that a later one of the same place takes the place of
struct BuildScratch {
    uint64_t *rec;
    float *val;             // value of the entry rec describes
    int32_t *row_start;     // [num_rows + 1]
    int64_t *tiles;         // [W+1] tiles per window, shifted by one
    int32_t *large;         // [1 + W] number of large windows, then their ids in no fixed order (bit 30: no two of its
                            // entries have one place, so they can be written in any order)
    int32_t *columns;       // [W] distinct columns of the large window listed at that place
    int32_t *ucol;          // column of every slot of a large window, from its first entry's place on
    void *cub_tmp;
    size_t cub_bytes;
    size_t total;
};

static size_t scan_temp_bytes(int64_t n) {
    size_t s = 0;
    cub::DeviceScan::InclusiveSum(nullptr, s, (const int64_t *)nullptr, (int64_t *)nullptr, (int)n);
    return s;
}

static BuildScratch carve(void *base, int64_t nnz, int64_t num_rows) {
    BuildScratch s;
    const int64_t W = ceil_div(num_rows, TILE_ROWS);
    char *p = static_cast<char *>(base);
    size_t off = 0;
    auto take = [&](size_t bytes) { char *q = p ? p + off : nullptr; off += align_up(bytes); return (void *)q; };
    const size_t n = (size_t)(nnz > 0 ? nnz : 1);
    s.rec = (uint64_t *)take(n * 8);
    s.val = (float *)take(n * 4);
    s.row_start = (int32_t *)take((size_t)(num_rows + 1) * 4);
    s.tiles = (int64_t *)take((size_t)(W + 1) * 8);
    s.large = (int32_t *)take((size_t)(W + 1) * 4);
    s.columns = (int32_t *)take((size_t)(W + 1) * 4);
    s.ucol = (int32_t *)take(n * 4);
    s.cub_bytes = scan_temp_bytes(W + 1);
    s.cub_tmp = take(s.cub_bytes);
    s.total = off;
    return s;
}

// Ascending bitonic sort of 32 * E keys held by one warp; key i is k[i % E] of lane i / E.
template <int E, typename Key>
__device__ __forceinline__ void warp_sort(Key (&k)[E], int lane) {
#pragma unroll
    for (int size = 2; size <= 32 * E; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= E) {
                const int ls = stride / E;
                const bool up = (lane & (size / E)) == 0;            // size == 32 * E: every lane's bit is 0
                const bool keep_min = ((lane & ls) == 0) == up;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const Key o = __shfl_xor_sync(0xffffffffu, k[e], ls);
                    k[e] = keep_min ? min(k[e], o) : max(k[e], o);
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    if (e & stride) continue;
                    const bool up = size < E ? (e & size) == 0 : (lane & (size / E)) == 0;
                    const Key lo = min(k[e], k[e + stride]), hi = max(k[e], k[e + stride]);
                    k[e] = up ? lo : hi;
                    k[e + stride] = up ? hi : lo;
                }
            }
        }
    }
}

// Gives every distinct column of one window its slot and writes the records in order.  A key is
// column << POS_BITS | position; the rows ascend with the position, so this is also the order by (column, row,
// position).  `ends`: in lanes 0..15, where the entries of that row end, counted from the window's first.
constexpr int POS_BITS = 9;                                           // SMALL_ENTRIES positions
template <int E, typename Key>
__device__ __forceinline__ int rank_window(Key (&k)[E], const EntrySource &src, int64_t s, int m, int ends, int lane,
                                           uint64_t *__restrict__ rec, float *__restrict__ val) {
    constexpr Key NONE = ~Key(0);
    warp_sort<E, Key>(k, lane);
    const Key before = __shfl_up_sync(0xffffffffu, k[E - 1], 1), after = __shfl_down_sync(0xffffffffu, k[0], 1);
    auto row_of = [&](Key key) {                                      // number of rows that end at or before the entry
        const int p = (int)(key & ((1u << POS_BITS) - 1u));
        int row = 0;
#pragma unroll
        for (int step = TILE_ROWS / 2; step > 0; step >>= 1) row += p >= __shfl_sync(0xffffffffu, ends, row + step - 1) ? step : 0;
        return row;
    };
    uint32_t heads = 0;                                               // bit e: key e opens a column
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const Key prev = e == 0 ? before : k[e > 0 ? e - 1 : 0];
        if (k[e] != NONE && ((e == 0 && lane == 0) || (prev >> POS_BITS) != (k[e] >> POS_BITS))) heads |= 1u << e;
    }
    int incl = __popc(heads);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    int slot = incl - 1, next_row = __shfl_down_sync(0xffffffffu, row_of(k[0]), 1);
#pragma unroll
    for (int e = E - 1; e >= 0; --e) {
        const int i = lane * E + e, row = row_of(k[e]);
        const Key next = e == E - 1 ? (lane == 31 ? NONE : after) : k[e < E - 1 ? e + 1 : 0];
        const bool drop = k[e] == NONE || (next != NONE && (next >> POS_BITS) == (k[e] >> POS_BITS) && next_row == row);
        if (i < m) {
            const uint32_t col = (uint32_t)(k[e] >> POS_BITS);
            rec[s + i] = (uint64_t)col << 32 | (uint64_t)((uint32_t)slot << 5 | (uint32_t)row << 1 | (drop ? 1u : 0u));
            val[s + i] = drop ? 0.f : __ldg(src.val + s + (int)(k[e] & ((1u << POS_BITS) - 1u)));
        }
        slot -= heads >> e & 1u;
        next_row = row;
    }
    return __shfl_sync(0xffffffffu, incl, 31);
}

// Keys of 32 bits where the window's columns leave room for the position (ids below 2^23 - 1: a min or max is one
// instruction then, and a key one shuffle), of 64 bits otherwise.  Both directions of a 169 k-node graph: 153 us with
// 64-bit keys throughout, 87 us with 32-bit ones.
template <int E>
__device__ __forceinline__ int sort_window(const EntrySource &src, int64_t s, int m, int ends, int lane,
                                           uint64_t *__restrict__ rec, float *__restrict__ val) {
    uint32_t c[E], live = 0, top = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int p = e * 32 + lane;
        const int32_t x = p < m ? __ldg(src.col + s + p) : 0;
        c[e] = (uint32_t)x;
        if (p < m && !src.empty(x)) {
            live |= 1u << e;
            top = max(top, c[e]);
        }
    }
    if (__reduce_max_sync(0xffffffffu, top) < (1u << (32 - POS_BITS)) - 1u) {
        uint32_t k[E];
#pragma unroll
        for (int e = 0; e < E; ++e) k[e] = live >> e & 1u ? c[e] << POS_BITS | (uint32_t)(e * 32 + lane) : ~0u;
        return rank_window<E, uint32_t>(k, src, s, m, ends, lane, rec, val);
    }
    unsigned long long k[E];
#pragma unroll
    for (int e = 0; e < E; ++e) k[e] = live >> e & 1u ? (unsigned long long)c[e] << POS_BITS | (uint32_t)(e * 32 + lane) : ~0ull;
    return rank_window<E, unsigned long long>(k, src, s, m, ends, lane, rec, val);
}

// One warp per window.  Bound by fetching its instructions and by the latency of its loads: warps stand 2.9 and 3.2 cycles an
// instruction for them on a 169 k-node graph (10,584 windows), up to 9 and 2 on a sampled block, the pipes are 42 % and
// less busy.  The sorting networks are unrolled for five sizes and two key widths, so that the time depends a
// little on where the linker puts them (36 or 40 us for the three hops of a mini-batch).  Against one radix sort of 64-bit (window, column, row) keys over all
// entries -- five to seven passes over keys and values, flags, two scans -- a mini-batch of 1,024 seeds and
// fan-out 15-10-5 was sampled and built in 519 us instead of 769.
__global__ void __launch_bounds__(COUNT_WARPS * 32, 3)
count_windows_kernel(const EntrySource src, int64_t W, BuildScratch s) {
    const int lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * COUNT_WARPS + (threadIdx.x >> 5);
    if (w >= W) return;
    const int64_t r0 = w * TILE_ROWS, row = r0 + lane;
    const int64_t end = src.row_start(row + 1);                       // rows past the last one are empty
    const int64_t first = __shfl_sync(0xffffffffu, src.row_start(r0), 0);
    const int64_t total = __shfl_sync(0xffffffffu, end, TILE_ROWS - 1) - first;
    if (lane < TILE_ROWS && row < src.num_rows) s.row_start[row + 1] = (int32_t)end;
    if (w == 0 && lane == 0) { s.row_start[0] = (int32_t)first; s.tiles[0] = 0; }
    if (total > SMALL_ENTRIES) {
        if (lane == 0) s.large[1 + atomicAdd(s.large, 1)] = (int32_t)w;
        return;
    }
    const int m = (int)total, ends = (int)(end - first);
    int n = 0;
    if (m > 256) n = sort_window<16>(src, first, m, ends, lane, s.rec, s.val);
    else if (m > 128) n = sort_window<8>(src, first, m, ends, lane, s.rec, s.val);
    else if (m > 64) n = sort_window<4>(src, first, m, ends, lane, s.rec, s.val);
    else if (m > 32) n = sort_window<2>(src, first, m, ends, lane, s.rec, s.val);
    else if (m > 0) n = sort_window<1>(src, first, m, ends, lane, s.rec, s.val);
    if (lane == 0) s.tiles[w + 1] = (n + TILE_COLS - 1) / TILE_COLS;
}

__device__ __forceinline__ uint32_t block_reduce(uint32_t v, bool take_min, uint32_t *warp_part) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = take_min ? __reduce_min_sync(0xffffffffu, v) : __reduce_max_sync(0xffffffffu, v);
    __syncthreads();                                                  // the previous use of warp_part is over
    if (lane == 0) warp_part[warp] = v;
    __syncthreads();
    v = warp_part[lane];                                              // LARGE_THREADS / 32 == 32 warps
    return take_min ? __reduce_min_sync(0xffffffffu, v) : __reduce_max_sync(0xffffffffu, v);
}

// exclusive prefix sum over a block of LARGE_THREADS.  FREE: a barrier has passed since warp_part was read last.
template <bool FREE = false>
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t *warp_part, uint32_t *all) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    if (!FREE) __syncthreads();                                       // the previous use of warp_part is over
    if (lane == 31) warp_part[warp] = incl;
    __syncthreads();
    const uint32_t part = warp_part[lane];
    const uint32_t ahead = __reduce_add_sync(0xffffffffu, lane < warp ? part : 0u);
    *all = __reduce_add_sync(0xffffffffu, part);
    return ahead + incl - v;
}

// Ascending bitonic sort of LARGE_THREADS * E keys by a CTA; key i is k[i % E] of thread i / E.  Every warp sorts its own in
// registers; a merge of sorted halves compares a key with its mirror image first, so that all of them ascend, and
// only the exchanges between warps go through shared memory (15, in two buffers by turns: one barrier each).
template <int E>
__device__ __forceinline__ void block_sort(uint32_t (&k)[E], uint32_t *buf) {
    const int tid = threadIdx.x, lane = tid & 31;
    warp_sort<E, uint32_t>(k, lane);
    int turn = 0;
    for (int warps = 2; warps <= LARGE_THREADS / 32; warps <<= 1) {
        for (int d = warps * 32 - 1; d >= 32; d = d == warps * 32 - 1 ? warps * 8 : d >> 1) {
            uint32_t *b = buf + turn * LARGE_THREADS * E;
            const bool mirror = d == warps * 32 - 1, low = (tid & (mirror ? warps * 16 : d)) == 0;
            turn ^= 1;
#pragma unroll
            for (int e = 0; e < E; ++e) b[e * LARGE_THREADS + tid] = k[e];
            __syncthreads();
#pragma unroll
            for (int e = 0; e < E; ++e) {
                const uint32_t o = b[(mirror ? E - 1 - e : e) * LARGE_THREADS + (tid ^ d)];
                k[e] = low ? min(k[e], o) : max(k[e], o);
            }
        }
#pragma unroll
        for (int stride = 16 * E; stride > 0; stride >>= 1) {
            if (stride >= E) {
                const bool low = (lane & (stride / E)) == 0;
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    const uint32_t o = __shfl_xor_sync(0xffffffffu, k[e], stride / E);
                    k[e] = low ? min(k[e], o) : max(k[e], o);
                }
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) {
                    if (e & stride) continue;
                    const uint32_t x = k[e], y = k[e + stride];
                    k[e] = min(x, y);
                    k[e + stride] = max(x, y);
                }
            }
        }
    }
    __syncthreads();                                                  // the buffers are free again
}

// Entries of one large window, in the order of the source
struct LargeWindow {
    EntrySource src;
    const int32_t *col;
    int64_t m;
    uint64_t *rec;
    int32_t *ucol;
    __device__ __forceinline__ LargeWindow(const EntrySource &from, const BuildScratch &s, int64_t w) : src(from) {
        const int64_t first = src.row_start(w * TILE_ROWS);
        m = src.row_start((w + 1) * TILE_ROWS) - first;
        col = src.col + first;
        rec = s.rec + first;
        ucol = s.ucol + first;
    }
};
extern __shared__ uint32_t large_smem[];             // LARGE_SMEM bytes
__device__ __forceinline__ uint32_t *large_part() {  // two words per warp
    __shared__ uint32_t part[2 * (LARGE_THREADS / 32)];
    return part;
}

// Numbers the columns of the m entries `entry` gives, which lie in [from, to], by a bitmap in shared memory (one per round:
// a range wider than the bitmap takes several, each from the smallest column not yet numbered) and a prefix sum of
// its bit counts.  Writes the records and the columns of the slots from `total` on; returns their end.
// ONE: the range is no wider than the bitmap (and the caller passes a barrier before shared memory is used again).
template <bool ONE, typename Entry>
__device__ __forceinline__ uint32_t number_by_bitmap(const LargeWindow &win, int64_t m, const Entry &entry, uint32_t from, uint32_t to, uint32_t total) {
    const int tid = threadIdx.x;
    uint32_t *bits = large_smem, *prefix = large_smem + BITMAP_WORDS;
    bool more = true;
    while (more) {
        const uint64_t left = (uint64_t)to - from + 1;
        const uint32_t span = left < BITMAP_COLS ? (uint32_t)left : BITMAP_COLS;
        const int pairs = (int)((span + 63) / 64);
        for (int i = tid; i < pairs; i += LARGE_THREADS) reinterpret_cast<uint2 *>(bits)[i] = make_uint2(0u, 0u);
        __syncthreads();
        uint32_t next = 0xffffffffu;
        bool beyond = false;
        for (int64_t k = tid; k < m; k += LARGE_THREADS) {
            const int32_t c = __ldg(win.col + entry(k));
            if (win.src.empty(c) || (!ONE && (uint32_t)c < from)) continue;
            const uint32_t x = (uint32_t)c - from;
            if (ONE || x < span) {
                atomicOr(bits + (x >> 5), 1u << (x & 31));
            } else {
                beyond = true;
                next = min(next, (uint32_t)c);
            }
        }
        if (ONE) { more = false; __syncthreads(); } else more = __syncthreads_or(beyond);
        // exclusive prefix of the bit counts, one word pair at a time per thread
        const int each = (pairs + LARGE_THREADS - 1) / LARGE_THREADS, p0 = tid * each, p1 = min(pairs, p0 + each);
        uint32_t sum = 0, round;
        for (int i = p0; i < p1; ++i) {
            const uint2 v = reinterpret_cast<uint2 *>(bits)[i];
            sum += __popc(v.x) + __popc(v.y);
        }
        uint32_t at = total + block_exclusive<true>(sum, large_part(), &round);
        for (int i = p0; i < p1; ++i) {
            const uint2 v = reinterpret_cast<uint2 *>(bits)[i];
            prefix[i] = at;
            const uint32_t c0 = from + (uint32_t)i * 64;
            for (uint32_t b = v.x; b; b &= b - 1) win.ucol[at++] = (int32_t)(c0 + __ffs(b) - 1);
            for (uint32_t b = v.y; b; b &= b - 1) win.ucol[at++] = (int32_t)(c0 + 31 + __ffs(b));
        }
        __syncthreads();
        for (int64_t k = tid; k < m; k += LARGE_THREADS) {
            const int64_t i = entry(k);
            const int32_t c = __ldg(win.col + i);
            if (win.src.empty(c) || (!ONE && (uint32_t)c < from)) continue;
            const uint32_t x = (uint32_t)c - from;
            if (!ONE && x >= span) continue;
            const uint2 v = reinterpret_cast<uint2 *>(bits)[x >> 6];
            const uint32_t below = (1u << (x & 31)) - 1u;
            const uint32_t slot = prefix[x >> 6] + (x & 32 ? __popc(v.x) + __popc(v.y & below) : __popc(v.x & below));
            win.rec[i] = (uint64_t)(uint32_t)c << 32 | slot;
        }
        total += round;
        if (more) from = block_reduce(next, true, large_part());
        if (!ONE) __syncthreads();                                    // bits and prefix are free again
    }
    return total;
}

// The same by a sort of at most LARGE_THREADS * E entries, whatever their columns span
template <int E, typename Entry>
__device__ __forceinline__ uint32_t number_by_sort(const LargeWindow &win, int m, const Entry &entry, uint32_t total) {
    const int tid = threadIdx.x;
    uint32_t k[E], real = 0, found;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        k[e] = 0xffffffffu;                                           // behind or beside the largest column
        const int i = e * LARGE_THREADS + tid;
        const int32_t c = i < m ? __ldg(win.col + entry(i)) : 0;
        if (i < m && !win.src.empty(c)) { k[e] = (uint32_t)c; ++real; }
    }
    block_exclusive(real, large_part(), &real);
    block_sort<E>(k, large_smem);
    large_smem[tid] = k[E - 1];                                         // the last key of every thread
    __syncthreads();
    uint32_t before = tid ? large_smem[tid - 1] : 0u, heads = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const uint32_t i = (uint32_t)(tid * E + e);
        if (i < real && (i == 0 || k[e] != before)) heads |= 1u << e;
        before = k[e];
    }
    uint32_t *distinct = large_smem + LARGE_THREADS * E, at = block_exclusive(__popc(heads), large_part(), &found);
#pragma unroll
    for (int e = 0; e < E; ++e)
        if (heads >> e & 1u) distinct[at++] = k[e];
    __syncthreads();
    for (int i = tid; i < (int)found; i += LARGE_THREADS) win.ucol[total + i] = (int32_t)distinct[i];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int j = e * LARGE_THREADS + tid;
        if (j >= m) break;
        const int64_t i = entry(j);
        const int32_t c = __ldg(win.col + i);
        if (!win.src.empty(c)) win.rec[i] = (uint64_t)(uint32_t)c << 32 | (total + (uint32_t)lower_bound(distinct, (int)found, (uint32_t)c));
    }
    __syncthreads();                                                  // the keys are free again
    return total + found;
}

template <typename Entry>
__device__ __forceinline__ uint32_t number_by_sort(const LargeWindow &win, int64_t m, const Entry &entry, uint32_t total) {
    if (m <= LARGE_THREADS) return number_by_sort<1>(win, (int)m, entry, total);
    if (m <= 2 * LARGE_THREADS) return number_by_sort<2>(win, (int)m, entry, total);
    if (m <= 4 * LARGE_THREADS) return number_by_sort<4>(win, (int)m, entry, total);
    return number_by_sort<8>(win, (int)m, entry, total);
}

// smallest and largest column of a large window; false: it has none.  One barrier: the caller passes another one before
// it is called again or large_part is written.
__device__ __forceinline__ bool column_span(const LargeWindow &win, uint32_t *lo_out, uint32_t *hi_out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *part = large_part(), lo = 0xffffffffu, hi = 0;
    for (int64_t i = threadIdx.x; i < win.m; i += LARGE_THREADS) {
        const int32_t c = __ldg(win.col + i);
        if (win.src.empty(c)) continue;
        lo = min(lo, (uint32_t)c);
        hi = max(hi, (uint32_t)c);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    if (lane == 0) {
        part[warp] = lo;
        part[LARGE_THREADS / 32 + warp] = hi;
    }
    __syncthreads();
    *lo_out = __reduce_min_sync(0xffffffffu, part[lane]);             // LARGE_THREADS / 32 == 32 warps
    *hi_out = __reduce_max_sync(0xffffffffu, part[LARGE_THREADS / 32 + lane]);
    return *lo_out <= *hi_out;
}

// The values of a large window; true where its rows are in strictly ascending order, that is, where every place at which
// the columns do not ascend lies between two rows
__device__ __forceinline__ bool copy_values(const LargeWindow &win, int64_t w, const float *__restrict__ from, float *__restrict__ to) {
    __shared__ int out_of_order;
    const int tid = threadIdx.x;
    if (tid == 0) out_of_order = 0;
    __syncthreads();
    int odd = 0;
    for (int64_t i = tid; i < win.m; i += LARGE_THREADS) {
        const int32_t c = __ldg(win.col + i);
        if (win.src.empty(c)) win.rec[i] = ~0ull;
        if (i + 1 < win.m && (uint32_t)c >= (uint32_t)__ldg(win.col + i + 1)) ++odd;
        to[i] = __ldg(from + i);
    }
    if (tid > 0 && tid < TILE_ROWS) {
        const int64_t first = win.src.row_start(w * TILE_ROWS);
        const int64_t at = win.src.row_start(w * TILE_ROWS + tid) - first, before = win.src.row_start(w * TILE_ROWS + tid - 1) - first;
        if (at > before && at < win.m && (uint32_t)__ldg(win.col + at - 1) >= (uint32_t)__ldg(win.col + at)) --odd;
    }
    if (odd) atomicAdd(&out_of_order, odd);
    __syncthreads();
    return out_of_order == 0;
}

// A large window whose columns span more than a few bitmaps is sorted in shared memory, so that its cost depends on its
// entries and not on the number of columns.  One of more than SORT_ENTRIES entries is divided by column ranges first
// (`order` lists them by range; it lies where their values will be) and goes on range by range, each with the way
// that takes it further.  Further bitmap rounds cost less where they are few and the entries many.  Whole builds, ms, with
// rounds / without: 4,800 entries a window, two rounds 2.2 / 2.6, three 2.5 / 2.5; 14,400 entries, six 3.5 / 3.7, eight
// 3.9 / 3.7; 96,000 entries, eight 5.6 / 7.7, twelve 6.6 / 7.7.
__device__ __forceinline__ uint32_t number_wide_window(const LargeWindow &win, uint32_t lo, uint32_t hi, int32_t *order) {
    __shared__ uint32_t bin_end[PART_BINS];
    const int tid = threadIdx.x;
    auto all_entries = [](int64_t k) { return k; };
    const uint32_t rounds = (hi - lo) / BITMAP_COLS + 1u;
    const uint32_t few = win.m > SORT_ENTRIES ? 7u + (uint32_t)min(win.m >> 14, (int64_t)7) : win.m > 2 * LARGE_THREADS ? 2u : 0u;
    if (rounds <= few)
        return number_by_bitmap<false>(win, win.m, all_entries, lo, hi, 0u);
    if (win.m <= SORT_ENTRIES) return number_by_sort(win, win.m, all_entries, 0u);
    int shift = 0;
    while ((hi - lo) >> shift >= (uint32_t)PART_BINS) ++shift;
    const int bins = (int)((hi - lo) >> shift) + 1;
    for (int i = tid; i < PART_BINS; i += LARGE_THREADS) bin_end[i] = 0;
    __syncthreads();
#pragma unroll 4
    for (int64_t i = tid; i < win.m; i += LARGE_THREADS) {
        const int32_t c = __ldg(win.col + i);
        if (!win.src.empty(c)) atomicAdd(bin_end + (((uint32_t)c - lo) >> shift), 1u);
    }
    __syncthreads();
    static_assert(PART_BINS == 2 * LARGE_THREADS, "two bins a thread");
    const uint32_t n0 = bin_end[2 * tid], n1 = bin_end[2 * tid + 1];
    uint32_t all;
    const uint32_t at = block_exclusive(n0 + n1, large_part(), &all);
    bin_end[2 * tid] = at;
    bin_end[2 * tid + 1] = at + n0;
    __syncthreads();
#pragma unroll 4
    for (int64_t i = tid; i < win.m; i += LARGE_THREADS) {
        const int32_t c = __ldg(win.col + i);
        if (!win.src.empty(c)) order[atomicAdd(bin_end + (((uint32_t)c - lo) >> shift), 1u)] = (int32_t)i;
    }
    __syncthreads();                                                  // bin_end now holds where each bin ends
    uint32_t total = 0;
    for (int bin = 0; bin < bins;) {
        const uint32_t k0 = bin ? bin_end[bin - 1] : 0u;
        const int by_width = (int)(BITMAP_COLS >> shift);             // bins a bitmap takes
        const int by_count = lower_bound(bin_end + bin, bins - bin, k0 + SORT_ENTRIES + 1u);       // bins a sort takes
        const int next = min(bins, bin + max(1, max(by_width, by_count)));
        const uint32_t from = lo + ((uint32_t)bin << shift), to = next < bins ? lo + ((uint32_t)next << shift) - 1u : hi;
        const int64_t m = bin_end[next - 1] - k0;
        const int32_t *mine = order + k0;
        auto entry = [mine](int64_t k) { return (int64_t)mine[k]; };
        bin = next;
        if (m == 0) continue;
        if (by_count > 0 && by_count >= by_width) total = number_by_sort(win, m, entry, total);
        else total = number_by_bitmap<false>(win, m, entry, from, to, total);
    }
    return total;
}

// Takes the records of all but the last entry of every (row, column slot) of a large window away.  A row is walked from its
// end, a chunk at a time, over a bitmap of the slots that have been met; entries of one slot in one chunk are told
// apart by a list of such slots.
__device__ __forceinline__ void drop_superseded(const LargeWindow &win, int64_t w, uint32_t total) {
    __shared__ int n_twice;
    uint32_t *bits = large_smem, *twice = large_smem + BITMAP_WORDS, *last = twice + LARGE_THREADS;
    const int tid = threadIdx.x;
    const int64_t first = win.src.row_start(w * TILE_ROWS);
    for (uint32_t base = 0; base < total; base += BITMAP_COLS) {
        const uint32_t span = min(total - base, BITMAP_COLS);
        for (int r = 0; r < TILE_ROWS; ++r) {
            const int64_t i0 = win.src.row_start(w * TILE_ROWS + r) - first, i1 = win.src.row_start(w * TILE_ROWS + r + 1) - first;
            for (int i = tid; i < (int)((span + 31) / 32); i += LARGE_THREADS) bits[i] = 0u;
            if (tid == 0) n_twice = 0;
            __syncthreads();
            for (int64_t end = i1; end > i0; end -= LARGE_THREADS) {
                const int64_t i = end - LARGE_THREADS + tid;
                const uint32_t x = i >= i0 ? (uint32_t)win.rec[i] - base : 0u, bit = 1u << (x & 31);
                const bool in = i >= i0 && x < span && (uint32_t)win.rec[i] != 0xffffffffu;
                const bool met = in && (bits[x >> 5] & bit) != 0;
                __syncthreads();
                bool lost = false;
                if (in && !met && (atomicOr(bits + (x >> 5), bit) & bit) != 0) {
                    lost = true;
                    const int j = atomicAdd(&n_twice, 1);
                    twice[j] = x;
                    last[j] = 0u;
                }
                if (met) win.rec[i] = ~0ull;
                if (!__syncthreads_or(lost)) continue;
                const int n = n_twice;
                for (int j = 0; j < n; ++j)
                    if (in && !met && twice[j] == x) atomicMax(last + j, (uint32_t)tid + 1u);
                __syncthreads();
                for (int j = 0; j < n; ++j)
                    if (in && !met && twice[j] == x && last[j] != (uint32_t)tid + 1u) win.rec[i] = ~0ull;
                if (tid == 0) n_twice = 0;
                __syncthreads();
            }
            __syncthreads();                                          // the row's bits are free again
        }
    }
}

// The windows that a CTA of count_large_kernel has left for later: those with columns further apart than a bitmap reaches
// are numbered, and entries in no order are rid of duplicates where they are many (a hub's row written in order keeps
// one warp busy for all of it).  A loop of its own: in one with the usual windows it cost those a quarter of their speed.
// Builds, ms, with a bitmap round for every 524,288 columns / like this / with one radix sort of all entries:
//   2.4 M rows of 52 entries, 2.4 M columns           33.2 / 10.4 / 14.9
//   1 M rows of 40 entries, 100 M columns            357   /  3.8 /  4.9
//   100 k rows of 300 entries, 600 k columns           2.0 /  2.2 /  3.6
//   1 M rows of 12 and 500 of 100 k, 100 M columns    41.6 /  8.3 /  7.2   (3.9 where the rows ascend)
//   16 rows of 1 M and nothing else, 100 M columns   111   / 15.0 /  3.9   (one CTA per hub: 132 of 148 SMs are idle)
//   the same, 400 k columns, in no order              12.3 /  4.6 /  3.9
__device__ __forceinline__ void count_left_windows(const EntrySource &src, const BuildScratch &s) {
    const int n_large = s.large[0];
    for (int q = blockIdx.x; q < n_large; q += gridDim.x) {
        const int32_t id = s.large[1 + q];
        if (!(id & (LARGE_WIDE | LARGE_MIXED))) continue;
        const int64_t w = id & ~(LARGE_WIDE | LARGE_MIXED);
        const LargeWindow win(src, s, w);
        uint32_t total = (uint32_t)s.columns[q];
        bool plain = false;
        if (id & LARGE_WIDE) {
            uint32_t lo, hi;
            column_span(win, &lo, &hi);
            __syncthreads();
            float *val = s.val + (win.rec - s.rec);
            total = number_wide_window(win, lo, hi, reinterpret_cast<int32_t *>(val));
            const bool ordered = copy_values(win, w, src.val + (win.col - src.col), val);
            plain = src.row_ptr && (src.unique || ordered);
        }
        if (src.row_ptr && !plain && win.m > SORT_ENTRIES) {
            drop_superseded(win, w, total);
            plain = true;
        }
        __syncthreads();                                              // every thread has read the window's id and columns
        if (threadIdx.x == 0) {
            s.tiles[w + 1] = ((int64_t)total + TILE_COLS - 1) / TILE_COLS;
            s.columns[q] = (int32_t)total;
            s.large[1 + q] = (int32_t)w | (plain ? LARGE_PLAIN : 0);
        }
    }
}

// Large windows, one CTA each: every distinct column gets its slot, usually by one bitmap of all columns.  Bound by the
// latency of its loads and barriers; two CTAs per SM (32 registers a thread) hide some of each other's.
__global__ void __launch_bounds__(LARGE_THREADS, 2)
count_large_kernel(const EntrySource src, const BuildScratch s) {
    bool left = false;
    const int n_large = s.large[0];
    for (int q = blockIdx.x; q < n_large; q += gridDim.x) {
        const int64_t w = s.large[1 + q];
        const LargeWindow win(src, s, w);
        uint32_t lo, hi, total = 0;
        int flags = LARGE_WIDE;
        const bool any = column_span(win, &lo, &hi);
        if (any && hi - lo >= BITMAP_COLS) {
            __syncthreads();
        } else {
            if (any) total = number_by_bitmap<true>(win, win.m, [](int64_t k) { return k; }, lo, hi, 0u);
            const bool ordered = copy_values(win, w, src.val + (win.col - src.col), s.val + (win.rec - s.rec));
            flags = !src.row_ptr ? 0 : src.unique || ordered ? LARGE_PLAIN : win.m > SORT_ENTRIES ? LARGE_MIXED : 0;
        }
        left |= (flags & (LARGE_WIDE | LARGE_MIXED)) != 0;
        if (threadIdx.x == 0) {
            s.tiles[w + 1] = ((int64_t)total + TILE_COLS - 1) / TILE_COLS;
            s.columns[q] = (int32_t)total;
            s.large[1 + q] = (int32_t)w | flags;
        }
    }
    if (left) {
        __syncthreads();
        count_left_windows(src, s);
    }
}

template <typename T> __device__ __forceinline__ T from_float(float v);
template <> __device__ __forceinline__ float from_float<float>(float v) { return v; }
template <> __device__ __forceinline__ __half from_float<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// 16 bytes of an output array at piece index i; an array that does not start on a 16-byte boundary takes
// them element by element
template <typename T>
__device__ __forceinline__ void store_piece(T *p, int64_t i, uint4 v, bool vec) {
    if (vec) {
        reinterpret_cast<uint4 *>(p)[i] = v;
    } else {
        const T *e = reinterpret_cast<const T *>(&v);
#pragma unroll
        for (int j = 0; j < 16 / (int)sizeof(T); ++j) p[i * (16 / (int)sizeof(T)) + j] = e[j];
    }
}

// One warp per window: the records are in slot order, so a group of consecutive tiles is a run of them; it is
// assembled in shared memory and written once, in 16-byte pieces.  Bound by the latency of the records' loads (a warp
// waits 13 cycles an instruction for them; DRAM is 19 % busy, 32 us for the 90 MB of a 169 k-node graph's fp16 tiles).
// All threads then empty the tiles behind the last one (arrays sized by a bound).
template <typename T>
__global__ void __launch_bounds__(FILL_WARPS * 32)
fill_windows_kernel(int64_t W, int64_t num_rows, int64_t num_tiles, const BuildScratch s, const int64_t *__restrict__ window_offset,
                    int32_t *__restrict__ out_cols, T *__restrict__ out_vals, bool vec) {
    constexpr int GROUP = FILL_BYTES / (TILE_ELEMS * (int)sizeof(T));           // tiles per group
    constexpr int TILE_V = TILE_ELEMS * (int)sizeof(T) / 16;                    // 16-byte pieces of a tile
    __shared__ __align__(16) T tile_buf[FILL_WARPS][GROUP * TILE_ELEMS];
    __shared__ __align__(16) int32_t col_buf[FILL_WARPS][GROUP * TILE_COLS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t w = (int64_t)blockIdx.x * FILL_WARPS + warp;
    if (w < W) {
        const int64_t t0 = window_offset[w], nt = window_offset[w + 1] - t0;
        const int64_t r1 = (w + 1) * TILE_ROWS < num_rows ? (w + 1) * TILE_ROWS : num_rows;
        int p = s.row_start[w * TILE_ROWS];
        const int end = s.row_start[r1];
        if (end - p <= SMALL_ENTRIES) {
            T *tb = tile_buf[warp];
            int32_t *cb = col_buf[warp];
            for (int g = 0; g < nt; g += GROUP) {
#pragma unroll
                for (int i = 0; i < FILL_BYTES / 512; ++i) reinterpret_cast<uint4 *>(tb)[i * 32 + lane] = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int i = 0; i < GROUP * TILE_COLS / 32; ++i) cb[i * 32 + lane] = -1;
                __syncwarp();
                while (p < end) {
                    const bool live = lane_has_entry(p, lane, end);
                    const uint64_t r = live ? __ldg(s.rec + p + lane) : ~0ull;
                    const float v = live ? __ldg(s.val + p + lane) : 0.f;
                    const uint32_t info = (uint32_t)r;
                    const int slot = (int)(info >> 5) - g * TILE_COLS;
                    const bool in = live && slot < GROUP * TILE_COLS;
                    if (in && !(info & 1u)) {
                        tb[(slot >> 3) * TILE_ELEMS + ((info >> 1) & (TILE_ROWS - 1)) * TILE_COLS + (slot & 7)] = from_float<T>(v);
                        cb[slot] = (int32_t)(r >> 32);
                    }
                    const int n = __popc(__ballot_sync(0xffffffffu, in));
                    p += n;
                    if (n < 32) break;
                }
                __syncwarp();
                const int live = nt - g < GROUP ? (int)(nt - g) : GROUP;
                T *ov = out_vals + (t0 + g) * TILE_ELEMS;
                int32_t *oc = out_cols + (t0 + g) * TILE_COLS;
                for (int i = lane; i < live * TILE_V; i += 32) store_piece(ov, i, reinterpret_cast<uint4 *>(tb)[i], vec);
                for (int i = lane; i < live * 2; i += 32) store_piece(oc, i, reinterpret_cast<uint4 *>(cb)[i], vec);
                __syncwarp();
            }
        }
    }
    const int64_t T0 = window_offset[W], stride = (int64_t)gridDim.x * blockDim.x, me = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t i = T0 * TILE_V + me; i < num_tiles * TILE_V; i += stride) store_piece(out_vals, i, make_uint4(0u, 0u, 0u, 0u), vec);
    for (int64_t i = T0 * 2 + me; i < num_tiles * 2; i += stride)
        store_piece(out_cols, i, make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu), vec);
}

// Large windows, one CTA each: column ids and empty tiles, then the entries are scattered.  Where no two have one place
// they go in any order, all threads side by side; otherwise a warp per row keeps their order, so that the last of
// several entries of one column is the one that stays.  Bound by the CTA with the most entries and the latency of its loads:
// a hub's row has thousands and its 15 neighbours few, so a warp per row leaves 15 of 16 warps waiting.  A 169 k-node
// graph and its transpose, fp32: 648 us built with a warp per row throughout, 548 us with distinct entries side by side.
template <typename T>
__global__ void __launch_bounds__(FILL_LARGE_THREADS)
fill_large_kernel(int64_t num_rows, const BuildScratch s, const int64_t *__restrict__ window_offset,
                  int32_t *__restrict__ out_cols, T *__restrict__ out_vals, bool vec) {
    constexpr int TILE_V = TILE_ELEMS * (int)sizeof(T) / 16;
    __shared__ int32_t start[TILE_ROWS + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_large = s.large[0];
    for (int q = blockIdx.x; q < n_large; q += gridDim.x) {
        const int32_t id = s.large[1 + q];
        const bool plain = id & LARGE_PLAIN;
        const int64_t w = id & ~LARGE_PLAIN, t0 = window_offset[w], nt = window_offset[w + 1] - t0;
        __syncthreads();                                  // the previous window's use of `start` is over
        if (tid <= TILE_ROWS) {
            const int64_t row = w * TILE_ROWS + tid;
            start[tid] = s.row_start[row < num_rows ? row : num_rows];
        }
        __syncthreads();
        const int first = start[0], end = start[TILE_ROWS], columns = s.columns[q];
        T *ov = out_vals + t0 * TILE_ELEMS;
        int32_t *oc = out_cols + t0 * TILE_COLS;
        for (int64_t i = tid; i < nt * TILE_V; i += FILL_LARGE_THREADS) store_piece(ov, i, make_uint4(0u, 0u, 0u, 0u), vec);
        for (int64_t i = tid; i < nt * TILE_COLS; i += FILL_LARGE_THREADS) oc[i] = i < columns ? __ldg(s.ucol + first + i) : -1;
        __syncthreads();
        if (plain) {
            for (int64_t b = first; b < end; b += FILL_LARGE_THREADS * 4) {
                uint32_t slot[4];
                float v[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int64_t i = b + j * FILL_LARGE_THREADS + tid;
                    slot[j] = i < end ? (uint32_t)__ldg(s.rec + i) : 0xffffffffu;
                    v[j] = i < end ? __ldg(s.val + i) : 0.f;
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int64_t i = b + j * FILL_LARGE_THREADS + tid;
                    int row = 0;
#pragma unroll
                    for (int step = TILE_ROWS / 2; step > 0; step >>= 1) row += i >= start[row + step] ? step : 0;
                    if (slot[j] != 0xffffffffu) ov[(int64_t)(slot[j] >> 3) * TILE_ELEMS + row * TILE_COLS + (slot[j] & 7)] = from_float<T>(v[j]);
                }
            }
            continue;
        }
        const int64_t last = start[warp + 1];
        for (int64_t b = start[warp]; b < last; b += 32 * FILL_AHEAD) {
            uint64_t r[FILL_AHEAD];
            float v[FILL_AHEAD];
#pragma unroll
            for (int j = 0; j < FILL_AHEAD; ++j) {
                const int64_t i = b + j * 32 + lane;
                r[j] = i < last ? __ldg(s.rec + i) : ~0ull;
                v[j] = i < last ? __ldg(s.val + i) : 0.f;
            }
#pragma unroll
            for (int j = 0; j < FILL_AHEAD; ++j) {
                const uint32_t slot = (uint32_t)r[j];                     // all ones in an empty entry, no slot is
                const unsigned same = __match_any_sync(0xffffffffu, slot);
                if (r[j] != ~0ull && lane == 31 - __clz(same))
                    ov[(int64_t)(slot >> 3) * TILE_ELEMS + warp * TILE_COLS + (slot & 7)] = from_float<T>(v[j]);
                __syncwarp();
            }
        }
    }
}

static inline unsigned blocks_for(int64_t n, int threads) {
    int64_t b = ceil_div(n > 0 ? n : 1, threads);
    return (unsigned)(b > 0x7fffffff ? 0x7fffffff : b);
}

// ------------------------------- BCSR -> transposed CSR -------------------------------------
template <typename T> __device__ __forceinline__ float to_float(T v);
template <> __device__ __forceinline__ float to_float<float>(float v) { return v; }
template <> __device__ __forceinline__ float to_float<__half>(__half v) { return __half2float(v); }
template <> __device__ __forceinline__ float to_float<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// four consecutive values of a tile as floats: one load per lane covers a tile
__device__ __forceinline__ float4 load4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }
__device__ __forceinline__ float4 load4(const __half *p) {
    const uint2 u = __ldg(reinterpret_cast<const uint2 *>(p));
    const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ float4 load4(const __nv_bfloat16 *p) {
    const uint2 u = __ldg(reinterpret_cast<const uint2 *>(p));
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&u.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}

constexpr int TRANSPOSE_WARPS = 8;
constexpr int TRANSPOSE_AHEAD = 4;     // tiles a warp has in flight

// MODE 0 counts the non-zero entries per column, MODE 1 scatters them.  The tiles are shared out evenly over the
// warps, whatever window they belong to: a hub's window has a hundred times the tiles of the others, and
// with a CTA per window its chain of load, atomic and store was the kernel's time (169 k nodes, 315 k tiles of
// fp32: counting 283 -> 51 us, scattering 383 -> 90 us; the tiles' bytes alone take 26 us).  vec: cols and vals start on
// 16-byte boundaries.
template <typename T, int MODE>
__global__ void __launch_bounds__(TRANSPOSE_WARPS * 32)
transpose_entries_kernel(int64_t W, const int64_t *__restrict__ window_offset, const int32_t *__restrict__ cols,
                         const T *__restrict__ vals, int64_t num_cols, int64_t *__restrict__ counts_or_cursor,
                         int32_t *__restrict__ out_col, float *__restrict__ out_val, bool vec) {
    const int lane = threadIdx.x & 31;
    const int64_t n_warps = (int64_t)gridDim.x * TRANSPOSE_WARPS, me = (int64_t)blockIdx.x * TRANSPOSE_WARPS + (threadIdx.x >> 5);
    // a range of the windows of a larger matrix, over that matrix's arrays, does not start at tile 0
    const int64_t T_first = __ldg(window_offset), T0 = __ldg(window_offset + W);
    int64_t share = (T0 - T_first + n_warps - 1) / n_warps;
    share = (share + TRANSPOSE_AHEAD - 1) / TRANSPOSE_AHEAD * TRANSPOSE_AHEAD;
    const int64_t t0 = T_first + me * share, t1 = t0 + share < T0 ? t0 + share : T0;
    if (t0 >= t1) return;
    int64_t w = warp_count_ends_le(window_offset, W, t0, lane);      // the window that holds tile t0
    int64_t end = __ldg(window_offset + w + 1);
    for (int64_t t = t0; t < t1; t += TRANSPOSE_AHEAD) {
        float4 v[TRANSPOSE_AHEAD];
        int4 c[TRANSPOSE_AHEAD];
#pragma unroll
        for (int q = 0; q < TRANSPOSE_AHEAD; ++q) {
            v[q] = make_float4(0.f, 0.f, 0.f, 0.f);
            c[q] = make_int4(-1, -1, -1, -1);
            if (t + q < t1) {
                const T *pv = vals + (t + q) * TILE_ELEMS + lane * 4;
                const int32_t *pc = cols + (t + q) * TILE_COLS + (lane & 1) * 4;
                if (vec) {
                    v[q] = load4(pv);
                    c[q] = __ldg(reinterpret_cast<const int4 *>(pc));
                } else {
                    v[q] = make_float4(to_float<T>(pv[0]), to_float<T>(pv[1]), to_float<T>(pv[2]), to_float<T>(pv[3]));
                    c[q] = make_int4(pc[0], pc[1], pc[2], pc[3]);
                }
            }
        }
        // all atomics of the tiles in flight first, then the stores that wait for their results
        int32_t row[TRANSPOSE_AHEAD];
        int64_t pos[TRANSPOSE_AHEAD][4];
#pragma unroll
        for (int q = 0; q < TRANSPOSE_AHEAD; ++q) {
            while (t + q < t1 && t + q >= end) end = __ldg(window_offset + ++w + 1);    // windows without tiles are passed over
            row[q] = (int32_t)(w * TILE_ROWS + (lane >> 1));
            const float vq[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
            const int32_t cq[4] = {c[q].x, c[q].y, c[q].z, c[q].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                pos[q][j] = -1;
                if (vq[j] == 0.0f || cq[j] < 0 || cq[j] >= num_cols) continue;
                if (MODE == 0) atomicAdd(reinterpret_cast<unsigned long long *>(counts_or_cursor + cq[j] + 1), 1ull);
                else pos[q][j] = (int64_t)atomicAdd(reinterpret_cast<unsigned long long *>(counts_or_cursor + cq[j]), 1ull);
            }
        }
        if (MODE == 1) {
#pragma unroll
            for (int q = 0; q < TRANSPOSE_AHEAD; ++q) {
                const float vq[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (pos[q][j] < 0) continue;
                    out_col[pos[q][j]] = row[q];
                    out_val[pos[q][j]] = vq[j];
                }
            }
        }
    }
}

// BCSR -> CSR (not transposed): one warp per window, lane r < 16 walks row r of every tile in
// order.  Column ids are ascending inside a window, so every CSR row comes out ascending.
// MODE 0 counts the non-zero entries of each row, MODE 1 writes them.
template <typename T, int MODE>
__global__ void bcsr_rows_kernel(int64_t W, int64_t num_rows, const int64_t *__restrict__ window_offset,
                                 const int32_t *__restrict__ cols, const T *__restrict__ vals,
                                 int64_t *__restrict__ row_ptr, int32_t *__restrict__ out_col,
                                 float *__restrict__ out_val) {
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int r = threadIdx.x & 31;
    if (w >= W || r >= TILE_ROWS) return;
    const int64_t row = w * TILE_ROWS + r;
    if (row >= num_rows) return;
    int64_t o = (MODE == 1) ? row_ptr[row] : 0;
    for (int64_t t = window_offset[w]; t < window_offset[w + 1]; ++t) {
#pragma unroll
        for (int c = 0; c < TILE_COLS; ++c) {
            const int32_t col = cols[t * TILE_COLS + c];
            const float v = to_float<T>(vals[t * TILE_ELEMS + r * TILE_COLS + c]);
            if (col < 0 || v == 0.0f) continue;
            if (MODE == 1) { out_col[o] = col; out_val[o] = v; }
            ++o;
        }
    }
    if (MODE == 0) row_ptr[row + 1] = o;
}

int block_build_fill(int64_t n_dst, int fanout, const int64_t *window_offset, int64_t num_tiles, int32_t *out_cols, void *out_vals,
                     int val_dtype, void *scratch, size_t scratch_bytes, cudaStream_t st);

}  // namespace grws

using namespace grws;

static int sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
        sms = 148;
    return sms;
}

// Inclusive prefix sum by one CTA.  Up to SCAN_ONE numbers (131,000 rows) one launch of this takes the time of the
// first of the device-wide scan's two.
constexpr int SCAN_THREADS = 1024, SCAN_ONE = 8 * SCAN_THREADS;
__global__ void __launch_bounds__(SCAN_THREADS)
scan_one_kernel(const int64_t *__restrict__ in, int64_t *__restrict__ out, int n) {
    __shared__ int64_t part[SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int each = (n + SCAN_THREADS - 1) / SCAN_THREADS, i0 = threadIdx.x * each;
    int64_t v[SCAN_ONE / SCAN_THREADS], sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ONE / SCAN_THREADS; ++k) {
        v[k] = k < each && i0 + k < n ? in[i0 + k] : 0;
        sum += v[k];
    }
    int64_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int64_t o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == 31) part[warp] = incl;
    __syncthreads();
    int64_t at = incl - sum;
    for (int k = 0; k < warp; ++k) at += part[k];
#pragma unroll
    for (int k = 0; k < SCAN_ONE / SCAN_THREADS; ++k) {
        at += v[k];
        if (k < each && i0 + k < n) out[i0 + k] = at;
    }
}

// Count phase of both front ends.  may_be_large: some window may have more than SMALL_ENTRIES entries.
static int count_entries(const BuildScratch &s, const EntrySource &src, int64_t W, bool may_be_large, int64_t *window_offset,
                         cudaStream_t st) {
    if (W == 0) {
        GRWS_CUDA_TRY(cudaMemsetAsync(window_offset, 0, 8, st));
        return GRWS_OK;
    }
    GRWS_CUDA_TRY(cudaMemsetAsync(s.large, 0, 4, st));
    count_windows_kernel<<<blocks_for(W, COUNT_WARPS), COUNT_WARPS * 32, 0, st>>>(src, W, s);
    if (may_be_large) {
        GRWS_CUDA_TRY(cudaFuncSetAttribute(count_large_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LARGE_SMEM));
        const int64_t grid = 2 * sm_count();
        count_large_kernel<<<(unsigned)(W < grid ? W : grid), LARGE_THREADS, LARGE_SMEM, st>>>(src, s);
    }
    if (W + 1 <= SCAN_ONE) {
        scan_one_kernel<<<1, SCAN_THREADS, 0, st>>>(s.tiles, window_offset, (int)(W + 1));
    } else {
        size_t tmp = s.cub_bytes;
        GRWS_CUDA_TRY(cub::DeviceScan::InclusiveSum(s.cub_tmp, tmp, s.tiles, window_offset, (int)(W + 1), st));
    }
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

template <typename T>
static int fill_entries(const BuildScratch &s, int64_t num_rows, int64_t num_tiles, bool may_be_large, const int64_t *window_offset,
                        int32_t *out_cols, void *out_vals, cudaStream_t st) {
    const int64_t W = ceil_div(num_rows, TILE_ROWS);
    const bool vec = aligned16(out_cols) && aligned16(out_vals);
    fill_windows_kernel<T><<<blocks_for(W, FILL_WARPS), FILL_WARPS * 32, 0, st>>>(W, num_rows, num_tiles, s, window_offset, out_cols,
                                                                                  static_cast<T *>(out_vals), vec);
    if (may_be_large) {
        const int64_t grid = 4 * sm_count();
        fill_large_kernel<T><<<(unsigned)(W < grid ? W : grid), FILL_LARGE_THREADS, 0, st>>>(num_rows, s, window_offset, out_cols,
                                                                                            static_cast<T *>(out_vals), vec);
    }
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

// eight CTAs per SM, fewer where there are not even that many windows' tiles to share out
static unsigned transpose_blocks(int64_t W) {
    const int64_t most = 8 * sm_count(), few = ceil_div(W, 2);
    return (unsigned)(few < most ? (few > 0 ? few : 1) : most);
}

template <typename T>
static int transpose_count(const int64_t *wo, const int32_t *cols, const void *vals, int64_t W, int64_t num_cols,
                           int64_t *row_ptr_t, void *scratch, cudaStream_t st) {
    int64_t *counts = static_cast<int64_t *>(scratch);
    void *cub_tmp = static_cast<char *>(scratch) + align_up((size_t)(num_cols + 1) * 8);
    size_t tmp = 0;
    cub::DeviceScan::InclusiveSum(nullptr, tmp, (const int64_t *)nullptr, (int64_t *)nullptr, (int)(num_cols + 1));
    GRWS_CUDA_TRY(cudaMemsetAsync(counts, 0, (size_t)(num_cols + 1) * 8, st));
    if (W > 0)
        transpose_entries_kernel<T, 0><<<transpose_blocks(W), TRANSPOSE_WARPS * 32, 0, st>>>(W, wo, cols, (const T *)vals, num_cols, counts,
                                                                                             nullptr, nullptr, aligned16(cols) && aligned16(vals));
    GRWS_CUDA_TRY(cub::DeviceScan::InclusiveSum(cub_tmp, tmp, counts, row_ptr_t, (int)(num_cols + 1), st));
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}


// a window of fixed-stride lists has 16 * fanout slots
static bool lists_may_be_large(int fanout) { return (int64_t)fanout * TILE_ROWS > SMALL_ENTRIES; }

static int fill_any(int64_t num_rows, int64_t nnz, bool may_be_large, const int64_t *window_offset, int64_t num_tiles, int32_t *out_cols,
                    void *out_vals, int val_dtype, void *scratch, size_t scratch_bytes, cudaStream_t st) {
    GRWS_REQUIRE(num_rows >= 0 && nnz >= 0 && num_tiles >= 0, "negative size");
    BuildScratch s = carve(scratch, nnz, num_rows);
    if (scratch_bytes < s.total) return fail(GRWS_ERR_SCRATCH, "csr_to_bcsr scratch too small");
    if (num_tiles == 0) return GRWS_OK;
    GRWS_REQUIRE(window_offset && out_cols && out_vals && scratch, "null pointer");
    switch (val_dtype) {
        case GRWS_F32: return fill_entries<float>(s, num_rows, num_tiles, may_be_large, window_offset, out_cols, out_vals, st);
        case GRWS_F16: return fill_entries<__half>(s, num_rows, num_tiles, may_be_large, window_offset, out_cols, out_vals, st);
        case GRWS_BF16: return fill_entries<__nv_bfloat16>(s, num_rows, num_tiles, may_be_large, window_offset, out_cols, out_vals, st);
    }
    return fail(GRWS_ERR_UNSUPPORTED, "bad value dtype %d", val_dtype);
}

// the fill phase of a block built from lists (sampler.cu): the host knows how large its windows can be
int grws::block_build_fill(int64_t n_dst, int fanout, const int64_t *window_offset, int64_t num_tiles, int32_t *out_cols, void *out_vals,
                           int val_dtype, void *scratch, size_t scratch_bytes, cudaStream_t st) {
    return fill_any(n_dst, n_dst * fanout, lists_may_be_large(fanout), window_offset, num_tiles, out_cols, out_vals, val_dtype, scratch,
                    scratch_bytes, st);
}

extern "C" {

__attribute__((visibility("default")))
size_t grws_csr_to_bcsr_scratch_bytes(int64_t num_rows, int64_t nnz) {
    if (num_rows < 0 || nnz < 0) return 0;
    return carve(nullptr, nnz, num_rows).total;
}

static int csr_count(int64_t num_rows, const int64_t *row_ptr, const int32_t *col_idx, const float *values, int64_t nnz, bool unique,
                     int64_t *window_offset, void *scratch, size_t scratch_bytes, void *stream) {
    GRWS_REQUIRE(num_rows >= 0 && nnz >= 0, "negative size");
    GRWS_REQUIRE(nnz < 0x7fffffffLL, "csr_to_bcsr handles fewer than 2^31 entries");
    const int64_t W = ceil_div(num_rows, TILE_ROWS);
    GRWS_REQUIRE(W < (1LL << 28), "too many windows");
    GRWS_REQUIRE(row_ptr && window_offset && scratch, "null pointer");
    GRWS_REQUIRE(nnz == 0 || (col_idx && values), "null CSR arrays");
    BuildScratch s = carve(scratch, nnz, num_rows);
    if (scratch_bytes < s.total) return fail(GRWS_ERR_SCRATCH, "csr_to_bcsr scratch too small: %zu < %zu", scratch_bytes, s.total);
    if (nnz == 0) {                            // row_ptr is not read then: it may be as short as the caller's entries
        GRWS_CUDA_TRY(cudaMemsetAsync(window_offset, 0, (size_t)(W + 1) * 8, static_cast<cudaStream_t>(stream)));
        return GRWS_OK;
    }
    const EntrySource src = {row_ptr, col_idx, values, num_rows, 0, unique};
    return count_entries(s, src, W, nnz > SMALL_ENTRIES, window_offset, static_cast<cudaStream_t>(stream));
}

__attribute__((visibility("default")))
int grws_csr_to_bcsr_count(int64_t num_rows, const int64_t *row_ptr, const int32_t *col_idx,
                           const float *values, int64_t nnz, int64_t *window_offset, void *scratch,
                           size_t scratch_bytes, void *stream) {
    return csr_count(num_rows, row_ptr, col_idx, values, nnz, false, window_offset, scratch, scratch_bytes, stream);
}

__attribute__((visibility("default")))
int grws_csr_to_bcsr_count_unique(int64_t num_rows, const int64_t *row_ptr, const int32_t *col_idx,
                                  const float *values, int64_t nnz, int64_t *window_offset, void *scratch,
                                  size_t scratch_bytes, void *stream) {
    return csr_count(num_rows, row_ptr, col_idx, values, nnz, true, window_offset, scratch, scratch_bytes, stream);
}

// The kernels only visit the entries that row_ptr covers, so a bound on their number needs nothing of its own.
__attribute__((visibility("default")))
int grws_csr_to_bcsr_count_bounded(int64_t num_rows, const int64_t *row_ptr, const int32_t *col_idx,
                                   const float *values, int64_t nnz_bound, int64_t num_cols_bound,
                                   int64_t *window_offset, void *scratch, size_t scratch_bytes, void *stream) {
    GRWS_REQUIRE(num_cols_bound >= 0, "negative size");
    return grws_csr_to_bcsr_count(num_rows, row_ptr, col_idx, values, nnz_bound, window_offset, scratch, scratch_bytes, stream);
}

__attribute__((visibility("default")))
int grws_block_build_count(const int32_t *local, const float *w, int64_t n_dst, int fanout, int64_t num_cols_bound,
                           int64_t *window_offset, void *scratch, size_t scratch_bytes, void *stream) {
    GRWS_REQUIRE(n_dst >= 0 && fanout > 0 && num_cols_bound >= 0, "bad size");
    const int64_t n_entries = n_dst * fanout;
    GRWS_REQUIRE(n_entries < 0x7fffffffLL, "hop too large");
    const int64_t W = ceil_div(n_dst, TILE_ROWS);
    GRWS_REQUIRE(window_offset && scratch && (n_entries == 0 || (local && w)), "null pointer");
    BuildScratch s = carve(scratch, n_entries, n_dst);
    if (scratch_bytes < s.total) return fail(GRWS_ERR_SCRATCH, "block build scratch too small: %zu < %zu", scratch_bytes, s.total);
    const EntrySource src = {nullptr, local, w, n_dst, fanout, false};
    return count_entries(s, src, W, lists_may_be_large(fanout), window_offset, static_cast<cudaStream_t>(stream));
}

__attribute__((visibility("default")))
int grws_csr_to_bcsr_fill(int64_t num_rows, int64_t nnz, const int64_t *window_offset, int64_t num_tiles,
                          int32_t *out_cols, void *out_vals, int val_dtype, void *scratch,
                          size_t scratch_bytes, void *stream) {
    return fill_any(num_rows, nnz, nnz > SMALL_ENTRIES, window_offset, num_tiles, out_cols, out_vals, val_dtype, scratch, scratch_bytes,
                    static_cast<cudaStream_t>(stream));
}

// counts[0] = 0, counts[c + 1] = non-zero entries in column c; then inclusive scan -> row_ptr of A^T
__attribute__((visibility("default")))
size_t grws_bcsr_transpose_scratch_bytes(int64_t num_cols) {
    size_t s3 = 0;
    cub::DeviceScan::InclusiveSum(nullptr, s3, (const int64_t *)nullptr, (int64_t *)nullptr, (int)(num_cols + 1));
    return align_up((size_t)(num_cols + 1) * 8) + align_up(s3);
}

__attribute__((visibility("default")))
int grws_bcsr_transpose_count(const int64_t *window_offset, const int32_t *cols, const void *vals, int val_dtype,
                              int64_t num_windows, int64_t num_cols, int64_t *row_ptr_t, void *scratch,
                              size_t scratch_bytes, void *stream) {
    GRWS_REQUIRE(num_windows >= 0 && num_cols >= 0, "negative size");
    GRWS_REQUIRE(num_windows < 0x7fffffffLL && num_cols < 0x7fffffffLL, "size beyond 2^31");
    GRWS_REQUIRE(window_offset && row_ptr_t && scratch, "null pointer");
    if (scratch_bytes < grws_bcsr_transpose_scratch_bytes(num_cols)) return fail(GRWS_ERR_SCRATCH, "transpose scratch too small");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (val_dtype) {
        case GRWS_F32: return transpose_count<float>(window_offset, cols, vals, num_windows, num_cols, row_ptr_t, scratch, st);
        case GRWS_F16: return transpose_count<__half>(window_offset, cols, vals, num_windows, num_cols, row_ptr_t, scratch, st);
        case GRWS_BF16: return transpose_count<__nv_bfloat16>(window_offset, cols, vals, num_windows, num_cols, row_ptr_t, scratch, st);
    }
    return fail(GRWS_ERR_UNSUPPORTED, "bad value dtype %d", val_dtype);
}

// scatters the entries; `scratch` must still hold what the count call left (it is reused as cursors)
__attribute__((visibility("default")))
int grws_bcsr_transpose_fill(const int64_t *window_offset, const int32_t *cols, const void *vals, int val_dtype,
                             int64_t num_windows, int64_t num_cols, const int64_t *row_ptr_t, int32_t *out_col,
                             float *out_val, void *scratch, size_t scratch_bytes, void *stream) {
    GRWS_REQUIRE(num_windows >= 0 && num_cols >= 0, "negative size");
    GRWS_REQUIRE(window_offset && row_ptr_t && scratch, "null pointer");
    if (scratch_bytes < grws_bcsr_transpose_scratch_bytes(num_cols)) return fail(GRWS_ERR_SCRATCH, "transpose scratch too small");
    if (num_windows == 0) return GRWS_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int64_t *cursor = static_cast<int64_t *>(scratch);
    GRWS_CUDA_TRY(cudaMemcpyAsync(cursor, row_ptr_t, (size_t)(num_cols + 1) * 8, cudaMemcpyDeviceToDevice, st));
    const unsigned nb = transpose_blocks(num_windows);
    const bool vec = aligned16(cols) && aligned16(vals);
    switch (val_dtype) {
        case GRWS_F32:
            transpose_entries_kernel<float, 1><<<nb, TRANSPOSE_WARPS * 32, 0, st>>>(num_windows, window_offset, cols, (const float *)vals, num_cols, cursor, out_col, out_val, vec);
            break;
        case GRWS_F16:
            transpose_entries_kernel<__half, 1><<<nb, TRANSPOSE_WARPS * 32, 0, st>>>(num_windows, window_offset, cols, (const __half *)vals, num_cols, cursor, out_col, out_val, vec);
            break;
        case GRWS_BF16:
            transpose_entries_kernel<__nv_bfloat16, 1><<<nb, TRANSPOSE_WARPS * 32, 0, st>>>(num_windows, window_offset, cols, (const __nv_bfloat16 *)vals, num_cols, cursor, out_col, out_val, vec);
            break;
        default:
            return fail(GRWS_ERR_UNSUPPORTED, "bad value dtype %d", val_dtype);
    }
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

// BCSR -> CSR of the same matrix, two phases like the other builders.
__attribute__((visibility("default")))
size_t grws_bcsr_to_csr_scratch_bytes(int64_t num_rows) {
    size_t s3 = 0;
    cub::DeviceScan::InclusiveSum(nullptr, s3, (const int64_t *)nullptr, (int64_t *)nullptr, (int)(num_rows + 1));
    return align_up(s3);
}

__attribute__((visibility("default")))
int grws_bcsr_to_csr_count(const int64_t *window_offset, const int32_t *cols, const void *vals, int val_dtype,
                           int64_t num_windows, int64_t num_rows, int64_t *row_ptr, void *scratch,
                           size_t scratch_bytes, void *stream) {
    GRWS_REQUIRE(num_windows >= 0 && num_rows >= 0 && num_rows <= num_windows * TILE_ROWS, "bad size");
    GRWS_REQUIRE(num_rows < 0x7fffffffLL, "size beyond 2^31");
    GRWS_REQUIRE(window_offset && row_ptr && scratch, "null pointer");
    if (scratch_bytes < grws_bcsr_to_csr_scratch_bytes(num_rows)) return fail(GRWS_ERR_SCRATCH, "bcsr_to_csr scratch too small");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    GRWS_CUDA_TRY(cudaMemsetAsync(row_ptr, 0, (size_t)(num_rows + 1) * 8, st));
    if (num_windows > 0) {
        const unsigned nb = blocks_for(num_windows * 32, 256);
        if (val_dtype == GRWS_F32) bcsr_rows_kernel<float, 0><<<nb, 256, 0, st>>>(num_windows, num_rows, window_offset, cols, (const float *)vals, row_ptr, nullptr, nullptr);
        else if (val_dtype == GRWS_F16) bcsr_rows_kernel<__half, 0><<<nb, 256, 0, st>>>(num_windows, num_rows, window_offset, cols, (const __half *)vals, row_ptr, nullptr, nullptr);
        else if (val_dtype == GRWS_BF16) bcsr_rows_kernel<__nv_bfloat16, 0><<<nb, 256, 0, st>>>(num_windows, num_rows, window_offset, cols, (const __nv_bfloat16 *)vals, row_ptr, nullptr, nullptr);
        else return fail(GRWS_ERR_UNSUPPORTED, "bad value dtype %d", val_dtype);
    }
    size_t tmp = scratch_bytes;
    GRWS_CUDA_TRY(cub::DeviceScan::InclusiveSum(scratch, tmp, row_ptr, row_ptr, (int)(num_rows + 1), st));
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

__attribute__((visibility("default")))
int grws_bcsr_to_csr_fill(const int64_t *window_offset, const int32_t *cols, const void *vals, int val_dtype,
                          int64_t num_windows, int64_t num_rows, const int64_t *row_ptr, int32_t *out_col,
                          float *out_val, void *stream) {
    GRWS_REQUIRE(num_windows >= 0 && num_rows >= 0, "bad size");
    if (num_windows == 0) return GRWS_OK;
    GRWS_REQUIRE(window_offset && row_ptr, "null pointer");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    int64_t *rp = const_cast<int64_t *>(row_ptr);
    const unsigned nb = blocks_for(num_windows * 32, 256);
    if (val_dtype == GRWS_F32) bcsr_rows_kernel<float, 1><<<nb, 256, 0, st>>>(num_windows, num_rows, window_offset, cols, (const float *)vals, rp, out_col, out_val);
    else if (val_dtype == GRWS_F16) bcsr_rows_kernel<__half, 1><<<nb, 256, 0, st>>>(num_windows, num_rows, window_offset, cols, (const __half *)vals, rp, out_col, out_val);
    else if (val_dtype == GRWS_BF16) bcsr_rows_kernel<__nv_bfloat16, 1><<<nb, 256, 0, st>>>(num_windows, num_rows, window_offset, cols, (const __nv_bfloat16 *)vals, rp, out_col, out_val);
    else return fail(GRWS_ERR_UNSUPPORTED, "bad value dtype %d", val_dtype);
    GRWS_CUDA_TRY(cudaGetLastError());
    return GRWS_OK;
}

}  // extern "C"
