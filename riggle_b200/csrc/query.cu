// The sweep: query_database's counting path (src/tasks/query/mod.rs:182-307) and
// query_sweep_windowed (src/sweep/query.rs:84-117) as one device pipeline.
//
// Per batch (all on the context stream, no host synchronisation, graph-capturable once the
// workspace is reserved):
//   1. k_expand_keys: each query interval becomes key (segment << 32 | start), value end, and a
//      second key (segment << 32 | end); segment = shard * rows + Q_SID.  Invalid intervals
//      (start >= end, sid >= rows) raise an error bit.
//   2. sort both key sets (the reference sorts by (sid, start), mod.rs:202; ends are sorted too,
//      which the rank formulation below needs): block by block when every input block is one
//      segment (tiles sorted in shared memory, then merge passes; ordered blocks copied through),
//      else a device-wide radix sort.
//   3. one scan over the sorted queries (k_q_reduce, k_q_apply): segment numbers, prefix sums of the
//      starts (PS) and the largest end of each segment's earlier queries; the same for the ends (PE).
//   4. K1 partition: for every (layer slot K, query i) the candidate range of the reference's scan,
//      [pp(start - max_K), pp(end)) with pp = partition point of the layer's starts
//      (src/sweep/query.rs:98-105), k_lohi; the non-empty ones laid out and merged into disjoint
//      ranges per (K, segment), k_emit; the ranges' unions, methods and places, k_range_*.
//   5. K2 sweep (k_sweep): a persistent kernel pulls fixed-size chunks of that concatenated range
//      space from a device counter.  Each thread takes one DB interval d and computes, against the
//      segment's sorted query starts S and ends E,
//          count(d) = #{q : q.start < d.end} - #{q : q.end <= d.start}
//          bp(d)    = Cov(d.end) - Cov(d.start),  Cov(x) = x (S<x - E<=x) - PS(S<x) + PE(E<=x)
//      which equal the number of overlapping query intervals and their summed intersection length
//      whenever every DB interval of layer K is non-empty and shorter than max_K — the size-class
//      invariant the reference's add establishes (src/io/meta.rs:33-58) and index validation checks.
//      Under that invariant the look-back bound q.start - max_K <= d.start of the reference's scan
//      never excludes an overlapping pair, so the counts are the reference's, bit for bit.  All
//      ranks lie inside the window of queries that produced d's range, so the searches are short.
//      Counts and base pairs are tallied per (row, source) in shared memory when a chunk belongs to
//      one row, else with global atomics.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <type_traits>

#include "block_sort.cuh"
#include "internal.h"
#include "pdl.cuh"

namespace rgl {

// A range swept by ranks.
struct RangeDesc {
    uint32_t db_lo;      // its first DB interval within the layer
    uint32_t layer_idx;  // index into the layer table
    uint32_t qrow;       // query row (Q_SID)
    uint32_t seg;        // query segment number
};

// One query's candidate run for the pair sweep: DB elements from `base` (of the index arrays) on; in the
// several-row sweep the query's row lies above the element (2^36 elements of 12 bytes are 824 GB).
struct __align__(16) PairSeg {
    uint64_t base;
    uint32_t qs, qe;
};
constexpr int kRunRowShift = 36;
constexpr uint32_t kMaxPackedRows = 1u << (64 - kRunRowShift);
template <int MULTI>
__device__ __forceinline__ uint64_t run_base(uint64_t b) {
    return MULTI ? b & ((1ull << kRunRowShift) - 1) : b;
}

// Rank table of one query segment: bin b (width 2^shift bp) holds, at tab2[off + b], the numbers
// of the segment's sorted starts and ends below b << shift, as absolute positions in the sorted
// arrays.  A rank is then one table read plus a search over at most one bin, and the two entries
// of a bin serve the start rank and the end rank of any x in it.
struct SegTab {
    uint32_t beg, end;  // the segment's positions in the sorted arrays
    uint32_t shift, nbins;
    uint32_t off;       // first entry of the segment's tables (nbins + 1 entries each)
    uint32_t pad;
};

enum : uint32_t { ERR_BAD_INTERVAL = 1u, ERR_BAD_ROW = 2u };

// ---- small device helpers ----------------------------------------------------------------------
__device__ __forceinline__ uint32_t lb_u32(const uint32_t* __restrict__ a, uint32_t lo, uint32_t hi, uint32_t x) {
    // first index in [lo, hi) with a[i] >= x
    while (lo < hi) {
        uint32_t m = lo + ((hi - lo) >> 1);
        if (__ldg(a + m) < x) lo = m + 1; else hi = m;
    }
    return lo;
}
__device__ __forceinline__ uint32_t ub_u32(const uint32_t* __restrict__ a, uint32_t lo, uint32_t hi, uint32_t x) {
    // first index in [lo, hi) with a[i] > x
    while (lo < hi) {
        uint32_t m = lo + ((hi - lo) >> 1);
        if (__ldg(a + m) <= x) lo = m + 1; else hi = m;
    }
    return lo;
}
// Partition points of (start < x) over a layer sorted by start, for x0 -> r0 and x1 -> r1: the
// bucket table gives the elements whose starts share x's bucket, searched by bisection.  The two
// run in lockstep (both bucket reads issued together, then one probe of each bisection per round),
// so their chains of dependent random reads overlap instead of following one another.
__device__ __forceinline__ void pp_layer2(const uint2* __restrict__ pos, const uint32_t* __restrict__ btab,
                                          const LayerQuery& L, uint32_t x0, uint32_t x1, uint32_t& r0, uint32_t& r1) {
    const uint32_t last = L.nb - 1;
    const uint32_t b0 = x0 >> L.bshift, b1 = x1 >> L.bshift;
    uint32_t lo0 = L.n, hi0 = L.n, lo1 = L.n, hi1 = L.n;
    if (b0 < last) {
        lo0 = __ldg(btab + b0);
        hi0 = __ldg(btab + b0 + 1);
    }
    if (b1 < last) {
        lo1 = __ldg(btab + b1);
        hi1 = __ldg(btab + b1 + 1);
    }
    while (lo0 < hi0 || lo1 < hi1) {
        const bool a0 = lo0 < hi0, a1 = lo1 < hi1;
        const uint32_t m0 = lo0 + ((hi0 - lo0) >> 1), m1 = lo1 + ((hi1 - lo1) >> 1);
        const uint32_t v0 = a0 ? __ldg(&pos[m0].x) : 0u, v1 = a1 ? __ldg(&pos[m1].x) : 0u;
        if (a0) {
            if (v0 < x0) lo0 = m0 + 1; else hi0 = m0;
        }
        if (a1) {
            if (v1 < x1) lo1 = m1 + 1; else hi1 = m1;
        }
    }
    r0 = lo0;
    r1 = lo1;
}

// ---- 1. keys ------------------------------------------------------------------------------------
// Zeroes the words of up to five regions (the run's counters, outputs, sort flags and per-segment sums):
// one launch instead of a memset each (7 of them, 4 us of stream time each).
struct ClearList {
    static constexpr int kMax = 5;
    uint32_t* p[kMax];
    uint64_t words[kMax];
    int count;
};
__global__ void __launch_bounds__(256) k_clear(ClearList list) {
    for (int r = 0; r < list.count; r++)
        for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < list.words[r];
             i += (uint64_t)gridDim.x * blockDim.x)
            list.p[r][i] = 0u;
}

template <bool PDL>
__global__ void k_expand_keys(uint32_t n, const rgl_interval* __restrict__ iv, const uint64_t* __restrict__ blk_off,
                              const uint32_t* __restrict__ blk_shard, const uint32_t* __restrict__ blk_row,
                              int row_from_block, uint32_t nblk, uint32_t rows, uint32_t row_base, uint32_t rb,
                              uint64_t* __restrict__ key, uint32_t* __restrict__ val, uint64_t* __restrict__ ekey,
                              uint32_t* __restrict__ err, uint32_t* __restrict__ unsorted,
                              const uint64_t* __restrict__ sdst, const uint32_t* __restrict__ sidx, int wide) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    // block b with blk_off[b] <= i < blk_off[b+1]: one search per warp, for its first element, then a short
    // walk (32 consecutive elements span few blocks)
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, w0 = i & ~31u;
    const uint32_t b0 = w0 < n ? find_block(blk_off, nblk, w0) : 0u;
    if (i >= n) return;
    uint32_t lo = b0;
    while (lo + 1 < nblk && blk_off[lo + 1] <= i) lo++;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(iv) + 3ull * i;
    // the block-local sort: block b's keys at sdst[b] + their place in the block (segment-order
    // layout) or in place; order flags of the block's rank k in that layout: starts (ends) out of
    // order -> unsorted[k] (unsorted[nblk + k]) = 1
    const uint64_t o = sdst ? sdst[lo] + (i - blk_off[lo]) : (uint64_t)i;
    // the row is the interval's sid, or with row_from_block its block's row (sid ignored)
    const uint32_t row = row_from_block ? blk_row[lo] : w[2];
    if (unsorted && i > blk_off[lo]) {
        const uint32_t k = sidx ? sidx[lo] : lo;
        const uint32_t before = wide ? w[-1] : row;  // (wide: rows come from the intervals)
        if (row < before || (row == before && w[0] < w[-3])) unsorted[k] = 1u;
        if (row < before || (row == before && w[1] < w[-2])) unsorted[nblk + k] = 1u;
    }
    uint32_t s = w[0], e = w[1], q = row - row_base;  // rows below row_base wrap to >= rows
    uint32_t bad = 0;
    if (s >= e) bad |= ERR_BAD_INTERVAL;
    if (q >= rows || (blk_row && row != blk_row[lo])) {
        bad |= ERR_BAD_ROW;
        // The run is refused at its end, but goes through to there: its key stays in its block's segment, so that
        // a block sorted on its own is one segment and there are no more segments than (shard, row) pairs.
        q = blk_row ? blk_row[lo] - row_base : 0u;
        if (wide && unsorted) {  // its key goes by row 0 now: out of order
            const uint32_t k = sidx ? sidx[lo] : lo;
            unsorted[k] = unsorted[nblk + k] = 1u;
        }
    }
    if (bad) atomicOr(err, bad);
    // segment = (shard, region, row): with regions (rb > 0) a row's intervals on a shard are cut
    // into 2^rb-bp regions of their starts, so that the rows' work on one region lies together
    const uint64_t nreg = rb ? (1ull << (32 - rb)) : 1ull, reg = rb ? (s >> rb) : 0u;
    uint64_t seg = ((uint64_t)blk_shard[lo] * nreg + reg) * rows + q;
    key[o] = (seg << 32) | s;
    val[o] = e;
    ekey[o] = (seg << 32) | e;
}

// ---- tile prefixes ------------------------------------------------------------------------------------
// The layout below is made of passes over tiles of a sequence, each with a summary per tile whose prefix
// the next pass needs.  Every block of that pass sums the summaries before its tile itself, with no launch
// in between, up to kMaxLook tiles (at most 8 reads a thread); beyond, groups of kGroup tiles are summed
// (k_group_sums) and every tile's prefix written in its place (k_group_scan), since a block that sums
// hundreds of them first starts its own reads 3 us late.
constexpr uint32_t kTileThreads = 256, kMaxLook = 2048, kGroup = 256;

// Summary of a span of the sorted queries: segment starts in it, the largest end since the last of them
// (since the span's start without one), and the sum of the starts.
struct QSum {
    uint32_t heads, emax;
    uint64_t sum;
    __device__ __forceinline__ static QSum zero() { return QSum{0u, 0u, 0ull}; }
    __device__ __forceinline__ static QSum add(const QSum& a, const QSum& b) {
        return QSum{a.heads + b.heads, b.heads ? b.emax : max(a.emax, b.emax), a.sum + b.sum};
    }
};
// Summary of a span of (slot, query) entries: live runs, ranges that start in it, candidates.
struct LSum {
    uint32_t live, ranges;
    uint64_t cand;
    __device__ __forceinline__ static LSum zero() { return LSum{0u, 0u, 0ull}; }
    __device__ __forceinline__ static LSum add(const LSum& a, const LSum& b) {
        return LSum{a.live + b.live, a.ranges + b.ranges, a.cand + b.cand};
    }
};
// Summary of a span of ranges: positions swept by ranks, candidates swept by pairs, ranges of the former.
struct RSum {
    uint64_t rank, pair;
    uint64_t nrank;
    __device__ __forceinline__ static RSum zero() { return RSum{0ull, 0ull, 0ull}; }
    __device__ __forceinline__ static RSum add(const RSum& a, const RSum& b) {
        return RSum{a.rank + b.rank, a.pair + b.pair, a.nrank + b.nrank};
    }
};
struct ESum {
    uint64_t sum;
    __device__ __forceinline__ static ESum zero() { return ESum{0ull}; }
    __device__ __forceinline__ static ESum add(const ESum& a, const ESum& b) { return ESum{a.sum + b.sum}; }
};
template <class T>
struct TileOp {
    __device__ __forceinline__ T operator()(const T& a, const T& b) const { return T::add(a, b); }
};

// v of the lane o above, of any struct of 32-bit words.
template <class T>
__device__ __forceinline__ T shfl_down_words(const T& v, int o) {
    T r;
    const uint32_t* a = reinterpret_cast<const uint32_t*>(&v);
    uint32_t* b = reinterpret_cast<uint32_t*>(&r);
#pragma unroll
    for (int w = 0; w < (int)(sizeof(T) / 4); w++) b[w] = __shfl_down_sync(0xffffffffu, a[w], o);
    return r;
}
// Sum of the lanes' values in order, lane 0's.
template <class T>
__device__ __forceinline__ T warp_total(T v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) v = T::add(v, shfl_down_words(v, o));  // lane 0: lanes 0 .. 2 o - 1, in order
    return v;
}
// Sum of s[0, m), for every thread of the block (kTileThreads threads, contiguous stretches, in order).
template <class T>
__device__ __forceinline__ T block_total(const T* __restrict__ s, uint32_t m) {
    __shared__ T part[kTileThreads / 32];
    const uint32_t per = (m + kTileThreads - 1) / kTileThreads;
    T v = T::zero();
    const uint32_t a = min(threadIdx.x * per, m), b = min(a + per, m);
    for (uint32_t k = a; k < b; k++) v = T::add(v, s[k]);
    v = warp_total(v);
    if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = v;
    __syncthreads();
    v = part[0];
#pragma unroll
    for (uint32_t w = 1; w < kTileThreads / 32; w++) v = T::add(v, part[w]);
    __syncthreads();  // part may be reused by the next call
    return v;
}
// Sum of sums[0, tile); with `scanned`, sums[tile] is that sum already.
template <class T>
__device__ __forceinline__ T tile_prefix(const T* __restrict__ sums, int scanned, uint32_t tile) {
    return scanned ? sums[tile] : block_total(sums, tile);
}
// groups[g] = sum of the g-th group's tiles, of nt tiles (or of those of *count elements).
template <class T>
__global__ void __launch_bounds__(kTileThreads) k_group_sums(const T* __restrict__ sums, uint32_t nt,
                                                             const uint32_t* __restrict__ count, uint32_t tile,
                                                             T* __restrict__ groups) {
    if (count) nt = (uint32_t)(((uint64_t)*count + tile - 1) / tile);
    const uint32_t a = blockIdx.x * kGroup;
    const T v = block_total(sums + a, a < nt ? min(kGroup, nt - a) : 0u);
    if (threadIdx.x == 0) groups[blockIdx.x] = v;
}

template <class T>
__device__ __forceinline__ T shfl_up_words(const T& v, int o) {
    T r;
    const uint32_t* a = reinterpret_cast<const uint32_t*>(&v);
    uint32_t* b = reinterpret_cast<uint32_t*>(&r);
#pragma unroll
    for (int w = 0; w < (int)(sizeof(T) / 4); w++) b[w] = __shfl_up_sync(0xffffffffu, a[w], o);
    return r;
}
template <class T>
__device__ __forceinline__ T shfl_words(const T& v, int src) {
    T r;
    const uint32_t* a = reinterpret_cast<const uint32_t*>(&v);
    uint32_t* b = reinterpret_cast<uint32_t*>(&r);
#pragma unroll
    for (int w = 0; w < (int)(sizeof(T) / 4); w++) b[w] = __shfl_sync(0xffffffffu, a[w], src);
    return r;
}
template <class T>
__device__ __forceinline__ T warp_scan(T v, uint32_t lane) {  // inclusive, in order
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T w = shfl_up_words(v, o);
        if (lane >= (uint32_t)o) v = T::add(w, v);
    }
    return v;
}
// Exclusive prefix of v over the block's threads, in order (kTileThreads threads).
template <class T>
__device__ __forceinline__ T block_exclusive(T v) {
    __shared__ T part[kTileThreads / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const T inc = warp_scan(v, lane);
    if (lane == 31) part[warp] = inc;
    __syncthreads();
    T ex = shfl_up_words(inc, 1);
    if (lane == 0) ex = T::zero();
    T before = T::zero();
    for (uint32_t w = 0; w < warp; w++) before = T::add(before, part[w]);
    __syncthreads();  // part may be reused by the next call
    return T::add(before, ex);
}
// Every tile of group blockIdx.x: sums[tile] becomes the sum of all tiles before it; *total: the whole.
template <class T>
__global__ void __launch_bounds__(kTileThreads) k_group_scan(T* __restrict__ sums, uint32_t nt,
                                                             const uint32_t* __restrict__ count, uint32_t tile,
                                                             const T* __restrict__ groups, T* __restrict__ total) {
    static_assert(kGroup == kTileThreads, "one tile a thread");
    if (count) nt = (uint32_t)(((uint64_t)*count + tile - 1) / tile);
    const uint32_t k = blockIdx.x * kGroup + threadIdx.x;
    const T before = block_total(groups, blockIdx.x);
    const T own = k < nt ? sums[k] : T::zero(), ex = block_exclusive(own);
    if (k < nt) sums[k] = T::add(before, ex);
    if (total && k + 1 == nt) *total = T::add(T::add(before, ex), own);
}

// ---- 3. the sorted queries ------------------------------------------------------------------------------
// One pass of summaries and one that writes, over the sorted start keys: starts, shards, rows and segment
// numbers, the first query of every segment, the exclusive prefix sums of the starts (n + 1), and for every
// query the largest end of the segment's earlier queries (0 for its first), by which the ranges are cut
// below.  Bound by the 12 bytes read twice and the 28 written per query; four consecutive queries a thread,
// in 16-byte reads and writes.
constexpr uint32_t kQItems = 4, kQTile = kTileThreads * kQItems;

// v[0, 4) from / to a[base, base + 4) (base a multiple of 4), below n.
template <class T>
__device__ __forceinline__ void load4(const T* __restrict__ a, uint32_t base, uint32_t n, T (&v)[4]) {
    if (base + 4 <= n) {
        const uint4* p = reinterpret_cast<const uint4*>(a + base);
        if constexpr (sizeof(T) == 4) {
            const uint4 w = p[0];
            v[0] = w.x, v[1] = w.y, v[2] = w.z, v[3] = w.w;
        } else {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const uint4 w = p[h];
                v[2 * h] = ((uint64_t)w.y << 32) | w.x;
                v[2 * h + 1] = ((uint64_t)w.w << 32) | w.z;
            }
        }
        return;
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; j++) v[j] = base + j < n ? a[base + j] : (T)0;
}
template <class T>
__device__ __forceinline__ void store4(T* __restrict__ a, uint32_t base, uint32_t n, const T (&v)[4]) {
    if (base + 4 <= n) {
        uint4* p = reinterpret_cast<uint4*>(a + base);
        if constexpr (sizeof(T) == 4) p[0] = make_uint4(v[0], v[1], v[2], v[3]);
        else {
#pragma unroll
            for (int h = 0; h < 2; h++)
                p[h] = make_uint4((uint32_t)v[2 * h], (uint32_t)(v[2 * h] >> 32), (uint32_t)v[2 * h + 1],
                                  (uint32_t)(v[2 * h + 1] >> 32));
        }
        return;
    }
#pragma unroll
    for (uint32_t j = 0; j < 4; j++)
        if (base + j < n) a[base + j] = v[j];
}

// The summaries of a thread's queries and their sum.
__device__ __forceinline__ QSum q_items(uint32_t n, uint32_t base, const uint64_t* __restrict__ key,
                                        const uint32_t* __restrict__ end, uint64_t (&k)[4], uint32_t (&e)[4],
                                        uint32_t* heads) {
    load4(key, base, n, k);
    load4(end, base, n, e);
    uint32_t prev = (base && base < n) ? (uint32_t)(key[base - 1] >> 32) : 0u;
    QSum s = QSum::zero();
    *heads = 0;
#pragma unroll
    for (uint32_t j = 0; j < kQItems; j++) {
        const uint32_t i = base + j, sg = (uint32_t)(k[j] >> 32);
        const uint32_t h = i < n && (i == 0 || sg != prev) ? 1u : 0u;
        *heads |= h << j;
        s = QSum::add(s, QSum{h, e[j], (uint32_t)k[j]});
        prev = sg;
    }
    return s;
}

template <bool PDL>
__global__ void __launch_bounds__(kTileThreads) k_q_reduce(uint32_t n, const uint64_t* __restrict__ key,
                                                           const uint32_t* __restrict__ end,
                                                           QSum* __restrict__ sums) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    __shared__ QSum part[kTileThreads / 32];
    uint64_t k[4];
    uint32_t e[4], heads;
    const QSum s = warp_total(q_items(n, blockIdx.x * kQTile + threadIdx.x * kQItems, key, end, k, e, &heads));
    if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        QSum t = part[0];
#pragma unroll
        for (uint32_t w = 1; w < kTileThreads / 32; w++) t = QSum::add(t, part[w]);
        sums[blockIdx.x] = t;
    }
}

template <bool PDL>
__global__ void __launch_bounds__(kTileThreads) k_q_apply(
    uint32_t n, uint32_t rows, uint32_t seg_per_shard, const uint64_t* __restrict__ key,
    const uint32_t* __restrict__ end, const QSum* __restrict__ sums, int scanned, uint32_t* __restrict__ starts,
    uint32_t* __restrict__ shard, uint32_t* __restrict__ row, uint32_t* __restrict__ segnum,
    uint32_t* __restrict__ seg_begin, uint64_t* __restrict__ ps, uint32_t* __restrict__ emax) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    const uint32_t base = blockIdx.x * kQTile + threadIdx.x * kQItems;
    uint64_t k[4];
    uint32_t e[4], heads;
    const QSum own = q_items(n, base, key, end, k, e, &heads);
    const QSum before = tile_prefix(sums, scanned, blockIdx.x);
    QSum run = QSum::add(before, block_exclusive(own));
    uint32_t st[4], sh[4], rw[4], num[4], em[4];
    uint64_t pre[4];
#pragma unroll
    for (uint32_t j = 0; j < kQItems; j++) {
        const uint32_t i = base + j, sg = (uint32_t)(k[j] >> 32), h = heads >> j & 1u;
        st[j] = (uint32_t)k[j];
        sh[j] = sg / seg_per_shard;
        rw[j] = rows > 1 ? sg % rows : 0u;
        pre[j] = run.sum;
        em[j] = h ? 0u : run.emax;
        if (h) seg_begin[run.heads] = i;
        run = QSum::add(run, QSum{h, e[j], st[j]});
        num[j] = run.heads;
        if (i + 1 == n) {
            ps[n] = run.sum;
            seg_begin[run.heads] = n;
        }
    }
    store4(starts, base, n, st);
    store4(shard, base, n, sh);
    if (rows > 1) store4(row, base, n, rw);
    store4(segnum, base, n, num);
    store4(emax, base, n, em);
    store4(ps, base, n, pre);
}

// The sorted end keys into ends and their exclusive prefix sums (n + 1).
template <bool PDL>
__global__ void __launch_bounds__(kTileThreads) k_e_reduce(uint32_t n, const uint64_t* __restrict__ ekey,
                                                           ESum* __restrict__ sums) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    __shared__ ESum part[kTileThreads / 32];
    uint64_t k[4];
    load4(ekey, blockIdx.x * kQTile + threadIdx.x * kQItems, n, k);
    const ESum s = warp_total(ESum{(k[0] & 0xFFFFFFFFull) + (uint32_t)k[1] + (uint32_t)k[2] + (uint32_t)k[3]});
    if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        ESum t = part[0];
#pragma unroll
        for (uint32_t w = 1; w < kTileThreads / 32; w++) t = ESum::add(t, part[w]);
        sums[blockIdx.x] = t;
    }
}
template <bool PDL>
__global__ void __launch_bounds__(kTileThreads) k_e_apply(uint32_t n, const uint64_t* __restrict__ ekey,
                                                          const ESum* __restrict__ sums, int scanned,
                                                          uint32_t* __restrict__ ends_s, uint64_t* __restrict__ pe) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    const uint32_t base = blockIdx.x * kQTile + threadIdx.x * kQItems;
    uint64_t k[4], pre[4], s = 0;
    uint32_t e[4];
    load4(ekey, base, n, k);
#pragma unroll
    for (uint32_t j = 0; j < kQItems; j++) {
        e[j] = (uint32_t)k[j];
        s += e[j];
    }
    const ESum before = tile_prefix(sums, scanned, blockIdx.x);
    uint64_t run = before.sum + block_exclusive(ESum{s}).sum;
#pragma unroll
    for (uint32_t j = 0; j < kQItems; j++) {
        pre[j] = run;
        run += e[j];
        if (base + j + 1 == n) pe[n] = run;
    }
    store4(ends_s, base, n, e);
    store4(pe, base, n, pre);
}

// Bin width per segment: about four bins per query, at least 64 bp, but no more than one bin per 8
// DB intervals the segment's rank-difference ranges sweep (need[]): each swept interval reads the
// table a few times, so a table much larger than its sweep costs more to build than its finer bins
// save (large query files against a small database).  A coarser bin only lengthens the search
// inside it.  A segment of m queries has at most 8 m + 2 entries (nbins + 1), so segment k's table
// starts at 8 beg + 2 k: the places need no scan.
__global__ void k_seg_tabsize(uint32_t n, const uint32_t* __restrict__ segnum, const uint32_t* __restrict__ seg_begin,
                              const unsigned long long* __restrict__ need, const uint32_t* __restrict__ ends_s,
                              SegTab* __restrict__ tabs) {
    const uint32_t sgi = blockIdx.x * blockDim.x + threadIdx.x;
    if (sgi >= segnum[n - 1]) return;
    const uint32_t beg = seg_begin[sgi], end = seg_begin[sgi + 1];
    if (!need[sgi]) {  // no range of this segment is swept by rank differences
        tabs[sgi] = SegTab{beg, end, 6, 0, 0, 0};
        return;
    }
    const uint64_t extent = (uint64_t)ends_s[end - 1] + 1;  // covers every start and end of the segment
    const uint64_t bins = max(1ull, min(4ull * (end - beg), need[sgi] / 8));
    const uint64_t want = extent / bins;
    uint32_t shift = want > 1 ? 63u - __clzll(want) : 0u;
    if (shift < 6) shift = 6;
    if (shift > 31) shift = 31;
    const uint32_t nbins = (uint32_t)(extent >> shift) + 1;  // <= 8 (end - beg) + 1
    tabs[sgi] = SegTab{beg, end, shift, nbins, 8 * beg + 2 * sgi, 0};
}

// The blocks (in the sort's layout) whose segment has no range swept by ranks: their ends stay unsorted.
__global__ void k_skip_ends(uint32_t nblk, const uint64_t* __restrict__ off, const uint32_t* __restrict__ segnum,
                            const unsigned long long* __restrict__ need, uint32_t* __restrict__ unsorted) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nblk || off[b] == off[b + 1]) return;
    if (!need[segnum[off[b]] - 1]) unsorted[b] = kSkipBlock;
}

// Rank tables from the sorted arrays: entry b of a segment holds the position of its first element of bin
// >= b, so element j fills the entries from its predecessor's bin (exclusive) through its own with j, and
// the last one the rest with the segment's end.  A lane fills up to kTabShort entries itself, longer
// stretches are filled by the whole warp.  Bound: 8 bytes written per entry.  Counting the elements per
// bin with atomics, two scans over the tables and interleaving them took twelve launches, and 1.6 ms for
// 3.1e7 intervals whose few-bin tables made thousands of atomics meet on one counter; this takes 0.26 ms.
constexpr uint32_t kTabShort = 8;
template <bool PDL>
__global__ void __launch_bounds__(256) k_tab_fill(uint32_t n, const uint32_t* __restrict__ segnum,
                                                  const SegTab* __restrict__ tabs,
                                                  const uint32_t* __restrict__ starts,
                                                  const uint32_t* __restrict__ ends_s, uint2* __restrict__ tab2) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    SegTab t{0, 0, 0, 0, 0, 0};
    if (j < n) t = tabs[segnum[j] - 1];
    if (!__ballot_sync(0xffffffffu, t.nbins != 0)) return;
#pragma unroll
    for (int side = 0; side < 2; side++) {
        const uint32_t* a = side ? ends_s : starts;
        uint32_t* col = reinterpret_cast<uint32_t*>(tab2) + side;  // entry b at col[2 (off + b)]
        uint32_t from = 0, to = 0;  // entries [from, to) of the table, as absolute entries
        uint32_t rest = 0;          // and [to, rest) by the segment's last element
        if (t.nbins) {  // (a refused interval may start past every end: its bin is held to the table)
            to = t.off + min(a[j] >> t.shift, t.nbins - 1) + 1;
            from = j == t.beg ? t.off : t.off + min(a[j - 1] >> t.shift, t.nbins - 1) + 1;
            rest = j + 1 == t.end ? t.off + t.nbins + 1 : to;
        }
        if (to - from <= kTabShort)
            for (uint32_t b = from; b < to; b++) col[2ull * b] = j;
        if (rest - to <= kTabShort)
            for (uint32_t b = to; b < rest; b++) col[2ull * b] = t.end;
#pragma unroll
        for (int part = 0; part < 2; part++) {
            const uint32_t f = part ? to : from, e = part ? rest : to, v = part ? t.end : j;
            for (uint32_t m = __ballot_sync(0xffffffffu, e - f > kTabShort); m; m &= m - 1) {
                const int src = __ffs(m) - 1;
                const uint32_t f1 = __shfl_sync(0xffffffffu, f, src), e1 = __shfl_sync(0xffffffffu, e, src);
                const uint32_t v1 = __shfl_sync(0xffffffffu, v, src);
                for (uint32_t b = f1 + lane; b < e1; b += 32) col[2ull * b] = v1;
            }
        }
    }
}

// Adds a 32-bit value to a 64-bit shared-memory counter with 32-bit atomics: the low word, and the
// high word only when the low word wraps (one pair's overlap always fits 32 bits).
__device__ __forceinline__ void add_u64_lo(unsigned long long* c, uint32_t v) {
    uint32_t* w = reinterpret_cast<uint32_t*>(c);  // little-endian: w[0] low, w[1] high
    const uint32_t old = atomicAdd(w, v);
    if (old + v < old) atomicAdd(w + 1, 1u);
}

// The same for a 64-bit value: low word, then the high word plus the carry when either is non-zero.
__device__ __forceinline__ void add_u64(unsigned long long* c, unsigned long long v) {
    uint32_t* w = reinterpret_cast<uint32_t*>(c);
    const uint32_t lo = (uint32_t)v, old = atomicAdd(w, lo);
    const uint32_t hi = (uint32_t)(v >> 32) + (old + lo < old ? 1u : 0u);
    if (hi) atomicAdd(w + 1, hi);
}

// ---- 4. K1 partition -----------------------------------------------------------------------------
// Entry (slot K, query i) in the order K, i.  Its candidate run is the reference's scan [lo, hi): lo =
// partition point of start - max_K, hi = that of end; an entry whose run is empty takes part in nothing.
// The live entries (the others) merge into disjoint ranges per (K, segment): a live entry starts a range
// when no earlier run of its row reaches past its lo.  The earlier runs' largest hi is the partition point
// of the segment's largest end so far, E (k_q_apply), the same for every slot, so that no scan over the
// entries is needed: with back = start - max_K,
//     back >= E            starts a range (the partition point is monotone);
//     E >= end             does not (its run ends at or before the partition point of E);
//     back < E < end       starts one when no start lies in [back, E), i.e. when the run's first element
//                          (live: it exists) starts at or after E.
// Pass 1 (k_lohi) searches, and stores the live entries of each tile (kTileThreads queries of one slot)
// side by side: first element, length, place in the tile and whether they start a range; it sums live
// entries, ranges and candidates per tile.  Pass 2 (k_emit) writes the live runs and the ranges at their
// places.  Pass 1 is bound by its random reads (bucket table and starts) and, where those hit L2, by issue:
// one query a thread, so that the blocks running at once lie close together and the rows of a chromosome
// find its starts in L2 (eight queries a thread: 0.75 -> 2.0 ms for 48 files against 2e8 intervals).
// Before, the flags, a compaction, a segmented running maximum and three scans over the entries took eleven
// launches (3.9 of the 11 ms of 3.1e7 intervals against 3.2e6); with every entry's [lo, hi) stored and read
// again, dead or live, k_emit took 2.1 of 8.9 ms there, now 1.2 of 6.4.
constexpr uint32_t kStartsRange = 1u << 15;  // in an entry's `place`, beside its number in the tile
__device__ __forceinline__ bool large_counts(uint32_t cnt) { return __any_sync(0xffffffffu, cnt >> 27); }

// Sum of the lanes' counts, in 32 bits unless a count is so large that it may not fit.
__device__ __forceinline__ uint64_t warp_count(uint32_t cnt) {
    if (!large_counts(cnt)) return __reduce_add_sync(0xffffffffu, cnt);
    uint64_t c = cnt;
#pragma unroll
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    return c;
}

template <bool PDL>
__global__ void __launch_bounds__(kTileThreads) k_lohi(
    uint32_t n, uint32_t nslots, const uint32_t* __restrict__ starts, const uint32_t* __restrict__ qend,
    const uint32_t* __restrict__ emax, const uint32_t* __restrict__ shard, const LayerQuery* __restrict__ layers,
    const uint2* __restrict__ pos, const uint32_t* __restrict__ btab, uint32_t* __restrict__ lo_out,
    uint32_t* __restrict__ cnt_out, uint16_t* __restrict__ place,
    LSum* __restrict__ sums) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    __shared__ LSum part[kTileThreads / 32];
    const uint32_t K = blockIdx.y, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t tile = K * gridDim.x + blockIdx.x;
    const uint32_t i = blockIdx.x * kTileThreads + threadIdx.x;
    uint32_t lo = 0, hi = 0;
    bool start = false;
    if (i < n) {
        const LayerQuery L = layers[(uint64_t)shard[i] * nslots + K];
        if (L.nb) {
            const uint2* p = pos + L.off;
            const uint32_t st = starts[i], en = qend[i], E = emax[i];
            const uint32_t back = st >= L.max_size ? st - L.max_size : 0u;  // saturating_sub, src/sweep/query.rs:98
            pp_layer2(p, btab + L.boff, L, back, en, lo, hi);
            if (hi < lo) hi = lo;
            if (hi > lo) start = back >= E || (E < en && __ldg(&p[lo].x) >= E);
        }
    }
    const uint32_t fl = __ballot_sync(0xffffffffu, start), live = __ballot_sync(0xffffffffu, hi > lo);
    const uint64_t cand = warp_count(hi - lo);
    if (lane == 0) part[warp] = LSum{(uint32_t)__popc(live), (uint32_t)__popc(fl), cand};
    __syncthreads();
    uint32_t before = 0;
    for (uint32_t w = 0; w < warp; w++) before += part[w].live;
    if (hi > lo) {
        const uint64_t at = (uint64_t)tile * kTileThreads + before + __popc(live & ((1u << lane) - 1u));
        lo_out[at] = lo;
        cnt_out[at] = hi - lo;
        place[at] = (uint16_t)(threadIdx.x | (start ? kStartsRange : 0u));
    }
    if (threadIdx.x == 0) {
        LSum s = part[0];
#pragma unroll
        for (uint32_t w = 1; w < kTileThreads / 32; w++) s = LSum::add(s, part[w]);
        sums[tile] = s;
    }
}

// The partition point of (start < x) alone (see pp_layer2).
__device__ __forceinline__ uint32_t pp_layer(const uint2* __restrict__ pos, const uint32_t* __restrict__ btab,
                                             const LayerQuery& L, uint32_t x) {
    const uint32_t b = x >> L.bshift;
    if (b >= L.nb - 1) return L.n;
    uint32_t lo = __ldg(btab + b), hi = __ldg(btab + b + 1);
    while (lo < hi) {
        const uint32_t m = lo + ((hi - lo) >> 1);
        if (__ldg(&pos[m].x) < x) lo = m + 1; else hi = m;
    }
    return lo;
}

// Inclusive sums of the lanes' counts, in 32 bits as warp_count.
__device__ __forceinline__ uint64_t warp_inclusive(uint32_t cnt, uint32_t lane) {
    if (!large_counts(cnt)) {
        uint32_t inc = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t w = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (uint32_t)o) inc += w;
        }
        return inc;
    }
    uint64_t inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t w = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += w;
    }
    return inc;
}

// What the runs carry beside their queries: nothing; the row, in the top bits of `base` (the several-row
// pair sweep, which reads it with the rest) or on its own (several rows tallied straight into the outputs);
// or shard and row (shard * rows + row; the pair list).
enum : int { RUN_PLAIN = 0, RUN_ROW = 1, RUN_SHARD_ROW = 2, RUN_PACKED = 3 };

// Live run c: its query's candidates psegs[c], the candidates before it pc[c], its range cr[c] and uhi[c],
// the end of the union of its range's runs through it (written only where the run may be its range's last).
// Range r: rt[r] = (its first live run, that run's entry K n + i).  The last tile's warp writes the totals: L, R
// and pc[L].  A warp takes one of k_lohi's tiles (per_slot of them a slot), 32 live entries at a time.
template <bool PDL>
__global__ void __launch_bounds__(kTileThreads) k_emit(
    uint32_t n, uint32_t nslots, uint32_t rows, uint32_t per_slot, uint32_t tiles, int tag,
    const uint32_t* __restrict__ starts, const uint32_t* __restrict__ qend, const uint32_t* __restrict__ emax,
    const uint32_t* __restrict__ shard, const uint32_t* __restrict__ row, const LayerQuery* __restrict__ layers,
    const uint2* __restrict__ pos, const uint32_t* __restrict__ btab, const uint32_t* __restrict__ lo_in,
    const uint32_t* __restrict__ cnt_in, const uint16_t* __restrict__ place,
    const LSum* __restrict__ sums, int scanned, PairSeg* __restrict__ psegs, uint32_t* __restrict__ prow,
    uint64_t* __restrict__ pc, uint32_t* __restrict__ cr, uint32_t* __restrict__ uhi, uint2* __restrict__ rt,
    uint32_t* __restrict__ rlo, uint32_t* __restrict__ Lp, uint32_t* __restrict__ Rp) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    constexpr uint32_t kWarps = kTileThreads / 32;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, tile0 = blockIdx.x * kWarps, tile = tile0 + warp;
    LSum at, all;  // before the tile, and through it
    if (scanned) {  // sums[tiles] is the whole
        at = tile < tiles ? sums[tile] : LSum::zero();
        all = tile < tiles ? sums[tile + 1] : at;
    } else {
        at = block_total(sums, tile0);
        for (uint32_t w = 0; w < warp && tile0 + w < tiles; w++) at = LSum::add(at, sums[tile0 + w]);
        all = tile < tiles ? LSum::add(at, sums[tile]) : at;
    }
    if (tile >= tiles) return;
    const uint32_t K = tile / per_slot, i0 = (tile - K * per_slot) * kTileThreads;
    const uint64_t base = (uint64_t)tile * kTileThreads;
    const uint32_t live = all.live - at.live;
    if (tile + 1 == tiles && lane == 0) {
        *Lp = all.live;
        *Rp = all.ranges;
        pc[all.live] = all.cand;
    }
    for (uint32_t j0 = 0; j0 < live; j0 += 32) {
        const uint32_t j = j0 + lane;
        const bool in = j < live;
        const uint32_t lo = in ? lo_in[base + j] : 0u, cnt = in ? cnt_in[base + j] : 0u;
        const uint32_t pl = in ? place[base + j] : 0u;
        const uint32_t i = i0 + (pl & (kStartsRange - 1));
        const uint32_t sh = in ? shard[i] : 0u, qs = in ? starts[i] : 0u, qe = in ? qend[i] : 0u, E = in ? emax[i] : 0u;
        const uint32_t fl = __ballot_sync(0xffffffffu, pl & kStartsRange);
        const uint64_t inc = warp_inclusive(cnt, lane);
        if (in) {
            const uint32_t c = at.live + j;
            const LayerQuery* L = layers + ((uint64_t)sh * nslots + K);
            const uint64_t first = L->off + lo;
            psegs[c] = PairSeg{tag == RUN_PACKED ? first | (uint64_t)row[i] << kRunRowShift : first, qs, qe};
            if (tag == RUN_ROW || tag == RUN_SHARD_ROW)
                prow[c] = (rows > 1 ? row[i] : 0u) + (tag == RUN_SHARD_ROW ? sh * rows : 0u);
            pc[c] = at.cand + inc - cnt;
            const uint32_t r = at.ranges + __popc(fl & ((2u << lane) - 1u)) - 1;  // the range it starts or continues
            cr[c] = r;
            if (pl & kStartsRange) {
                rt[r] = make_uint2(c, K * n + i);
                rlo[r] = lo;
            }
            // its range's last run unless the next live entry of the 32 goes on with the range
            if (lane == 31 || j + 1 == live || (fl >> (lane + 1) & 1u)) {
                uint32_t end = lo + cnt;
                if (E > qe) {  // an earlier query reaches further
                    const LayerQuery Lq = *L;
                    end = pp_layer(pos + Lq.off, btab + Lq.boff, Lq, E);
                }
                uhi[c] = end;
            }
        }
        at.ranges += __popc(fl);
        at.cand += __shfl_sync(0xffffffffu, inc, 31);
    }
}

// Per range: the reference's candidate count (sum over its runs of hi - lo) against the size of the
// union.  Where the two are close (narrow layers) the pair sweep reads each candidate once with
// trivial per-pair work; where candidate windows overlap heavily (broad layers) the rank sweep reads
// each union element once.  The unions of all ranges are summed into *union_total (the swept count of the
// metric), those swept by ranks per segment into seg_need.
constexpr uint32_t kRItems = 4, kRTile = kTileThreads * kRItems;

// Whether a range of `runs` runs, `cand` candidates and a union of `len` is swept by ranks.  A position of
// the rank sweep costs about pair_ratio candidates of the pair sweep; and a range swept by ranks needs its
// segment's ends sorted and summed and a rank table: about run_cost candidates a query.
__device__ __forceinline__ bool by_ranks(uint64_t cand, uint32_t len, uint32_t runs, uint32_t pair_ratio,
                                         uint32_t run_cost) {
    return cand > (uint64_t)pair_ratio * len + (uint64_t)run_cost * runs;
}

template <bool PDL>
__global__ void __launch_bounds__(kTileThreads) k_range_reduce(
    const uint32_t* __restrict__ Lp, const uint32_t* __restrict__ Rp, uint32_t n, const uint2* __restrict__ rt,
    const uint64_t* __restrict__ pc, const uint32_t* __restrict__ uhi, const uint32_t* __restrict__ rlo,
    const uint32_t* __restrict__ segnum, uint32_t pair_ratio, uint32_t run_cost, uint32_t* __restrict__ ulen,
    unsigned long long* __restrict__ seg_need, unsigned long long* __restrict__ union_total,
    RSum* __restrict__ sums) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    __shared__ RSum part[kTileThreads / 32];
    const uint32_t L = *Lp, R = *Rp, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned long long uni = 0;
    for (uint64_t tile = blockIdx.x; tile * kRTile < R; tile += gridDim.x) {
        RSum s = RSum::zero();
        uint2 f[kRItems];
        uint32_t c1[kRItems];
#pragma unroll
        for (uint32_t k = 0; k < kRItems; k++) {
            const uint64_t r = tile * kRTile + k * kTileThreads + threadIdx.x;
            f[k] = r < R ? rt[r] : make_uint2(0, 0);
            c1[k] = r + 1 < R ? rt[r + 1].x : L;
        }
#pragma unroll
        for (uint32_t k = 0; k < kRItems; k++) {
            const uint64_t r = tile * kRTile + k * kTileThreads + threadIdx.x;
            if (r >= R) continue;
            const uint64_t cand = pc[c1[k]] - pc[f[k].x];
            const uint32_t len = uhi[c1[k] - 1] - rlo[r];
            ulen[r] = len;
            uni += len;
            if (!by_ranks(cand, len, c1[k] - f[k].x, pair_ratio, run_cost)) s.pair += cand;
            else {
                s.rank += len;
                s.nrank++;
                atomicAdd(&seg_need[segnum[f[k].y % n] - 1], (unsigned long long)len);  // rank-swept positions
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            s.pair += __shfl_down_sync(0xffffffffu, s.pair, o);
            s.rank += __shfl_down_sync(0xffffffffu, s.rank, o);
            s.nrank += __shfl_down_sync(0xffffffffu, s.nrank, o);
        }
        if (lane == 0) part[warp] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (uint32_t w = 1; w < kTileThreads / 32; w++) s = RSum::add(s, part[w]);
            sums[tile] = s;
        }
        __syncthreads();  // part is reused
    }
    // one atomic per warp on the shared total
#pragma unroll
    for (int o = 16; o; o >>= 1) uni += __shfl_down_sync(0xffffffffu, uni, o);
    if (lane == 0 && uni) atomicAdd(union_total, uni);
}

// The rank work space: range q of those swept by ranks covers positions [rpos[q], rpos[q + 1]).  For the
// pair work space every range gets rpair[r]: kRankRange | the pair candidates before it, for a range
// swept by ranks (its runs take no room there), or the candidates of the rank ranges before it, for one
// swept by pairs (to be taken off its runs' pc).  The totals go to the counter block.
constexpr uint64_t kRankRange = 1ull << 63;
template <bool PDL>
__global__ void __launch_bounds__(kTileThreads) k_range_apply(
    const uint32_t* __restrict__ Lp, const uint32_t* __restrict__ Rp, uint32_t n, uint32_t nslots, uint32_t rows,
    const uint2* __restrict__ rt, const uint64_t* __restrict__ pc, const uint32_t* __restrict__ ulen,
    const uint32_t* __restrict__ rlo, const uint32_t* __restrict__ shard, const uint32_t* __restrict__ row,
    const uint32_t* __restrict__ segnum, const int32_t* __restrict__ slot, uint32_t pair_ratio, uint32_t run_cost,
    const RSum* __restrict__ sums, int scanned, RangeDesc* __restrict__ ranges,
    uint64_t* __restrict__ rpos, uint64_t* __restrict__ rpair, uint64_t* __restrict__ ppos,
    uint32_t* __restrict__ rank_count, unsigned long long* __restrict__ totals) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    constexpr uint32_t kWarps = kTileThreads / 32, kChunks = kWarps * kRItems;
    __shared__ RSum chunk[kChunks];
    const uint32_t L = *Lp, R = *Rp, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (R == 0 && blockIdx.x == 0 && threadIdx.x == 0) {
        rpos[0] = 0;
        ppos[0] = 0;
        *rank_count = 0;
        totals[0] = 0;
        totals[1] = 0;
    }
    for (uint64_t tile = blockIdx.x; tile * kRTile < R; tile += gridDim.x) {
        uint64_t first[kRItems], cand[kRItems];
        uint32_t len[kRItems], ent[kRItems], runs[kRItems];
#pragma unroll
        for (uint32_t k = 0; k < kRItems; k++) {
            const uint64_t r = tile * kRTile + k * kTileThreads + threadIdx.x;
            const uint2 f = r < R ? rt[r] : make_uint2(0, 0);
            const uint32_t c1 = r < R ? (r + 1 < R ? rt[r + 1].x : L) : 0u;
            ent[k] = f.y;
            runs[k] = c1 - f.x;
            first[k] = pc[f.x];
            cand[k] = pc[c1] - first[k];
            len[k] = r < R ? ulen[r] : 0u;
        }
        uint32_t rank = 0;  // bit k: range k of this thread is swept by ranks (see by_ranks)
#pragma unroll
        for (uint32_t k = 0; k < kRItems; k++) {
            const uint64_t r = tile * kRTile + k * kTileThreads + threadIdx.x;
            if (r >= R) cand[k] = 0;
            else if (by_ranks(cand[k], len[k], runs[k], pair_ratio, run_cost)) rank |= 1u << k;
            RSum s = RSum::zero();
            if (__any_sync(0xffffffffu, rank >> k & 1u)) {
                s = rank >> k & 1u ? RSum{len[k], 0ull, 1ull} : RSum{0ull, cand[k], 0ull};
                s = warp_total(s);
            } else {
                s.pair = cand[k];
#pragma unroll
                for (int o = 16; o; o >>= 1) s.pair += __shfl_down_sync(0xffffffffu, s.pair, o);
            }
            if (lane == 0) chunk[k * kWarps + warp] = s;
        }
        const RSum before = tile_prefix(sums, scanned, (uint32_t)tile);
        __syncthreads();
        static_assert(kChunks == 32, "one chunk a lane");
        const RSum mine = chunk[lane];
        RSum ex_chunk = shfl_up_words(warp_scan(mine, lane), 1);  // lane h: the chunks before h
        ex_chunk = lane ? RSum::add(before, ex_chunk) : before;
#pragma unroll
        for (uint32_t k = 0; k < kRItems; k++) {
            const uint64_t r = tile * kRTile + k * kTileThreads + threadIdx.x;
            const RSum at = shfl_words(ex_chunk, k * kWarps + warp);
            const bool by_rank = rank >> k & 1u;
            const RSum own = by_rank ? RSum{len[k], 0ull, 1ull} : RSum{0ull, cand[k], 0ull};
            RSum inc = own;
            if (__any_sync(0xffffffffu, by_rank)) inc = warp_scan(own, lane);
            else {
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint64_t w = __shfl_up_sync(0xffffffffu, inc.pair, o);
                    if (lane >= (uint32_t)o) inc.pair += w;
                }
            }
            inc = RSum::add(at, inc);
            if (r >= R) continue;
            if (by_rank) {
                const uint32_t K = ent[k] / n, i = ent[k] % n;
                const uint64_t q = inc.nrank - 1;
                rpair[r] = kRankRange | inc.pair;
                rpos[q] = inc.rank - len[k];
                ranges[q] = RangeDesc{rlo[r], (uint32_t)slot[(uint64_t)shard[i] * nslots + K],
                                      rows > 1 ? row[i] : 0u, segnum[i] - 1};
            } else {
                rpair[r] = first[k] - (inc.pair - cand[k]);
            }
            if (r + 1 == R) {
                rpos[inc.nrank] = inc.rank;
                ppos[L] = inc.pair;
                *rank_count = (uint32_t)inc.nrank;
                totals[0] = inc.rank;
                totals[1] = inc.pair;
            }
        }
        __syncthreads();  // chunk is reused
    }
}

// Pair work space: live run c's candidates begin at ppos[c].
template <bool PDL>
__global__ void k_run_pos(const uint32_t* __restrict__ Lp, const uint32_t* __restrict__ cr,
                          const uint64_t* __restrict__ pc, const uint64_t* __restrict__ rpair,
                          uint64_t* __restrict__ ppos) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    const uint32_t L = *Lp;
    for (uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; c < L; c += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t v = rpair[cr[c]];
        ppos[c] = v & kRankRange ? v & ~kRankRange : pc[c] - v;
    }
}

struct SweepParams {
    const uint64_t* rpos;   // exclusive scan of rank-range lengths, R + 1 entries; rpos[R] = total
    const uint32_t* rcount; // R (device): ranges swept by ranks
    const uint32_t* pcount; // L (device): live candidate runs
    const RangeDesc* ranges;
    const LayerDev* layers;
    const uint2* pos;
    const uint32_t* sid;
    const uint32_t* starts;  // sorted (segment, start)
    const uint32_t* ends;    // sorted (segment, end)
    const uint64_t* ps;      // exclusive prefix sums of starts
    const uint64_t* pe;      // exclusive prefix sums of ends
    uint32_t* counts;        // rows x D
    unsigned long long* bp;  // rows x D (may be null)
    uint32_t* queue;         // work counter
    const uint32_t* item_r0; // first range of each work item (items < item_cap)
    const uint64_t* ppos;    // pair work space: exclusive scan of candidate runs, L + 1 entries
    const PairSeg* psegs;
    const uint32_t* prow;    // rows of the runs (several rows, no histogram)
    const uint32_t* item_t0; // first run of each pair work item
    const SegTab* segtabs;   // per query segment
    const uint2* tab2;       // rank tables, bin b = (#starts, #ends) below b << shift
    uint64_t item_cap;
    uint32_t rows, D, chunk;
    uint32_t spread;         // work items wanted at least (0: items of exactly `chunk` positions)
    int smem_tally;          // 1: one row, shared-memory histograms
};

// Positions per work item of a work space of `total` positions: `chunk`, or fewer where that would
// leave fewer than `spread` items, in whole pair-sweep steps of 128 and at least one.  A run's totals
// are known only on the device, so every kernel that walks the items computes this for itself.
// Without it a small work space runs on a few warps, one step after the other: the 272 thousand
// candidates of 37 rows (102 thousand intervals) against 3.2e6 database intervals were 5 block items
// of 8,192 positions a warp, and the call took 1,306 us; sized so, 534 us.  Work spaces of at least
// `spread` full items are cut as before (2.1e8 candidates: 1,374 and 1,382 us a call, within noise).
__host__ __device__ __forceinline__ uint32_t item_size(uint64_t total, uint32_t chunk, uint32_t spread) {
    if (!spread) return chunk;
    const uint64_t even = ((total + spread - 1) / spread + 127) & ~127ull;
    return even < 128 ? (chunk < 128u ? chunk : 128u) : even < chunk ? (uint32_t)even : chunk;
}

// Galloping (exponential) search from a lower bound: first index in [lo, hi) with a[i] >= x
// (UPPER = false) or a[i] > x (UPPER = true).  Cost ~2 log2(answer - lo), so a rank found from
// the previous, nearby rank takes one or two probes.
template <bool UPPER>
__device__ __forceinline__ uint32_t gallop(const uint32_t* __restrict__ a, uint32_t lo, uint32_t hi, uint32_t x) {
    if (lo >= hi) return lo;
    uint32_t v = __ldg(a + lo);
    if (UPPER ? (v > x) : (v >= x)) return lo;
    uint32_t prev = lo, step = 1, nxt;
    for (;;) {  // invariant: a[prev] is below the bound
        if (step >= hi - prev) {
            nxt = hi;
            break;
        }
        nxt = prev + step;
        v = __ldg(a + nxt);
        if (UPPER ? (v > x) : (v >= x)) break;
        prev = nxt;
        step <<= 1;
    }
    return UPPER ? ub_u32(a, prev + 1, nxt, x) : lb_u32(a, prev + 1, nxt, x);
}

// Last range r in [r, rmax] with rpos[r] <= p (ranges are visited in increasing p).
__device__ __forceinline__ uint32_t range_advance(const uint64_t* __restrict__ rpos, uint32_t r, uint32_t rmax,
                                                  uint64_t p) {
    if (r >= rmax || __ldg(rpos + r + 1) > p) return r;
    uint32_t lo = r + 1, step = 1, hi;
    for (;;) {  // invariant: rpos[lo] <= p
        if (step > rmax - lo) {
            hi = rmax;
            break;
        }
        hi = lo + step;
        if (__ldg(rpos + hi) > p) {
            hi--;
            break;
        }
        lo = hi;
        step <<= 1;
    }
    while (lo < hi) {  // last m in [lo, hi] with rpos[m] <= p
        uint32_t m = (lo + hi + 1) >> 1;
        if (__ldg(rpos + m) <= p) lo = m; else hi = m - 1;
    }
    return lo;
}

// Work-item partition: item i covers positions [i * chunk, (i + 1) * chunk) of the concatenated
// ranges; item_r0[i] = the range holding its first position (last r with rpos[r] <= i * chunk),
// found by binary search over the range offsets.  One launch serves the rank ranges (rpos, *Rp
// ranges) and the pair runs (ppos, *Lp runs), grid-stride over the items of both.
template <bool PDL>
__global__ void k_item_ranges(const uint32_t* __restrict__ Rp,
                              const uint64_t* __restrict__ rpos, const uint32_t* __restrict__ Lp,
                              const uint64_t* __restrict__ ppos, uint32_t chunk, uint32_t spread, uint64_t item_cap,
                              uint32_t* __restrict__ item_r0, uint32_t* __restrict__ item_t0) {
    if constexpr (PDL) {
        pdl_wait();
        pdl_release();
    }
    const uint32_t R = *Rp, L = *Lp;
    const uint64_t rtot = rpos[R], ptot = ppos[L];
    const uint64_t g0 = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    const uint32_t rc = item_size(rtot, chunk, spread), pc = item_size(ptot, chunk, spread);
    const uint64_t ri = min((rtot + rc - 1) / rc, item_cap);
    const uint64_t pi = min((ptot + pc - 1) / pc, item_cap);
    for (uint64_t g = g0; g < ri + pi; g += (uint64_t)gridDim.x * blockDim.x) {
        const bool rank = g < ri;
        const uint64_t* a = rank ? rpos : ppos;
        const uint64_t i = rank ? g : g - ri;
        const uint64_t p = i * (rank ? rc : pc);
        uint64_t lo = 0, hi = rank ? R : L;
        while (lo < hi) {
            uint64_t m = (lo + hi + 1) >> 1;
            if (__ldg(a + m) <= p) lo = m; else hi = m - 1;
        }
        (rank ? item_r0 : item_t0)[i] = (uint32_t)lo;
    }
}

// A lane's position in the range list, with the range's descriptor cached in registers.
struct Cursor {
    uint32_t r;
    uint64_t rlo, rhi;  // [rpos[r], rpos[r + 1])
    RangeDesc rd;
    uint64_t base;      // element offset of the range's first DB interval in the index arrays
    SegTab tab;         // rank table of the range's query segment
};

__device__ __forceinline__ void cursor_load(const SweepParams& P, Cursor& c, uint32_t r) {
    c.r = r;
    c.rlo = __ldg(P.rpos + r);
    c.rhi = __ldg(P.rpos + r + 1);
    c.rd = P.ranges[r];
    c.base = P.layers[c.rd.layer_idx].off + c.rd.db_lo;
    c.tab = P.segtabs[c.rd.seg];
}

__device__ __forceinline__ void cursor_seek(const SweepParams& P, Cursor& c, uint64_t p, uint32_t rcap) {
    if (p >= c.rhi) cursor_load(P, c, range_advance(P.rpos, c.r, rcap, p));
}

// Bin entries (#starts, #ends) b and b + 1 for the bin of x, or (end, end) twice past the table.
__device__ __forceinline__ void bin_pair(const SweepParams& P, const SegTab& t, uint32_t x, uint2& lo, uint2& hi) {
    const uint32_t b = x >> t.shift;
    if (b >= t.nbins) {
        lo = hi = make_uint2(t.end, t.end);
        return;
    }
    lo = __ldg(P.tab2 + t.off + b);
    hi = __ldg(P.tab2 + t.off + b + 1);
}
// Ranks inside one bin: #starts < x given the bin's start counts, #ends <= x given its end counts.
__device__ __forceinline__ uint32_t starts_in(const SweepParams& P, uint32_t lo, uint32_t hi, uint32_t x) {
    return lo == hi ? lo : lb_u32(P.starts, lo, hi, x);
}
__device__ __forceinline__ uint32_t ends_in(const SweepParams& P, uint32_t lo, uint32_t hi, uint32_t x) {
    return lo == hi ? lo : ub_u32(P.ends, lo, hi, x);
}

// One DB interval d with the table entries of its start's bin (a0, a1) and its end's bin (b0, b1):
// count(d) = #{q.start < d.end} - #{q.end <= d.start}, and for a non-zero count the overlap
// Cov(d.end) - Cov(d.start) and the tally.
template <bool WITH_BP, bool MULTI>
__device__ __forceinline__ void sweep_one(const SweepParams& P, uint32_t qrow, uint2 d, uint32_t sid, uint2 a0,
                                          uint2 a1, uint2 b0, uint2 b1, uint32_t* s_cnt,
                                          unsigned long long* s_bp, uint32_t cta_row) {
    const uint32_t el_s = ends_in(P, a0.y, a1.y, d.x);
    const uint32_t sl_e = starts_in(P, b0.x, b1.x, d.y);
    const uint32_t cnt = sl_e - el_s;
    if (!cnt) return;
    unsigned long long bpv = 0;
    if (WITH_BP) {
        const uint32_t sl_s = starts_in(P, a0.x, a1.x, d.x);
        const uint32_t el_e = ends_in(P, b0.y, b1.y, d.y);
        if (sl_e == sl_s && el_e == el_s) {
            // no query starts or ends inside d: every overlapping query covers all of d
            bpv = (unsigned long long)(d.y - d.x) * cnt;
        } else {
            const unsigned long long ce = (unsigned long long)d.y * (unsigned long long)(sl_e - el_e) -
                                          __ldg(P.ps + sl_e) + __ldg(P.pe + el_e);
            const unsigned long long cs = (unsigned long long)d.x * (unsigned long long)(sl_s - el_s) -
                                          __ldg(P.ps + sl_s) + __ldg(P.pe + el_s);
            bpv = ce - cs;
        }
    }
    // one-row runs tally in the block's histogram; several-row runs (MULTI) in the histogram of the
    // block's current row, and only the other rows in the output matrix
    if (MULTI ? qrow == cta_row : P.smem_tally != 0) {
        atomicAdd(&s_cnt[sid], cnt);
        if (WITH_BP) add_u64(&s_bp[sid], bpv);
    } else {
        const uint64_t cell = (uint64_t)qrow * P.D + sid;
        atomicAdd(&P.counts[cell], cnt);
        if (WITH_BP) atomicAdd(&P.bp[cell], bpv);
    }
}

// Work items of the several-row sweeps are pulled by whole blocks: block item ci is the kCtaItems
// warp items [ci * kCtaItems, (ci + 1) * kCtaItems), one per warp.
constexpr uint32_t kCtaItems = 8;  // warps of a 256-thread block

// The row of the middle of block item ci (its warp item ci * kCtaItems + kCtaItems / 2, or the last
// item), from the first range (RANK) or run of that warp item: the row the block's histogram serves.
template <bool RANK>
__device__ __forceinline__ uint32_t cta_item_row(const SweepParams& P, uint32_t chunk, uint64_t ci, uint64_t items,
                                                 uint32_t rcap) {
    const uint64_t wi = min(ci * kCtaItems + kCtaItems / 2, items - 1);
    const uint64_t* off = RANK ? P.rpos : P.ppos;
    uint32_t r;
    if (wi < P.item_cap) {
        r = __ldg((RANK ? P.item_r0 : P.item_t0) + wi);
    } else {
        const uint64_t p = wi * chunk;
        uint64_t lo = 0, hi = rcap;
        while (lo < hi) { uint64_t m = (lo + hi + 1) >> 1; if (__ldg(off + m) <= p) lo = m; else hi = m - 1; }
        r = (uint32_t)lo;
    }
    return RANK ? P.ranges[r].qrow : (uint32_t)(__ldg(&P.psegs[r].base) >> kRunRowShift);
}

// The outer loop of the several-row sweeps.  Blocks pull block items (kCtaItems warp items) from the
// queue one at a time, so that the blocks running at once work on neighbouring items: with the
// region work order they read the same database region, from L2 after the first.  The block's
// histogram serves one row at a time: before an item whose row differs from the row it holds, it is
// added to the outputs and cleared (and once more at the end).  item_fn(warp_item, row) walks one
// warp item; flush_fn(row) adds and clears the histogram.
template <bool RANK, typename ItemFn, typename FlushFn>
__device__ __forceinline__ void multi_row_loop(const SweepParams& P, uint32_t chunk, uint64_t items, uint32_t rcap,
                                               ItemFn item_fn, FlushFn flush_fn) {
    __shared__ uint32_t s_ctl[2][2];  // (item, row) of this turn and of the next
    constexpr uint32_t kNone = 0xFFFFFFFFu;
    uint32_t cur = kNone;  // the row the histogram holds (block-uniform)
    auto publish = [&](uint32_t turn, uint32_t ci) {
        s_ctl[turn][0] = ci;
        if ((uint64_t)ci * kCtaItems < items) s_ctl[turn][1] = cta_item_row<RANK>(P, chunk, ci, items, rcap);
    };
    if (threadIdx.x == 0) publish(0, atomicAdd(P.queue, 1u));
    __syncthreads();
    for (uint32_t turn = 0;; turn ^= 1) {
        const uint64_t ci = s_ctl[turn][0];
        if (ci * kCtaItems >= items) break;
        const uint32_t row = s_ctl[turn][1];
        if (row != cur) {
            if (cur != kNone) {
                flush_fn(cur);
                __syncthreads();
            }
            cur = row;
        }
        uint32_t next = 0;
        if (threadIdx.x == 0) next = atomicAdd(P.queue, 1u);  // arrives while the item is walked
        const uint64_t item = ci * kCtaItems + (threadIdx.x >> 5);
        if (item < items) item_fn((uint32_t)item, cur);
        if (threadIdx.x == 0) publish(turn ^ 1, next);  // read by all before this turn: one barrier ago
        __syncthreads();  // the item is done before the histogram may be flushed
    }
    if (cur != kNone) flush_fn(cur);
}

// Adds the block's histogram to row `row` of the outputs and clears it (between two __syncthreads).
template <bool WITH_BP>
__device__ __forceinline__ void flush_row(const SweepParams& P, uint32_t row, uint32_t* s_cnt,
                                          unsigned long long* s_bp) {
    const uint64_t base = (uint64_t)row * P.D;
    for (uint32_t k = threadIdx.x; k < P.D; k += blockDim.x) {
        const uint32_t c = s_cnt[k];
        if (c) {
            atomicAdd(&P.counts[base + k], c);
            s_cnt[k] = 0;
        }
        if (WITH_BP) {
            const unsigned long long b = s_bp[k];
            if (b) {
                atomicAdd(&P.bp[base + k], b);
                s_bp[k] = 0;
            }
        }
    }
}

constexpr uint32_t kUnroll = 2;      // DB intervals per lane per step of the rank sweep
constexpr uint32_t kPairUnroll = 4;  // candidates per lane per step of the pair sweep
// Run boundaries inside a step up to which they are counted one by one (nine instructions each); beyond,
// pairs_step_dense (a hundred and fifty or so for any number, and a call).
constexpr uint32_t kFewBounds = 16;

// One work item of the rank sweep: positions [item * chunk, (item + 1) * chunk) of the concatenated
// rank ranges, walked by one warp.
template <bool WITH_BP, bool MULTI>
__device__ __forceinline__ void sweep_item(const SweepParams& P, uint32_t chunk, uint32_t item, uint32_t lane, uint32_t rcap,
                                           uint64_t total, uint32_t* s_cnt, unsigned long long* s_bp,
                                           uint32_t cta_row) {
    const uint64_t p0 = (uint64_t)item * chunk;
    const uint64_t p1 = min(p0 + chunk, total);
    uint32_t r0;
    if (item < P.item_cap) {
        r0 = __ldg(P.item_r0 + item);
    } else {
        uint64_t lo = 0, hi = rcap;
        while (lo < hi) { uint64_t m = (lo + hi + 1) >> 1; if (__ldg(P.rpos + m) <= p0) lo = m; else hi = m - 1; }
        r0 = (uint32_t)lo;
    }
    Cursor c;
    cursor_load(P, c, r0);
    for (uint64_t pb = p0 + lane; pb < p1; pb += 32 * kUnroll) {
        const uint64_t plast = min(pb + 32 * (kUnroll - 1), p1 - 1 - ((p1 - 1 - pb) & 31));
        cursor_seek(P, c, pb, rcap);
        if (plast < c.rhi) {
            // all of this lane's positions of the step lie in one range: batch the loads
            const SegTab t = c.tab;
            const uint64_t off = c.base - c.rlo;
            uint2 d[kUnroll];
            uint32_t sid[kUnroll];
#pragma unroll
            for (uint32_t j = 0; j < kUnroll; j++) {
                const uint64_t pj = pb + 32 * j;
                if (pj < p1) {
                    d[j] = __ldg(P.pos + off + pj);
                    sid[j] = __ldg(P.sid + off + pj);
                } else {
                    d[j] = make_uint2(0, 0);
                    sid[j] = 0;
                }
            }
            uint2 a0[kUnroll], a1[kUnroll], b0[kUnroll], b1[kUnroll];
#pragma unroll
            for (uint32_t j = 0; j < kUnroll; j++) {
                bin_pair(P, t, d[j].x, a0[j], a1[j]);
                bin_pair(P, t, d[j].y, b0[j], b1[j]);
            }
#pragma unroll
            for (uint32_t j = 0; j < kUnroll; j++)
                if (pb + 32 * j < p1)
                    sweep_one<WITH_BP, MULTI>(P, c.rd.qrow, d[j], sid[j], a0[j], a1[j], b0[j], b1[j], s_cnt, s_bp, cta_row);
        } else {
            // the step crosses a range boundary: one position at a time
            for (uint64_t pj = pb; pj < p1 && pj <= pb + 32 * (kUnroll - 1); pj += 32) {
                cursor_seek(P, c, pj, rcap);
                const uint64_t di = c.base + (pj - c.rlo);
                const uint2 d = __ldg(P.pos + di);
                uint2 a0, a1, b0, b1;
                bin_pair(P, c.tab, d.x, a0, a1);
                bin_pair(P, c.tab, d.y, b0, b1);
                sweep_one<WITH_BP, MULTI>(P, c.rd.qrow, d, __ldg(P.sid + di), a0, a1, b0, b1, s_cnt, s_bp, cta_row);
            }
        }
    }
}

template <bool WITH_BP, bool MULTI>
__global__ void __launch_bounds__(256, 5) k_sweep(const __grid_constant__ SweepParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned long long* s_bp = reinterpret_cast<unsigned long long*>(smem);
    uint32_t* s_cnt = reinterpret_cast<uint32_t*>(smem + (WITH_BP ? (size_t)P.D * 8 : 0));
    const uint32_t lane = threadIdx.x & 31u;

    const uint32_t rcap = *P.rcount;
    const uint64_t total = P.rpos[rcap];
    const uint32_t chunk = item_size(total, P.chunk, P.spread);
    // a block with no item for any of its warps (every warp pulls on until the items run out)
    if ((uint64_t)blockIdx.x * kCtaItems * chunk >= total) return;
    if (P.smem_tally) {
        for (uint32_t k = threadIdx.x; k < P.D; k += blockDim.x) {
            s_cnt[k] = 0;
            if (WITH_BP) s_bp[k] = 0;
        }
    }
    __syncthreads();
    if constexpr (MULTI) {
        // several rows: blocks pull block items (kCtaItems warp items each); the block's histogram
        // serves the row of the current item and is added to the outputs on a row change
        const uint64_t items = (total + chunk - 1) / chunk;
        multi_row_loop<true>(
            P, chunk, items, rcap,
            [&](uint32_t item, uint32_t row) {
                sweep_item<WITH_BP, true>(P, chunk, item, lane, rcap, total, s_cnt, s_bp, row);
            },
            [&](uint32_t row) { flush_row<WITH_BP>(P, row, s_cnt, s_bp); });
    } else {
        // Warps pull work items independently (no block-wide barrier inside the loop).  A step covers
        // 32 * kUnroll consecutive positions; lane l takes positions pb + l + 32 j, so every load of the
        // DB arrays is coalesced, and the kUnroll DB intervals of a lane and their rank-table entries
        // are all requested before any of them is used.  count(d) = #{q.start < d.end} -
        // #{q.end <= d.start} needs two ranks, each one rank-table read plus, rarely, a search inside
        // one bin.
        for (;;) {
            uint32_t item = 0;
            if (lane == 0) item = atomicAdd(P.queue, 1u);
            item = __shfl_sync(0xffffffffu, item, 0);
            if ((uint64_t)item * chunk >= total) break;
            sweep_item<WITH_BP, false>(P, chunk, item, lane, rcap, total, s_cnt, s_bp, 0u);
        }
        if (P.smem_tally) {
            __syncthreads();
            for (uint32_t k = threadIdx.x; k < P.D; k += blockDim.x) {
                if (s_cnt[k]) atomicAdd(&P.counts[k], s_cnt[k]);
                if (WITH_BP && s_bp[k]) atomicAdd(&P.bp[k], s_bp[k]);
            }
        }
    }
}

// A pair candidate d of the run with query interval [qs, qe) and Q_SID qrow: when d.end > qs it
// adds 1 and min(ends) - max(starts) to cell (qrow, sid) — in the block's shared histograms (SMEM,
// one query row) or in the output matrix.
template <bool WITH_BP, bool SMEM, int MULTI>
__device__ __forceinline__ void pair_tally(uint32_t* counts, unsigned long long* bp, uint32_t D, uint32_t qs,
                                           uint32_t qe, uint32_t qrow, uint2 d, uint32_t sid, uint32_t* s_cnt,
                                           unsigned long long* s_bp, uint32_t cta_row) {
    if (d.y <= qs) return;
    if (SMEM && (!MULTI || qrow == cta_row)) {
        atomicAdd(&s_cnt[sid], 1u);
        if (WITH_BP) add_u64_lo(&s_bp[sid], min(qe, d.y) - max(qs, d.x));
    } else {
        const uint64_t cell = (uint64_t)qrow * D + sid;
        atomicAdd(&counts[cell], 1u);
        if (WITH_BP) atomicAdd(&bp[cell], (unsigned long long)(min(qe, d.y) - max(qs, d.x)));
    }
}

// One step of the pair sweep (positions pb + [0, span], the first of them in run t) over many short runs:
// the boundaries inside the step are counted per position in shared memory (`cntr`, 128 words of the warp's
// own) and the counts summed along the step, which gives every position's run; its descriptor, element and
// tally follow with all four positions of a lane in flight.  A stretch of more than kDenseGroups x 32
// boundaries (empty runs of ranges swept by ranks) is searched position by position instead.
// Files of 1e6 intervals against 3.2e6 have about two candidates a run: 52e9 candidates/s with a search per
// position, 1.3e11 so.
constexpr int kDenseGroups = 16;
template <bool WITH_BP, bool SMEM, int MULTI>
__device__ __forceinline__ void pairs_step_dense(const uint64_t* __restrict__ ppos, const PairSeg* __restrict__ psegs,
                                              const uint32_t* __restrict__ prow, const uint2* __restrict__ pos,
                                              const uint32_t* __restrict__ sidv, uint32_t* counts,
                                              unsigned long long* bp, uint32_t D, uint32_t t, uint32_t rcap,
                                              uint64_t pb, uint32_t span, uint32_t lane, uint32_t* cntr,
                                              uint32_t* s_cnt, unsigned long long* s_bp, uint32_t cta_row) {
    reinterpret_cast<uint4*>(cntr)[lane] = make_uint4(0, 0, 0, 0);
    __syncwarp();
    bool all = false;
    for (int g = 0; g < kDenseGroups && !all; g++) {
        const uint64_t k = (uint64_t)t + 1 + 32 * g + lane;
        const uint64_t B = k <= rcap ? __ldg(ppos + k) : ~0ull;
        const bool in = B - pb <= span;  // B > pb: run t holds pb
        if (in) atomicAdd(&cntr[(uint32_t)(B - pb)], 1u);
        all = __any_sync(0xffffffffu, !in);
    }
    __syncwarp();
    if (all) {  // counts into sums along the step
        uint4 c = reinterpret_cast<uint4*>(cntr)[lane];
        c.y += c.x;
        c.z += c.y;
        c.w += c.z;
        uint32_t inc = c.w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t w = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= (uint32_t)o) inc += w;
        }
        inc -= c.w;
        reinterpret_cast<uint4*>(cntr)[lane] = make_uint4(c.x + inc, c.y + inc, c.z + inc, c.w + inc);
    } else {
#pragma unroll 1
        for (uint32_t o = lane; o <= span; o += 32) cntr[o] = range_advance(ppos, t, rcap, pb + o) - t;
    }
    __syncwarp();
    constexpr uint32_t U = kPairUnroll / 2;  // four at once need more registers than the sweep has
#pragma unroll 1
    for (uint32_t o0 = lane; o0 <= span; o0 += 32 * U) {
        uint2 d[U], q[U];
        uint32_t sid[U], row[U];
#pragma unroll
        for (uint32_t j = 0; j < U; j++) {
            const uint32_t o = o0 + 32 * j;
            d[j] = make_uint2(0, 0);  // never a hit: d.y = 0 <= qs
            q[j] = make_uint2(0, 0);
            sid[j] = row[j] = 0;
            if (o <= span) {
                const uint32_t run = t + cntr[o];
                const uint4 w = __ldg(reinterpret_cast<const uint4*>(psegs + run));
                const uint64_t di = run_base<MULTI>(((uint64_t)w.y << 32) | w.x) + (pb + o - __ldg(ppos + run));
                q[j] = make_uint2(w.z, w.w);
                d[j] = __ldg(pos + di);
                sid[j] = __ldg(sidv + di);
                if (MULTI) row[j] = w.y >> (kRunRowShift - 32);
                else if (!SMEM && prow) row[j] = __ldg(prow + run);
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < U; j++)
            pair_tally<WITH_BP, SMEM, MULTI>(counts, bp, D, q[j].x, q[j].y, row[j], d[j], sid[j], s_cnt, s_bp, cta_row);
    }
    __syncwarp();  // cntr is reused by the next step
}

// The same as a call.  Inlined into the one-row sweep, which has 32 registers a thread, it spills into the loop; a
// call in the several-row sweep leaves 16 registers for all that lives across it, and that spilled 148 bytes a thread
// there: 48 files against 2e8 intervals 4,201 us so (six blocks an SM), 3,638 inlined.
template <bool WITH_BP, bool SMEM>
__device__ __noinline__ void pairs_step_dense_call(const uint64_t* __restrict__ ppos, const PairSeg* __restrict__ psegs,
                                                   const uint32_t* __restrict__ prow, const uint2* __restrict__ pos,
                                                   const uint32_t* __restrict__ sidv, uint32_t* counts,
                                                   unsigned long long* bp, uint32_t D, uint32_t t, uint32_t rcap,
                                                   uint64_t pb, uint32_t span, uint32_t lane, uint32_t* cntr,
                                                   uint32_t* s_cnt, unsigned long long* s_bp) {
    pairs_step_dense<WITH_BP, SMEM, 0>(ppos, psegs, prow, pos, sidv, counts, bp, D, t, rcap, pb, span, lane, cntr, s_cnt,
                                       s_bp, 0u);
}

// The pair sweep: the reference's scan (src/sweep/query.rs:104-115) over the candidate runs of the
// queries of pair ranges, every candidate read once by one lane (consecutive positions of a run are
// consecutive DB elements, so the loads coalesce).  A candidate d of query q overlaps when
// d.end > q.start (d.start < q.end and the look-back bound hold by construction of the run); it
// adds 1 and min(ends) - max(starts).
//
// A warp takes work items of `chunk` positions from the queue and walks each in steps of 32 *
// kPairUnroll consecutive positions, lane l taking l + 32 j, in 32-bit offsets from the item's first.
// The warp keeps the run t of the step's first position (uniform), so the choice between the forms
// below never splits the warp.  When the step lies in run t, every lane requests all its DB intervals
// and sids before using any.  When it spans several runs (most steps, at the seventy candidates a run
// of whole-genome files), lane l holds the boundary ppos[t + 1 + l] of the following runs: a position's
// run is t plus the number of boundaries at or below it, counted over the few boundaries inside the
// step, and the run descriptors come from L1.
// Bound: L1 wavefronts (70% of its cycles: 12 bytes and two shared-memory atomics a candidate) and
// issue (65%).  Blocks an SM, 1.04e9 candidates of 48 files against 2e8 intervals and 256 files against 3.2e6,
// several-row form: five 3,826 and 893 us; six (40 registers, 16 bytes spilled) 3,638 and 823; eight (32 registers, 36
// bytes spilled, as seven compiles too) 3,530 to 3,545 and 681 to 685.
// One work item of the pair sweep (positions [item * chunk, (item + 1) * chunk) of the concatenated
// candidate runs), walked by one warp.
template <bool WITH_BP, bool SMEM, int MULTI>
__device__ __forceinline__ void pairs_item(const SweepParams& P, uint32_t chunk, uint32_t item, uint32_t lane, uint32_t rcap,
                                           uint64_t total, uint32_t* cntr, uint32_t* s_cnt,
                                           unsigned long long* s_bp, uint32_t cta_row) {
    const uint64_t p0 = (uint64_t)item * chunk;
    const uint32_t len = (uint32_t)min((uint64_t)chunk, total - p0);
    uint32_t t;
    if (item < P.item_cap) {
        t = __ldg(P.item_t0 + item);
    } else {
        uint64_t lo = 0, hi = rcap;
        while (lo < hi) { uint64_t m = (lo + hi + 1) >> 1; if (__ldg(P.ppos + m) <= p0) lo = m; else hi = m - 1; }
        t = (uint32_t)lo;
    }
    // the row of a run: packed in its base (MULTI), or beside it where the tally goes straight to several rows
    const bool rowed = !SMEM && P.rows > 1;
    // run t: its candidates are the elements base + (offset in the item), up to offset rhi
    uint64_t base;
    uint32_t rhi, qs, qe, prow;
    auto load_run = [&]() {
        const uint64_t lo = __ldg(P.ppos + t), hi = __ldg(P.ppos + t + 1);
        const uint4 w = __ldg(reinterpret_cast<const uint4*>(P.psegs + t));
        base = run_base<MULTI>(((uint64_t)w.y << 32) | w.x) - lo + p0;
        rhi = (uint32_t)min(hi - p0, (uint64_t)0xffffffffu);
        qs = w.z;
        qe = w.w;
        prow = MULTI ? w.y >> (kRunRowShift - 32) : rowed ? __ldg(P.prow + t) : 0u;
    };
    load_run();
    for (uint32_t ob = 0; ob < len; ob = len - ob > 32 * kPairUnroll ? ob + 32 * kPairUnroll : len) {
        const uint32_t span = min(32 * kPairUnroll, len - ob) - 1;
        if (ob >= rhi) {
            t = range_advance(P.ppos, t, rcap, p0 + ob);
            load_run();
        }
        if (ob + span < rhi) {
            const uint2* pos = P.pos + (base + ob);
            const uint32_t* sidv = P.sid + (base + ob);
            uint2 d[kPairUnroll];
            uint32_t sid[kPairUnroll];
#pragma unroll
            for (uint32_t j = 0; j < kPairUnroll; j++) {
                const uint32_t o = lane + 32 * j;
                d[j] = make_uint2(0, 0);  // never a hit: d.y = 0 <= qs
                sid[j] = 0;
                if (o <= span) {
                    d[j] = __ldg(pos + o);
                    sid[j] = __ldg(sidv + o);
                }
            }
#pragma unroll
            for (uint32_t j = 0; j < kPairUnroll; j++)
                pair_tally<WITH_BP, SMEM, MULTI>(P.counts, P.bp, P.D, qs, qe, prow, d[j], sid[j], s_cnt, s_bp, cta_row);
            continue;
        }
        // lane l: boundary ppos[t + 1 + l] as an offset in the step (> 0, since run t holds its first
        // position); offsets inside the step fit 32 bits
        const uint64_t B = (uint64_t)t + 1 + lane <= rcap ? __ldg(P.ppos + t + 1 + lane) - (p0 + ob) : ~0ul;
        const uint32_t rel = (uint32_t)min(B, (uint64_t)0xffffffffu);
        const uint32_t nb = __popc(__ballot_sync(0xffffffffu, rel <= span));
        if (nb > kFewBounds) {
            if constexpr (MULTI)
                pairs_step_dense<WITH_BP, SMEM, MULTI>(P.ppos, P.psegs, nullptr, P.pos, P.sid, P.counts, P.bp, P.D, t,
                                                       rcap, p0 + ob, span, lane, cntr, s_cnt, s_bp, cta_row);
            else
                pairs_step_dense_call<WITH_BP, SMEM>(P.ppos, P.psegs, rowed ? P.prow : nullptr, P.pos, P.sid, P.counts,
                                                     P.bp, P.D, t, rcap, p0 + ob, span, lane, cntr, s_cnt, s_bp);
            continue;  // the next step starts past rhi: range_advance finds its run
        }
        // byte j of kk: position lane + 32 j lies in run t + that; a boundary at offset v counts for the
        // positions at or past it, which are those of j >= (v + 31 - lane) / 32
        uint32_t kk = 0;
        for (uint32_t i = 0; i < nb; i++)  // rel[0..nb) are the boundaries inside the step
            kk += __funnelshift_lc(0u, 0x01010101u, ((__shfl_sync(0xffffffffu, rel, i) + 31 - lane) >> 2) & 0x38u);
        uint2 d[kPairUnroll];
        uint32_t sid[kPairUnroll];
#pragma unroll
        for (uint32_t j = 0; j < kPairUnroll; j++) {
            // run t + k (k > 0) starts at offset rel[k - 1]; t + k < rcap since ppos[rcap] = total > the step's last
            const uint32_t k = (kk >> (8 * j)) & 0xffu, o = lane + 32 * j;
            const uint32_t rb = __shfl_sync(0xffffffffu, rel, k - 1);
            d[j] = make_uint2(0, 0);
            sid[j] = 0;
            if (o <= span) {
                const uint64_t di = k ? run_base<MULTI>(__ldg(&P.psegs[t + k].base)) + (o - rb) : base + (ob + o);
                d[j] = __ldg(P.pos + di);
                sid[j] = __ldg(P.sid + di);
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < kPairUnroll; j++) {
            const uint32_t run = t + ((kk >> (8 * j)) & 0xffu);
            const uint4 w = __ldg(reinterpret_cast<const uint4*>(P.psegs + run));
            const uint32_t qrow = MULTI ? w.y >> (kRunRowShift - 32) : rowed ? __ldg(P.prow + run) : 0u;
            pair_tally<WITH_BP, SMEM, MULTI>(P.counts, P.bp, P.D, w.z, w.w, qrow, d[j], sid[j], s_cnt, s_bp, cta_row);
        }
        // the run of the next step's first position, from the boundaries in hand (at least one, ppos[t + 1],
        // lies at or below it)
        const uint32_t kn = __popc(__ballot_sync(0xffffffffu, rel <= span + 1));
        if (ob + span + 1 < len && kn < 32) {
            t += kn;
            load_run();
        }
    }
}

template <bool WITH_BP, bool SMEM, int MULTI>
__global__ void __launch_bounds__(256, 8) k_pairs(const __grid_constant__ SweepParams P) {
    extern __shared__ __align__(16) unsigned char smem[];
    unsigned long long* s_bp = reinterpret_cast<unsigned long long*>(smem);
    uint32_t* s_cnt = reinterpret_cast<uint32_t*>(smem + (WITH_BP ? (size_t)P.D * 8 : 0));
    __shared__ __align__(16) uint32_t s_cntr[8][32 * kPairUnroll];  // pairs_step_dense, one row per warp
    uint32_t* cntr = s_cntr[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t rcap = *P.pcount;
    const uint64_t total = P.ppos[rcap];
    const uint32_t chunk = item_size(total, P.chunk, P.spread);
    if ((uint64_t)blockIdx.x * kCtaItems * chunk >= total) return;  // as k_sweep
    if (SMEM)
        for (uint32_t k = threadIdx.x; k < P.D; k += blockDim.x) {
            s_cnt[k] = 0;
            if (WITH_BP) s_bp[k] = 0;
        }
    __syncthreads();
    if constexpr (MULTI) {
        // several rows: block items, the histogram serves one row at a time (as k_sweep)
        const uint64_t items = (total + chunk - 1) / chunk;
        multi_row_loop<false>(
            P, chunk, items, rcap,
            [&](uint32_t item, uint32_t row) {
                pairs_item<WITH_BP, true, 1>(P, chunk, item, lane, rcap, total, cntr, s_cnt, s_bp, row);
            },
            [&](uint32_t row) { flush_row<WITH_BP>(P, row, s_cnt, s_bp); });
    } else {
        for (;;) {
            uint32_t item = 0;
            if (lane == 0) item = atomicAdd(P.queue, 1u);
            item = __shfl_sync(0xffffffffu, item, 0);
            if ((uint64_t)item * chunk >= total) break;
            pairs_item<WITH_BP, SMEM, 0>(P, chunk, item, lane, rcap, total, cntr, s_cnt, s_bp, 0u);
        }
        if (SMEM) {
            __syncthreads();
            for (uint32_t k = threadIdx.x; k < P.D; k += blockDim.x) {
                if (s_cnt[k]) atomicAdd(&P.counts[k], s_cnt[k]);
                if (WITH_BP && s_bp[k]) atomicAdd(&P.bp[k], s_bp[k]);
            }
        }
    }
}

// `--intervals` mode (query_sweep_pairs, src/sweep/query.rs:11-41): every overlapping pair of the
// candidate runs, listed in the order of the pair work space (layer slot, shard, row, query start,
// DB start).  Item i = positions [i * chunk, (i + 1) * chunk) is walked by one warp, 32 positions
// per step: the count pass stores the item's hits, the emit pass writes them from the item's
// offset (an exclusive scan of the counts) at their ballot ranks, so the list needs no atomics and
// comes out in the same order every time.
template <bool EMIT>
__global__ void __launch_bounds__(256) k_pair_list(const uint64_t* __restrict__ ppos,
                                                   const uint32_t* __restrict__ pcount,
                                                   const PairSeg* __restrict__ psegs,
                                                   const uint32_t* __restrict__ prow, uint32_t rows,
                                                   const uint2* __restrict__ pos, const uint32_t* __restrict__ sid,
                                                   uint64_t items, uint32_t chunk,
                                                   uint64_t* __restrict__ item_hits,
                                                   const uint64_t* __restrict__ item_base, rgl_pair* __restrict__ out) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint32_t rcap = *pcount;
    const uint64_t total = ppos[rcap];
    for (uint64_t item = warp; item < items; item += nwarps) {
        const uint64_t p0 = item * chunk, p1 = min(p0 + chunk, total);
        uint64_t lo = 0, hi = rcap;  // last run t with ppos[t] <= p0
        while (lo < hi) {
            const uint64_t m = (lo + hi + 1) >> 1;
            if (__ldg(ppos + m) <= p0) lo = m; else hi = m - 1;
        }
        uint32_t t = (uint32_t)lo;
        uint64_t rhi = __ldg(ppos + t + 1), rlo = __ldg(ppos + t);
        PairSeg ps = psegs[t];
        const uint64_t base = EMIT ? item_base[item] : 0;
        uint64_t done = 0;
        for (uint64_t s = p0; s < p1; s += 32) {
            const uint64_t p = s + lane;
            bool hit = false;
            uint2 d = make_uint2(0, 0);
            uint64_t di = 0;
            if (p < p1) {
                if (p >= rhi) {
                    t = range_advance(ppos, t, rcap, p);
                    rlo = __ldg(ppos + t);
                    rhi = __ldg(ppos + t + 1);
                    ps = psegs[t];
                }
                di = ps.base + (p - rlo);
                d = __ldg(pos + di);
                hit = d.y > ps.qs;
            }
            const uint32_t ballot = __ballot_sync(0xffffffffu, hit);
            if (EMIT && hit) {
                const uint32_t rank = __popc(ballot & ((1u << lane) - 1u));
                rgl_pair r;
                r.query_start = ps.qs;
                r.query_end = ps.qe;
                r.db_start = d.x;
                r.db_end = d.y;
                const uint32_t sr = __ldg(prow + t);  // shard * rows + row
                r.row = sr % rows;
                r.sid = __ldg(sid + di);
                r.shard = sr / rows;
                r.intersection_bp = min(ps.qe, d.y) - max(ps.qs, d.x);
                out[base + done + rank] = r;
            }
            done += __popc(ballot);
        }
        if (!EMIT && lane == 0) item_hits[item] = done;
    }
}

}  // namespace rgl

using namespace rgl;

// ================================================================================================
// Context
// ================================================================================================
struct rgl_context {
    rgl_index* idx = nullptr;  // holds one reference of the index
    int device = 0;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    // second stream for the independent chains of a run (the end-key sort, the prefix sums of the
    // starts and ends, the rank tables), forked from and joined back into `stream`
    cudaStream_t side = nullptr;
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    int num_sms = 148;
    DevBuf iv, blk_off, blk_shard, key_a, key_b, val_a, val_b, ekey_a, ekey_b;
    DevBuf starts, ends, shard, row, segnum, seg_begin, ps, pe, emax;
    DevBuf lo, cnt, place, ranges, rpos, cub_tmp, small, out_counts, out_bp, item_r0;
    DevBuf segtab, tab2;
    DevBuf pc, cr, uhi, rt, rlo, ulen, rpair, ppos, psegs, prow, item_t0, seg_need;
    DevBuf sums, esums;  // tile summaries, of the main and of the side stream
    DevBuf cub_tmp2;  // the side stream's own scratch
    DevBuf sortplan;  // block-local sort: order flags, tile and merge-chunk prefix counts, two pass words
    DevBuf sort_tab, sort_rank;  // its segment-order layout, for the single-call entry points
    DevBuf item_hits, item_base, pairs;  // intervals mode
    DevBuf bt_off, bt_shard, acc;  // batched form: sub-batch block tables (offsets; shards then rows), stats
    uint32_t* h_small = nullptr;  // pinned mirror of `small`
    unsigned char* h_io = nullptr;  // pinned staging of the host entry points (kHostIoBytes)
    unsigned long long* h_acc = nullptr;  // pinned mirror of `acc`
    uint64_t ws_sig = 0;          // changes whenever a workspace buffer is reallocated
    // the CUDA graph of the last batch run with RGL_BF_GRAPH, replayed while the batch is unchanged
    struct GraphCache {
        std::vector<uint64_t> key;
        cudaGraph_t graph = nullptr;
        cudaGraphExec_t exec = nullptr;
        DevBuf t_off, t_shard;  // the graph's own copies of the block tables
        uint32_t nodes = 0, launches = 0, subs = 0;
    } gc;
    // host-input batches: two staging buffers filled on a copy stream while the other is swept
    DevBuf stage[2];
    cudaStream_t copy_stream = nullptr;
    cudaEvent_t ev_copied[2] = {nullptr, nullptr}, ev_used[2] = {nullptr, nullptr};
    bool has_tuned = false;       // rgl_batch_autotune result
    rgl_query_opts tuned{};
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
    uint64_t res_n = 0;           // the workspace covers runs of res_n intervals, res_rows rows and
    uint32_t res_rows = 0;        // res_blk blocks (every buffer's size depends on one of the three)
    uint32_t res_blk = 0;
    bool ws_ready = false;        // res_* describe the workspace (set by the first full sizing)
    // sweep-kernel timing on the launch stream (rgl_context_set_timing)
    bool timing = false;
    std::vector<cudaEvent_t> tev;  // pairs (start, end)
    size_t tev_used = 0;
    // state of the last launch, for stats
    uint64_t last_tot = 0;
    uint32_t last_launches = 0;
    uint32_t last_n = 0;
    uint32_t last_chunk = 1024, last_spread = 0;  // its work-item size (see item_size)
};

namespace {

// Work items whose first range is precomputed; items beyond it search the range list themselves.
constexpr uint64_t kItemCap = 1ull << 22;

// Default work-item size of runs with several output rows.
constexpr uint32_t kMultiRowChunk = 8192;

// What a query of a range swept by ranks costs besides, in candidates of the pair sweep (see by_ranks).
// 256 files against 3.2e6 intervals: hardly a range is worth it (7.6 -> 6.4 ms); 48 files against 2e8: 16
// moved ranges to the pair sweep that were faster by ranks (k_pairs + k_sweep 6.2 -> 6.4 ms), 4 does not.
constexpr uint32_t kRankRunCost = 4;

// Runs up to this many query intervals chain their kernels with programmatic dependent launch.
constexpr uint64_t kPdlMaxIntervals = 1ull << 21;

// Query intervals per pipeline run: the rank tables (up to 10 entries per interval) use 31-bit offsets.
constexpr uint64_t kMaxRunIntervals = 200000000ull;

// Sizes every workspace buffer for a run of n query intervals, `rows` output rows and nblk input
// blocks.  With plan != nullptr nothing is allocated: *plan receives the bytes that growing the
// buffers would add (a buffer grows by freeing and reallocating it at the larger size).
int size_workspace(rgl_context* c, uint64_t n, uint32_t rows, uint32_t nblk, uint64_t* plan) {
    rgl_index* idx = c->idx;
    if (n > kMaxRunIntervals) return fail(RGL_ERR_INVALID_ARGUMENT, "at most 200,000,000 query intervals per run");
    const uint64_t ns = std::max<uint32_t>(idx->num_slots, 1);
    const uint64_t tot = n * ns;
    if (plan) *plan = 0;
    if (c->ws_ready && n <= c->res_n && rows <= c->res_rows && nblk <= c->res_blk) return RGL_OK;  // nothing grows
    struct Sizer {
        uint64_t* plan;
        int ensure_in(DevBuf& b, size_t bytes) {
            if (!plan) return b.ensure(bytes);
            if (bytes > b.cap) *plan += bytes - b.cap;
            return RGL_OK;
        }
    } z{plan};
    RGL_TRY(z.ensure_in(c->iv, n * sizeof(rgl_interval) + (nblk + 1ull) * 32 + 64));  // and the block tables
    RGL_TRY(z.ensure_in(c->blk_off, (nblk + 1) * 8ull));
    RGL_TRY(z.ensure_in(c->blk_shard, (nblk + 1) * 4ull));
    RGL_TRY(z.ensure_in(c->sortplan, (4ull * nblk + 8) * 4));
    // the block tables of a run with rows taken from the blocks (offsets, the sort's segment-order
    // offsets and destinations; shards, rows, ranks), sized here so that no run reallocates them
    RGL_TRY(z.ensure_in(c->bt_off, 3ull * (nblk + 1) * 8 + 8));
    RGL_TRY(z.ensure_in(c->bt_shard, 3ull * (nblk + 1) * 4 + 4));
    // and of the single-call entry points, whose blocks of several rows are sorted block by block too
    RGL_TRY(z.ensure_in(c->sort_tab, 2ull * (nblk + 1) * 8));
    RGL_TRY(z.ensure_in(c->sort_rank, (nblk + 1) * 4ull));
    RGL_TRY(z.ensure_in(c->key_a, n * 8 + 8));
    RGL_TRY(z.ensure_in(c->key_b, n * 8 + 8));
    RGL_TRY(z.ensure_in(c->val_a, n * 4 + 4));
    RGL_TRY(z.ensure_in(c->val_b, n * 4 + 4));
    RGL_TRY(z.ensure_in(c->ekey_a, n * 8 + 8));
    RGL_TRY(z.ensure_in(c->ekey_b, n * 8 + 8));
    RGL_TRY(z.ensure_in(c->starts, n * 4 + 4));
    RGL_TRY(z.ensure_in(c->ends, n * 4 + 4));
    RGL_TRY(z.ensure_in(c->shard, n * 4 + 4));
    RGL_TRY(z.ensure_in(c->row, n * 4 + 4));
    RGL_TRY(z.ensure_in(c->segnum, n * 4 + 4));
    RGL_TRY(z.ensure_in(c->seg_begin, n * 4 + 4));
    RGL_TRY(z.ensure_in(c->seg_need, n * 8 + 8));
    RGL_TRY(z.ensure_in(c->ps, n * 8 + 16));
    RGL_TRY(z.ensure_in(c->pe, n * 8 + 16));
    const uint64_t tiled = tot + ns * kTileThreads;  // entries of whole tiles
    RGL_TRY(z.ensure_in(c->lo, tiled * 4));
    RGL_TRY(z.ensure_in(c->cnt, tiled * 4));
    RGL_TRY(z.ensure_in(c->place, tiled * 2));
    RGL_TRY(z.ensure_in(c->rlo, tot * 4 + 4));
    RGL_TRY(z.ensure_in(c->ranges, (tot / 2 + 2) * sizeof(RangeDesc)));  // a range swept by ranks has two runs or more
    RGL_TRY(z.ensure_in(c->rpos, (tot / 2 + 2) * 8));
    RGL_TRY(z.ensure_in(c->small, 256));
    RGL_TRY(z.ensure_in(c->item_r0, kItemCap * 4));
    RGL_TRY(z.ensure_in(c->item_t0, kItemCap * 4));
    RGL_TRY(z.ensure_in(c->emax, n * 4 + 4));
    RGL_TRY(z.ensure_in(c->pc, tot * 8 + 16));
    RGL_TRY(z.ensure_in(c->cr, tot * 4 + 4));
    RGL_TRY(z.ensure_in(c->uhi, tot * 4 + 4));
    RGL_TRY(z.ensure_in(c->rt, tot * 8 + 8));
    RGL_TRY(z.ensure_in(c->ulen, tot * 4 + 4));
    RGL_TRY(z.ensure_in(c->rpair, tot * 8 + 8));
    RGL_TRY(z.ensure_in(c->sums, (tot / kTileThreads + tot / kTileThreads / kGroup + 3 * ns + n / kQTile + 8) * sizeof(RSum)));
    RGL_TRY(z.ensure_in(c->esums, (n / kQTile + n / kQTile / kGroup + 4) * sizeof(ESum)));
    RGL_TRY(z.ensure_in(c->ppos, tot * 8 + 16));
    RGL_TRY(z.ensure_in(c->psegs, tot * sizeof(PairSeg) + sizeof(PairSeg)));
    RGL_TRY(z.ensure_in(c->prow, tot * 4 + 4));
    RGL_TRY(z.ensure_in(c->segtab, (n + 1) * sizeof(SegTab)));
    RGL_TRY(z.ensure_in(c->tab2, (10 * n + 18) * 8));
    RGL_TRY(z.ensure_in(c->acc, 64));
    // CUB temporary storage: the maximum over every primitive used, at these sizes.
    size_t need = 0, b = 0;
    int nn = (int)std::max<uint64_t>(n, 1);
    cub::DeviceRadixSort::SortPairs(nullptr, b, (uint64_t*)nullptr, (uint64_t*)nullptr, (uint32_t*)nullptr,
                                    (uint32_t*)nullptr, nn, 0, 64, c->stream);
    need = std::max(need, b);
    cub::DeviceRadixSort::SortKeys(nullptr, b, (uint64_t*)nullptr, (uint64_t*)nullptr, nn, 0, 64, c->stream);
    need = std::max(need, b);
    cub::DeviceScan::ExclusiveSum(nullptr, b, (uint64_t*)nullptr, (uint64_t*)nullptr, nn + 1, c->stream);
    need = std::max(need, b);
    RGL_TRY(z.ensure_in(c->cub_tmp, need + 256));
    RGL_TRY(z.ensure_in(c->cub_tmp2, need + 256));
    if (rows) {
        RGL_TRY(z.ensure_in(c->out_counts, (uint64_t)rows * idx->num_sources * 4 + 16));
        RGL_TRY(z.ensure_in(c->out_bp, (uint64_t)rows * idx->num_sources * 12 + 32));  // both, see HostIO
    }
    if (plan) return RGL_OK;
    c->res_n = std::max(c->res_n, n);
    c->res_rows = std::max(c->res_rows, rows);
    c->res_blk = std::max(c->res_blk, nblk);
    c->ws_ready = true;
    uint64_t sig = 1469598103934665603ull;
    for (DevBuf* b : {&c->iv, &c->key_a, &c->key_b, &c->val_a, &c->val_b, &c->ekey_a, &c->ekey_b, &c->starts,
                      &c->ends, &c->shard, &c->row, &c->segnum, &c->seg_begin, &c->ps, &c->pe, &c->emax, &c->lo, &c->cnt,
                      &c->place, &c->rlo, &c->ranges, &c->rpos, &c->cub_tmp, &c->small, &c->item_r0, &c->item_t0, &c->segtab,
                      &c->tab2, &c->pc, &c->cr, &c->uhi, &c->rt, &c->ulen, &c->rpair, &c->sums, &c->esums, &c->ppos,
                      &c->psegs, &c->prow, &c->seg_need, &c->acc, &c->cub_tmp2, &c->sortplan})
        sig = (sig ^ (uint64_t)(uintptr_t)b->p ^ ((uint64_t)b->cap << 17)) * 1099511628211ull;
    c->ws_sig = sig;
    return RGL_OK;
}

int ensure_workspace(rgl_context* c, uint64_t n, uint32_t rows, uint32_t nblk) {
    return size_workspace(c, n, rows, nblk, nullptr);
}

inline unsigned grid_for(uint64_t n, unsigned block) { return (unsigned)((n + block - 1) / block); }

struct Launch {
    uint32_t chunk, ctas_per_sm, block, pair_ratio;
    uint32_t spread;  // see item_size; set per run unless the caller chose the work-item size
};

Launch pick_launch(const rgl_query_opts* o) {
    Launch l{1024, 8, 256, 4, 0};
    if (o) {
        if (o->chunk) l.chunk = o->chunk;
        if (o->ctas_per_sm) l.ctas_per_sm = o->ctas_per_sm;
        if (o->block) l.block = 256;  // the kernel is compiled for 256 threads
        if (o->pair_ratio) l.pair_ratio = o->pair_ratio;
    }
    l.chunk = (l.chunk + 31) & ~31u;  // keep warps whole
    if (l.chunk < 32) l.chunk = 32;
    if (l.ctas_per_sm < 1) l.ctas_per_sm = 1;
    if (l.ctas_per_sm > 8) l.ctas_per_sm = 8;
    return l;
}

int timing_record(rgl_context* c, bool start) {
    if (start) {
        while (c->tev.size() < 2 * (c->tev_used + 1)) {
            cudaEvent_t e;
            RGL_CUDA(cudaEventCreate(&e));
            c->tev.push_back(e);
        }
        RGL_CUDA(cudaEventRecord(c->tev[2 * c->tev_used], c->stream));
    } else {
        RGL_CUDA(cudaEventRecord(c->tev[2 * c->tev_used + 1], c->stream));
        c->tev_used++;
    }
    return RGL_OK;
}

// After the stream has been synchronised: error bits and stats of the last launch.
int finish(rgl_context* c, const Launch& L, rgl_query_stats* stats) {
    if (stats) {
        float t_sweep = 0, t_all = 0;
        if (c->last_n) {  // the events are recorded only when the pipeline ran
            RGL_CUDA(cudaEventElapsedTime(&t_sweep, c->ev[1], c->ev[2]));
            RGL_CUDA(cudaEventElapsedTime(&t_all, c->ev[0], c->ev[2]));
        }
        stats->query_intervals = c->last_n;
        // the pipeline's device counters (small[4..5] union, [9] ranges, [10..11] / [12..13] rank /
        // pair work) were copied to h_small after the run
        stats->ranges = c->last_n ? c->h_small[9] : 0;
        uint64_t T = 0;
        if (c->last_n) std::memcpy(&T, c->h_small + 4, 8);
        stats->db_swept = T;
        uint64_t TR = 0, TP = 0;
        if (c->last_n) {
            std::memcpy(&TR, c->h_small + 10, 8);
            std::memcpy(&TP, c->h_small + 12, 8);
        }
        stats->rank_positions = TR;
        stats->pair_candidates = TP;
        const uint32_t rc = item_size(TR, c->last_chunk, c->last_spread);
        const uint32_t pc = item_size(TP, c->last_chunk, c->last_spread);
        stats->work_items = (TR + rc - 1) / rc + (TP + pc - 1) / pc;
        stats->sweep_ms = c->last_n ? t_sweep : 0.f;
        stats->device_ms = c->last_n ? t_all : 0.f;
        stats->chunk = L.chunk;
        stats->ctas_per_sm = L.ctas_per_sm;
        stats->block = L.block;
        stats->kernel_launches = c->last_launches;
    }
    if (c->h_small[0] & ERR_BAD_INTERVAL) return fail(RGL_ERR_INVALID_ARGUMENT, "a query interval has start >= end");
    if (c->h_small[0] & ERR_BAD_ROW) return fail(RGL_ERR_INVALID_ARGUMENT, "a query interval's sid >= num_rows");
    return RGL_OK;
}

// Tile summaries into exclusive prefixes (nt tiles, or those of *count elements), by groups of kGroup.
template <class T>
void scan_groups(T* sums, uint32_t nt, const uint32_t* count, uint32_t tile, T* groups, uint32_t ng, cudaStream_t st,
                 T* total = nullptr) {
    k_group_sums<T><<<ng, kTileThreads, 0, st>>>(sums, nt, count, tile, groups);
    k_group_scan<T><<<ng, kTileThreads, 0, st>>>(sums, nt, count, tile, groups, total);
}

// `to` waits for everything enqueued on `from` so far.
int stream_after(cudaStream_t to, cudaStream_t from, cudaEvent_t e) {
    RGL_CUDA(cudaEventRecord(e, from));
    RGL_CUDA(cudaStreamWaitEvent(to, e, 0));
    return RGL_OK;
}

// Shape of a run's block-local key sort, from the host's block offsets.
struct LocalSort {
    bool wide = false;       // blocks of several rows (one per shard): sorted by the whole key
    uint64_t max_block = 0;  // the largest block: sets the number of merge passes
    uint64_t tiles = 0;      // tiles of kBlockSortCap intervals over all blocks
    uint64_t chunks = 0;     // merge chunks of the blocks of more than one tile
    // When the blocks are not in segment order (file-major blocks of several rows), the sorted keys
    // are laid out segment by segment, as a device-wide sort would lay them out, so that the sweeps
    // take every row's work on one chromosome together: block b's keys go to [dst[b], dst[b] +
    // cnt_b), its rank in segment order is idx[b], and soff (nblk + 1) are the offsets of the blocks
    // in that order.  Empty: the blocks are in segment order already.
    std::vector<uint64_t> soff, dst;
    std::vector<uint32_t> idx;
};

// Input of one pipeline run: n intervals at `iv` (device), block b = [blk_off[b], blk_off[b+1]) on
// shard blk_shard[b] (both tables on the device), rows [row_base, row_base + rows) of the output.
struct PipeIn {
    const rgl_interval* iv;
    uint64_t n;
    uint32_t rows, row_base, nblk;
    const uint64_t* blk_off;
    const uint32_t* blk_shard;
    const uint32_t* blk_row;  // optional: the row every interval of the block must carry
    int row_from_block = 0;   // 1: rows come from blk_row, interval sids are ignored
    int block_local = 0;      // 1: one segment per block, no segment in two blocks (block-local key sort)
    LocalSort ls;             // with block_local: the sort's tile and merge-chunk counts
    // with block_local and a segment-order layout: device copies of ls.soff, ls.dst, ls.idx
    const uint64_t* sort_off = nullptr;
    const uint64_t* sort_dst = nullptr;
    const uint32_t* sort_idx = nullptr;
    uint32_t region_bits = 0; // > 0: segments are (shard, 2^region_bits-bp region of the start, row)
};

// Whether a run's blocks allow the block-local key sort: with one row, or rows taken from the
// blocks, every block is one segment, and they must be distinct; blocks of several rows hold the
// segments of one shard, and the shards must be distinct (a wide sort: 37 rows in 24 blocks of sorted
// files took two device-wide radix sorts, 12 passes of 9 us).  off: nblk + 1 host offsets; row:
// the blocks' rows (null: from the intervals).  *ls receives the shape of the sort.
bool blocks_local(uint32_t nblk, const uint64_t* off, const uint32_t* shard, const uint32_t* row, uint32_t rows,
                  uint32_t row_base, LocalSort* ls) {
    *ls = LocalSort();
    std::vector<std::pair<uint64_t, uint32_t>> segs;  // (segment, block) of the non-empty blocks
    segs.reserve(nblk);
    LocalSort t;
    t.wide = !row && rows != 1;
    bool ordered = true;
    for (uint32_t b = 0; b < nblk; b++) {
        const uint64_t cnt = off[b + 1] - off[b];
        t.max_block = std::max(t.max_block, cnt);
        t.tiles += sort_tiles(cnt);
        t.chunks += merge_chunks(cnt);
        const uint64_t sg = (uint64_t)shard[b] * rows + (row ? row[b] - row_base : 0u);
        if (cnt) {
            if (!segs.empty() && sg < segs.back().first) ordered = false;
            segs.push_back({sg, b});
        }
    }
    std::vector<std::pair<uint64_t, uint32_t>> sorted(segs);
    std::stable_sort(sorted.begin(), sorted.end(),
                     [](const std::pair<uint64_t, uint32_t>& a, const std::pair<uint64_t, uint32_t>& b) {
                         return a.first < b.first;
                     });
    for (size_t k = 1; k < sorted.size(); k++)
        if (sorted[k].first == sorted[k - 1].first) return false;  // a segment in two blocks
    if (!ordered) {
        // empty blocks keep their place in the order (rank) and take no room
        std::vector<uint32_t> order;
        order.reserve(nblk);
        size_t k = 0;
        for (uint32_t b = 0; b < nblk; b++)
            if (off[b + 1] == off[b]) order.push_back(b);
        std::vector<uint32_t> empties(order);
        order.clear();
        for (const auto& e : sorted) order.push_back(e.second);
        order.insert(order.end(), empties.begin(), empties.end());
        t.soff.assign(nblk + 1, 0);
        t.dst.assign(nblk + 1, 0);
        t.idx.assign(nblk + 1, 0);
        uint64_t at = 0;
        for (k = 0; k < order.size(); k++) {
            const uint32_t b = order[k];
            t.soff[k] = at;
            t.dst[b] = at;
            t.idx[b] = (uint32_t)k;
            at += off[b + 1] - off[b];
        }
        t.soff[nblk] = at;
        t.dst[nblk] = at;
    }
    *ls = std::move(t);
    return true;
}

// What a run does besides the sweep: the single-call entry points zero their rows, reset the error
// word and record stats events; the sub-batches of a batched call leave all of that to the caller
// and add their stats into a device accumulator.
struct PipeMode {
    bool zero_out = true;
    bool reset_err = true;
    bool events = true;  // stats events and sweep timing (off inside a graph capture)
    bool no_sweep = false;  // stop once the pair work space (ppos, psegs) is laid out
    unsigned long long* acc = nullptr;
};

__global__ void k_acc_stats(unsigned long long* acc, const uint32_t* ranges, const unsigned long long* uni,
                            const unsigned long long* rank_pos, const unsigned long long* pair_cand, uint32_t n) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        acc[0] += *ranges;
        acc[1] += *uni;
        acc[2] += *rank_pos;
        acc[3] += *pair_cand;
        acc[4] += n;
    }
}

// Runs steps 1-5 of the pipeline on the context stream, with no host synchronisation.
int run_pipeline(rgl_context* c, const PipeIn& in, const rgl_query_opts* opts, uint32_t* d_counts,
                 unsigned long long* d_bp, rgl_query_stats* stats, const PipeMode& mode = PipeMode()) {
    rgl_index* idx = c->idx;
    cudaStream_t st = c->stream;
    const uint32_t D = idx->num_sources;
    const uint32_t ns = idx->num_slots;
    const uint32_t n = (uint32_t)in.n;
    const uint32_t rows = in.rows;
    Launch L = pick_launch(opts);
    // several rows: the block items flush their row histogram, so larger work items pay (measured
    // on the 2e9-interval database: 1024 -> 8192 positions, sweeps 3.45 -> 2.46 s per 4,096 files)
    if (rows > 1 && !(opts && opts->chunk)) L.chunk = kMultiRowChunk;
    // four work items for every warp of the sweeps' grid, unless the caller set the items' size
    if (!(opts && opts->chunk)) L.spread = (uint32_t)c->num_sms * L.ctas_per_sm * kCtaItems * 4;
    const bool with_bp = d_bp != nullptr && !(opts && (opts->flags & RGL_QF_NO_OVERLAP));
    const bool ev = mode.events && stats;
    const bool pdl = in.n <= kPdlMaxIntervals;
    // a caller's pair ratio is taken alone
    const uint32_t run_cost = (opts && opts->pair_ratio) ? 0u : kRankRunCost;

    uint32_t* d_small = c->small.as<uint32_t>();  // [0] error bits, [1] queue, [2..] scratch
    ClearList clear{};
    auto to_clear = [&](void* p, uint64_t words) {
        if (p && words) {
            clear.p[clear.count] = static_cast<uint32_t*>(p);
            clear.words[clear.count++] = words;
        }
    };
    auto run_clear = [&] {
        uint64_t most = 0;
        for (int r = 0; r < clear.count; r++) most = std::max(most, clear.words[r]);
        k_clear<<<(unsigned)std::min<uint64_t>(grid_for(most, 256), (uint64_t)c->num_sms * 16), 256, 0, st>>>(clear);
    };
    if (mode.reset_err) to_clear(d_small, 16);
    else to_clear(d_small + 1, 15);
    if (mode.zero_out) {
        to_clear(d_counts, (uint64_t)rows * D);
        to_clear(d_bp, (uint64_t)rows * D * 2);
    }
    if (n == 0 || ns == 0) {
        run_clear();
        c->last_n = 0;
        c->last_tot = 0;
        c->last_launches = 0;
        if (stats) std::memset(stats, 0, sizeof(*stats));
        if (mode.reset_err) RGL_CUDA(cudaMemcpyAsync(c->h_small, d_small, 4, cudaMemcpyDeviceToHost, st));
        return RGL_OK;
    }
    if (!rows) return fail(RGL_ERR_INVALID_ARGUMENT, "a query interval's sid >= num_rows");
    // key width: segment = shard * rows + row
    const uint32_t rb = in.region_bits;
    if (rb && (rb < 16 || rb > 31)) return fail(RGL_ERR_INVALID_ARGUMENT, "region bits must be in [16, 31]");
    const uint64_t nreg = rb ? (1ull << (32 - rb)) : 1ull;
    uint64_t nseg = (uint64_t)idx->num_shards * nreg * rows;
    int segbits = 1;
    while (segbits < 32 && (1ull << segbits) < nseg) segbits++;
    if (nseg >= (1ull << 32))
        return fail(RGL_ERR_INVALID_ARGUMENT, "num_shards x regions x num_rows must be < 2^32");
    const uint32_t sps = (uint32_t)(nreg * rows);  // segments per shard

    // tally: one row in a block-wide histogram for the whole kernel (1); several rows in a histogram
    // of each block item's row (2); else (or with RGL_QF_GLOBAL_TALLY) atomics on the outputs (0)
    size_t smem = (size_t)D * (with_bp ? 12 : 4);
    const int tally = smem > 160 * 1024 ? 0 : rows == 1 ? 1
                      : (opts && (opts->flags & RGL_QF_GLOBAL_TALLY)) || rows > kMaxPackedRows ? 0 : 2;

    if (ev) RGL_CUDA(cudaEventRecord(c->ev[0], st));
    // Two streams: `st` carries the chain from the sorted starts to the sweeps, `sd` the chains that
    // only the rank sweep needs (the end-key sort and unpack, the prefix sums of starts and ends,
    // the rank tables), so that the small kernels of both overlap; `sd` is joined back before the
    // sweeps.
    cudaStream_t sd = c->side;
    uint32_t launches = 0;
    // block-local sort with a segment-order layout: callers that did not upload its tables (the
    // single-call entry points, never inside a graph capture) have them uploaded here
    const uint64_t* sort_off = in.sort_off;
    const uint64_t* sort_dst = in.sort_dst;
    const uint32_t* sort_idx = in.sort_idx;
    if (in.block_local && !in.ls.dst.empty() && !sort_dst) {
        const uint64_t nb1 = (uint64_t)in.nblk + 1;
        RGL_TRY(c->sort_tab.ensure(2 * nb1 * 8));
        RGL_TRY(c->sort_rank.ensure(nb1 * 4));
        RGL_CUDA(cudaMemcpyAsync(c->sort_tab.p, in.ls.soff.data(), nb1 * 8, cudaMemcpyHostToDevice, st));
        RGL_CUDA(cudaMemcpyAsync(c->sort_tab.as<uint64_t>() + nb1, in.ls.dst.data(), nb1 * 8, cudaMemcpyHostToDevice,
                                 st));
        RGL_CUDA(cudaMemcpyAsync(c->sort_rank.p, in.ls.idx.data(), nb1 * 4, cudaMemcpyHostToDevice, st));
        sort_off = c->sort_tab.as<uint64_t>();
        sort_dst = sort_off + nb1;
        sort_idx = c->sort_rank.as<uint32_t>();
    }
    // block-local sort: per-block order flags ([0, nblk) starts, [nblk, 2 nblk) ends), the two sorts'
    // pass words, then the tile and merge-chunk prefix counts
    uint32_t* d_unsorted = c->sortplan.as<uint32_t>();
    uint32_t* d_maxp = d_unsorted + 2ull * in.nblk;
    uint32_t* d_tile_pre = d_maxp + 2;
    uint32_t* d_chunk_pre = d_tile_pre + in.nblk + 1;
    if (in.block_local) to_clear(d_unsorted, 2ull * in.nblk + 2);
    const uint32_t max_segs = (uint32_t)std::min<uint64_t>(n, nseg);
    to_clear(c->seg_need.p, 2ull * max_segs);
    run_clear();
    (void)launch_chain(pdl, k_expand_keys<true>, k_expand_keys<false>, grid_for(n, 256), 256, 0, st, n, in.iv,
                       in.blk_off, in.blk_shard, in.blk_row, in.row_from_block, in.nblk, rows, in.row_base, rb,
                       c->key_a.as<uint64_t>(), c->val_a.as<uint32_t>(), c->ekey_a.as<uint64_t>(), d_small,
                       in.block_local ? d_unsorted : nullptr, in.block_local ? sort_dst : nullptr,
                       in.block_local ? sort_idx : nullptr, (int)(in.block_local && in.ls.wide));
    launches += 2;
    // the sort's view of the blocks: their offsets in the layout the keys were written in
    const uint64_t* soff = sort_dst ? sort_off : in.blk_off;
    const uint32_t passes = in.block_local ? sort_passes(in.ls.max_block) : 0u;
    if (in.block_local)  // the plan (before the fork), then the end keys here and the start keys there
        launches += block_sort_enqueue(in.nblk, soff, 0, 0, 0, d_tile_pre, d_chunk_pre, nullptr, nullptr, nullptr,
                                       nullptr, nullptr, nullptr, st, true, pdl);
    RGL_TRY(stream_after(sd, st, c->ev_fork));
    size_t tb = c->cub_tmp2.cap;
    // the end keys: on the side stream at once; or, in large runs whose blocks are segments, once it is
    // known which of them a rank sweep needs (the sort, sums and tables of 3.1e7 ends were 1.6 of 8.9 ms
    // of a batch against a small database that hardly any range sweeps by ranks)
    const bool late_ends = in.block_local && !in.ls.wide && !pdl;
    auto sort_ends = [&] {
        launches += block_sort_enqueue(in.nblk, soff, in.ls.tiles, in.ls.chunks, passes, d_tile_pre, d_chunk_pre,
                                       d_unsorted + in.nblk, c->ekey_a.as<uint64_t>(), nullptr,
                                       c->ekey_b.as<uint64_t>(), nullptr, d_maxp + 1, sd, false, pdl, in.ls.wide);
    };
    if (in.block_local) {
        if (!late_ends) sort_ends();
        launches += block_sort_enqueue(in.nblk, soff, in.ls.tiles, in.ls.chunks, passes, d_tile_pre, d_chunk_pre,
                                       d_unsorted, c->key_a.as<uint64_t>(), c->val_a.as<uint32_t>(),
                                       c->key_b.as<uint64_t>(), c->val_b.as<uint32_t>(), d_maxp, st, false, pdl,
                                       in.ls.wide);
    } else {
        RGL_CUDA(cub::DeviceRadixSort::SortKeys(c->cub_tmp2.p, tb, c->ekey_a.as<uint64_t>(), c->ekey_b.as<uint64_t>(),
                                                (int)n, 0, 32 + segbits, sd));
        tb = c->cub_tmp.cap;
        RGL_CUDA(cub::DeviceRadixSort::SortPairs(c->cub_tmp.p, tb, c->key_a.as<uint64_t>(), c->key_b.as<uint64_t>(),
                                                 c->val_a.as<uint32_t>(), c->val_b.as<uint32_t>(), (int)n, 0,
                                                 32 + segbits, st));
    }
    // the side stream goes on with the ends (their prefix sums), the main one with the starts
    const uint64_t tot = (uint64_t)n * ns;
    if (tot + 1 >= (1ull << 31)) {
        RGL_TRY(stream_after(st, sd, c->ev_join));
        return fail(RGL_ERR_INVALID_ARGUMENT, "query intervals x layer slots must be < 2^31 per run");
    }
    const uint32_t qt = (n + kQTile - 1) / kQTile;
    const uint32_t qg = qt > kMaxLook ? (qt + kGroup - 1) / kGroup : 0u;  // groups of tiles, if any
    ESum* eg = qg ? c->esums.as<ESum>() + qt : nullptr;
    QSum* qgs = qg ? c->sums.as<QSum>() + qt : nullptr;
    auto sum_ends = [&] {
        (void)launch_chain(pdl, k_e_reduce<true>, k_e_reduce<false>, qt, kTileThreads, 0, sd, n,
                           c->ekey_b.as<uint64_t>(), c->esums.as<ESum>());
        if (qg) scan_groups(c->esums.as<ESum>(), qt, nullptr, 0, eg, qg, sd);
        (void)launch_chain(pdl, k_e_apply<true>, k_e_apply<false>, qt, kTileThreads, 0, sd, n, c->ekey_b.as<uint64_t>(),
                           c->esums.as<ESum>(), (int)(qg != 0), c->ends.as<uint32_t>(), c->pe.as<uint64_t>());
        launches += qg ? 4 : 2;
    };
    if (!late_ends) sum_ends();
    (void)launch_chain(pdl, k_q_reduce<true>, k_q_reduce<false>, qt, kTileThreads, 0, st, n,
                       c->key_b.as<uint64_t>(), c->val_b.as<uint32_t>(), c->sums.as<QSum>());
    if (qg) scan_groups(c->sums.as<QSum>(), qt, nullptr, 0, qgs, qg, st);
    (void)launch_chain(pdl, k_q_apply<true>, k_q_apply<false>, qt, kTileThreads, 0, st, n, rows, sps,
                       c->key_b.as<uint64_t>(), c->val_b.as<uint32_t>(), c->sums.as<QSum>(), (int)(qg != 0),
                       c->starts.as<uint32_t>(), c->shard.as<uint32_t>(), c->row.as<uint32_t>(),
                       c->segnum.as<uint32_t>(), c->seg_begin.as<uint32_t>(),
                       c->ps.as<uint64_t>(), c->emax.as<uint32_t>());
    launches += qg ? 4 : 2;
    uint32_t* Lp = d_small + 8;   // live runs L
    uint32_t* Rp = d_small + 9;   // ranges R
    uint32_t* RRp = d_small + 14;  // ranges swept by ranks
    // partition points, live runs and ranges
    const dim3 lgrid(grid_for(n, kTileThreads), ns);
    const uint32_t lt = lgrid.x * ns, lg = lt > kMaxLook ? (lt + kGroup - 1) / kGroup : 0u;
    LSum* lsums = c->sums.as<LSum>();
    LSum* lgs = lg ? lsums + lt + 1 : nullptr;  // (the whole at lsums[lt])
    (void)launch_chain(pdl, k_lohi<true>, k_lohi<false>, lgrid, kTileThreads, 0, st, n, ns, c->starts.as<uint32_t>(),
                       c->val_b.as<uint32_t>(), c->emax.as<uint32_t>(), c->shard.as<uint32_t>(), idx->d_lq,
                       idx->d_pos, idx->d_btab, c->lo.as<uint32_t>(), c->cnt.as<uint32_t>(),
                       c->place.as<uint16_t>(), lsums);
    if (lg) scan_groups(lsums, lt, nullptr, 0, lgs, lg, st, lsums + lt);
    const int tag = mode.no_sweep ? RUN_SHARD_ROW : tally == 2 ? RUN_PACKED : rows > 1 ? RUN_ROW : RUN_PLAIN;
    (void)launch_chain(pdl, k_emit<true>, k_emit<false>, grid_for(lt, kTileThreads / 32), kTileThreads, 0, st, n, ns,
                       rows, lgrid.x, lt, tag, c->starts.as<uint32_t>(), c->val_b.as<uint32_t>(),
                       c->emax.as<uint32_t>(), c->shard.as<uint32_t>(), c->row.as<uint32_t>(), idx->d_lq,
                       idx->d_pos, idx->d_btab, c->lo.as<uint32_t>(), c->cnt.as<uint32_t>(), c->place.as<uint16_t>(),
                       lsums, (int)(lg != 0), c->psegs.as<PairSeg>(),
                       c->prow.as<uint32_t>(), c->pc.as<uint64_t>(), c->cr.as<uint32_t>(), c->uhi.as<uint32_t>(),
                       c->rt.as<uint2>(), c->rlo.as<uint32_t>(), Lp, Rp);
    // the ranges' unions, methods and places; R is a device count, at most tot
    const unsigned rgrid = (unsigned)std::min<uint64_t>(tot / kRTile + 1, (uint64_t)c->num_sms * 16);
    RSum* rsums = c->sums.as<RSum>();
    const uint32_t rtl = (uint32_t)(tot / kRTile + 1), rg = rtl > kMaxLook ? (rtl + kGroup - 1) / kGroup : 0u;
    RSum* rgs = rg ? rsums + rtl : nullptr;
    (void)launch_chain(pdl, k_range_reduce<true>, k_range_reduce<false>, rgrid, kTileThreads, 0, st, Lp, Rp, n,
                       c->rt.as<uint2>(), c->pc.as<uint64_t>(), c->uhi.as<uint32_t>(), c->rlo.as<uint32_t>(),
                       c->segnum.as<uint32_t>(), L.pair_ratio, run_cost, c->ulen.as<uint32_t>(),
                       c->seg_need.as<unsigned long long>(), reinterpret_cast<unsigned long long*>(d_small + 4), rsums);
    launches += lg ? 5 : 3;
    // side stream: rank tables of the query segments that have a rank-difference range
    RGL_TRY(stream_after(sd, st, c->ev_fork));
    if (late_ends) {
        k_skip_ends<<<grid_for(in.nblk, 256), 256, 0, sd>>>(in.nblk, soff, c->segnum.as<uint32_t>(),
                                                            c->seg_need.as<unsigned long long>(),
                                                            d_unsorted + in.nblk);
        launches++;
        sort_ends();
        sum_ends();
    }
    k_seg_tabsize<<<grid_for(max_segs, 256), 256, 0, sd>>>(n, c->segnum.as<uint32_t>(), c->seg_begin.as<uint32_t>(),
                                                           c->seg_need.as<unsigned long long>(),
                                                           c->ends.as<uint32_t>(), c->segtab.as<SegTab>());
    (void)launch_chain(pdl, k_tab_fill<true>, k_tab_fill<false>, grid_for(n, 256), 256, 0, sd, n,
                     c->segnum.as<uint32_t>(), c->segtab.as<SegTab>(), c->starts.as<uint32_t>(),
                     c->ends.as<uint32_t>(), c->tab2.as<uint2>());
    launches += 2;
    // main stream: the two work spaces
    if (rg) scan_groups(rsums, 0, Rp, kRTile, rgs, rg, st);
    (void)launch_chain(pdl, k_range_apply<true>, k_range_apply<false>, rgrid, kTileThreads, 0, st, Lp, Rp, n, ns, rows,
                       c->rt.as<uint2>(), c->pc.as<uint64_t>(), c->ulen.as<uint32_t>(), c->rlo.as<uint32_t>(),
                       c->shard.as<uint32_t>(), c->row.as<uint32_t>(), c->segnum.as<uint32_t>(), idx->d_slot,
                       L.pair_ratio, run_cost, rsums, (int)(rg != 0),
                       c->ranges.as<RangeDesc>(), c->rpos.as<uint64_t>(), c->rpair.as<uint64_t>(),
                       c->ppos.as<uint64_t>(), RRp, reinterpret_cast<unsigned long long*>(d_small + 10));
    const unsigned gc = (unsigned)std::min<uint64_t>(grid_for(tot, 256), (uint64_t)c->num_sms * 32);
    (void)launch_chain(pdl, k_run_pos<true>, k_run_pos<false>, gc, 256, 0, st, Lp, c->cr.as<uint32_t>(),
                       c->pc.as<uint64_t>(), c->rpair.as<uint64_t>(), c->ppos.as<uint64_t>());
    launches += rg ? 4 : 2;
    if (mode.no_sweep) {
        RGL_TRY(stream_after(st, sd, c->ev_join));
        c->last_tot = tot;
        c->last_launches = launches;
        c->last_n = n;
        if (mode.reset_err) RGL_CUDA(cudaMemcpyAsync(c->h_small, d_small, 4, cudaMemcpyDeviceToHost, st));
        return RGL_OK;
    }
    (void)launch_chain(pdl, k_item_ranges<true>, k_item_ranges<false>, (unsigned)(c->num_sms * 8), 256, 0, st,
                     RRp, c->rpos.as<uint64_t>(), Lp, c->ppos.as<uint64_t>(), L.chunk, L.spread, kItemCap,
                     c->item_r0.as<uint32_t>(), c->item_t0.as<uint32_t>());
    launches++;
    SweepParams P;
    P.item_r0 = c->item_r0.as<uint32_t>();
    P.item_t0 = c->item_t0.as<uint32_t>();
    P.ppos = c->ppos.as<uint64_t>();
    P.psegs = c->psegs.as<PairSeg>();
    P.prow = c->prow.as<uint32_t>();
    P.segtabs = c->segtab.as<SegTab>();
    P.tab2 = c->tab2.as<uint2>();
    P.item_cap = kItemCap;
    P.rpos = c->rpos.as<uint64_t>();
    P.rcount = RRp;
    P.pcount = Lp;
    P.ranges = c->ranges.as<RangeDesc>();
    P.layers = idx->d_layers;
    P.pos = idx->d_pos;
    P.sid = idx->d_sid;
    P.starts = c->starts.as<uint32_t>();
    P.ends = c->ends.as<uint32_t>();
    P.ps = c->ps.as<uint64_t>();
    P.pe = c->pe.as<uint64_t>();
    P.counts = d_counts;
    P.bp = with_bp ? d_bp : nullptr;
    P.queue = d_small + 1;
    P.rows = rows;
    P.D = D;
    P.chunk = L.chunk;
    P.spread = L.spread;
    c->last_chunk = L.chunk;
    c->last_spread = L.spread;
    P.smem_tally = tally;
    if (!tally) smem = 0;
    unsigned grid = (unsigned)(c->num_sms * L.ctas_per_sm);
    // the rank tables are joined before the sweeps; the two sweeps run one after the other on
    // `st` (each fills every SM with persistent blocks; run side by side they were slower)
    RGL_TRY(stream_after(st, sd, c->ev_join));
    if (ev) RGL_CUDA(cudaEventRecord(c->ev[1], st));
    if (c->timing && mode.events) RGL_TRY(timing_record(c, true));
    if (P.smem_tally == 2) {
        if (with_bp) k_sweep<true, true><<<grid, 256, smem, st>>>(P);
        else k_sweep<false, true><<<grid, 256, smem, st>>>(P);
    } else {
        if (with_bp) k_sweep<true, false><<<grid, 256, smem, st>>>(P);
        else k_sweep<false, false><<<grid, 256, smem, st>>>(P);
    }
    P.queue = d_small + 2;  // the pair sweep pulls from its own counter
    if (P.smem_tally == 2) {
        if (with_bp) k_pairs<true, true, 1><<<grid, 256, smem, st>>>(P);
        else k_pairs<false, true, 1><<<grid, 256, smem, st>>>(P);
    } else if (P.smem_tally) {
        if (with_bp) k_pairs<true, true, 0><<<grid, 256, smem, st>>>(P);
        else k_pairs<false, true, 0><<<grid, 256, smem, st>>>(P);
    } else {
        if (with_bp) k_pairs<true, false, 0><<<grid, 256, smem, st>>>(P);
        else k_pairs<false, false, 0><<<grid, 256, smem, st>>>(P);
    }
    launches++;
    launches++;
    RGL_CUDA(cudaGetLastError());
    if (c->timing && mode.events) RGL_TRY(timing_record(c, false));
    if (mode.acc) {
        k_acc_stats<<<1, 32, 0, st>>>(mode.acc, d_small + 9, reinterpret_cast<unsigned long long*>(d_small + 4),
                                      reinterpret_cast<unsigned long long*>(d_small + 10),
                                      reinterpret_cast<unsigned long long*>(d_small + 12), n);
        launches++;
    }
    c->last_tot = tot;
    c->last_launches = launches;
    c->last_n = n;
    if (ev) {
        RGL_CUDA(cudaEventRecord(c->ev[2], st));
        RGL_CUDA(cudaMemcpyAsync(c->h_small + 4, d_small + 4, 48, cudaMemcpyDeviceToHost, st));
    }
    if (mode.reset_err) RGL_CUDA(cudaMemcpyAsync(c->h_small, d_small, 4, cudaMemcpyDeviceToHost, st));
    return RGL_OK;
}

// Maps a batch's shards to index shard ids; shards absent from the index are skipped, as the
// reference skips shards not in meta.shards (src/tasks/query/mod.rs:194-196).
int resolve_blocks(rgl_context* c, const rgl_query_batch* b, std::vector<uint32_t>* shard_ids,
                   std::vector<const rgl_query_shard*>* blocks) {
    for (uint32_t i = 0; i < b->num_shards; i++) {
        const rgl_query_shard& s = b->shards[i];
        uint32_t id;
        if (s.shard_name) {
            auto it = c->idx->shard_ids.find(s.shard_name);
            if (it == c->idx->shard_ids.end()) continue;
            id = it->second;
        } else {
            id = s.shard_id;
            if (id >= c->idx->num_shards) continue;
        }
        if (s.count == 0) continue;
        if (!s.intervals) return fail(RGL_ERR_INVALID_ARGUMENT, "query shard without intervals");
        shard_ids->push_back(id);
        blocks->push_back(&s);
    }
    return RGL_OK;
}

// Page-locked staging per context, for inputs and outputs of the host entry points.
constexpr uint64_t kHostIoBytes = 512ull << 10;
// Blocks of less than this on average are staged.  24 copies of pageable memory took 3.2, 3.3, 4.0, 5.3, 6.0, 8.9, 13.8 us
// each at 0.5, 16, 32, 48, 64, 100, 200 KB; gathered into the buffer and sent as one, 20 us and 80 us per MB in all: 27, 46,
// 70, 101, 141, 207, 390 us against 77, 79, 97, 126, 144, 214, 332.
constexpr uint64_t kStagePerCopy = 48ull << 10;

// The run's input on the device: the blocks' host intervals at offsets off in the context's interval
// buffer, and after them the block tables (offsets, shards, and the sort's segment-order layout where it
// has one).  Short blocks are gathered into the staging buffer, tables included, and sent in one copy;
// longer ones are copied from where they lie, one copy per run of blocks that lie back to back in host
// memory (a file read into one buffer), and the tables in one.  (24 short blocks and their tables took
// 26 copies, 100 of the 200 us of a 1,000-interval call.)
int upload_blocks(rgl_context* c, const std::vector<const rgl_query_shard*>& blocks, const std::vector<uint64_t>& off,
                  const std::vector<uint32_t>& ids, PipeIn* in, cudaStream_t st) {
    const size_t nb = blocks.size(), nb1 = nb + 1;
    if (!nb) return RGL_OK;
    const bool layout = in->block_local && !in->ls.dst.empty();
    const uint64_t iv_bytes = off[nb] * sizeof(rgl_interval);
    const uint64_t at = (iv_bytes + 15) & ~15ull;  // the tables: off, soff, dst (8 bytes each), shards, idx
    const uint64_t tab_bytes = nb1 * (layout ? 32 : 12);
    size_t copies = 1;
    for (size_t i = 1; i < nb; i++)
        if (blocks[i]->intervals != blocks[i - 1]->intervals + blocks[i - 1]->count) copies++;
    RGL_TRY(c->iv.ensure(at + tab_bytes));
    unsigned char* dev = c->iv.as<unsigned char>();
    const bool stage = at + tab_bytes <= kHostIoBytes && iv_bytes <= copies * kStagePerCopy;
    std::vector<unsigned char> big;
    unsigned char* tab = c->h_io + (stage ? at : 0);
    if (!stage && tab_bytes > kHostIoBytes) {
        big.resize(tab_bytes);
        tab = big.data();
    }
    std::memcpy(tab, off.data(), nb1 * 8);
    if (layout) {
        std::memcpy(tab + nb1 * 8, in->ls.soff.data(), nb1 * 8);
        std::memcpy(tab + nb1 * 16, in->ls.dst.data(), nb1 * 8);
        std::memcpy(tab + nb1 * 28, in->ls.idx.data(), nb1 * 4);
    }
    std::memcpy(tab + nb1 * (layout ? 24 : 8), ids.data(), nb * 4);
    if (stage) {
        for (size_t i = 0; i < nb; i++)
            std::memcpy(c->h_io + off[i] * sizeof(rgl_interval), blocks[i]->intervals,
                        blocks[i]->count * sizeof(rgl_interval));
        RGL_CUDA(cudaMemcpyAsync(dev, c->h_io, at + tab_bytes, cudaMemcpyHostToDevice, st));
    } else {
        for (size_t i = 0; i < nb;) {
            size_t j = i + 1;
            while (j < nb && blocks[j]->intervals == blocks[j - 1]->intervals + blocks[j - 1]->count) j++;
            RGL_CUDA(cudaMemcpyAsync(dev + off[i] * sizeof(rgl_interval), blocks[i]->intervals,
                                     (off[j] - off[i]) * sizeof(rgl_interval), cudaMemcpyHostToDevice, st));
            i = j;
        }
        RGL_CUDA(cudaMemcpyAsync(dev + at, tab, tab_bytes, cudaMemcpyHostToDevice, st));
        if (!big.empty()) RGL_CUDA(cudaStreamSynchronize(st));
    }
    in->iv = reinterpret_cast<const rgl_interval*>(dev);
    in->blk_off = reinterpret_cast<const uint64_t*>(dev + at);
    in->blk_shard = reinterpret_cast<const uint32_t*>(dev + at + nb1 * (layout ? 24 : 8));
    if (layout) {
        in->sort_off = in->blk_off + nb1;
        in->sort_dst = in->blk_off + 2 * nb1;
        in->sort_idx = reinterpret_cast<const uint32_t*>(dev + at + nb1 * 28);
    }
    return RGL_OK;
}

// ---- batched form ------------------------------------------------------------------------------
// A batch is cut into sub-batches of at most `sub` intervals (cutting blocks where needed: counts and
// base pairs are sums over pairs, so a row split across sub-batches adds up to the same cells).
struct SubBatch {
    uint64_t begin, n;        // element range in d_intervals
    uint32_t row_lo, rows;    // output rows the sub-batch may touch
    uint32_t tab_at, nblk;    // its block table: entries [tab_at, tab_at + nblk] of the offsets, [tab_at, +nblk) of shards
};

struct BatchPlan {
    std::vector<SubBatch> subs;
    std::vector<uint64_t> off;   // per sub-batch: nblk + 1 offsets relative to its begin
    std::vector<uint32_t> shard; // per sub-batch: nblk shard ids (padded to the offsets' layout)
    std::vector<uint32_t> row;   // per sub-batch: nblk block rows (same layout; unused without block_rows)
    uint64_t max_n = 0;
    uint32_t max_rows = 0, max_blk = 0;
    // per sub-batch: whether the block-local key sort applies, and its shape
    std::vector<char> local;
    std::vector<LocalSort> ls;
    // the sorts' segment-order layouts, in the offsets' (soff, sdst) and shards' (sidx) layouts
    std::vector<uint64_t> soff, sdst;
    std::vector<uint32_t> sidx;
    void prepare(bool block_rows) {
        local.assign(subs.size(), 0);
        ls.assign(subs.size(), LocalSort());
        soff = off;
        sdst = off;
        sidx.assign(shard.size(), 0);
        for (size_t k = 0; k < subs.size(); k++) {
            const SubBatch& sb = subs[k];
            local[k] = blocks_local(sb.nblk, &off[sb.tab_at], &shard[sb.tab_at],
                                    block_rows ? &row[sb.tab_at] : nullptr, sb.rows, sb.row_lo, &ls[k]);
            if (!local[k] || ls[k].dst.empty()) continue;
            std::copy(ls[k].soff.begin(), ls[k].soff.end(), soff.begin() + sb.tab_at);
            std::copy(ls[k].dst.begin(), ls[k].dst.end(), sdst.begin() + sb.tab_at);
            std::copy(ls[k].idx.begin(), ls[k].idx.end(), sidx.begin() + sb.tab_at);
        }
    }
    std::vector<uint64_t> off_table() const {  // the device table: offsets, then soff, then sdst
        std::vector<uint64_t> v(off);
        v.insert(v.end(), soff.begin(), soff.end());
        v.insert(v.end(), sdst.begin(), sdst.end());
        return v;
    }
    std::vector<uint32_t> shard_rows() const {  // the device table: shards, then rows, then sidx
        std::vector<uint32_t> v(shard);
        v.insert(v.end(), row.begin(), row.end());
        v.insert(v.end(), sidx.begin(), sidx.end());
        return v;
    }
    // The pipeline input of sub-batch k over intervals iv, with the device tables d_off / d_sr.
    PipeIn pipe_in(size_t k, const rgl_interval* iv, const uint64_t* d_off, const uint32_t* d_sr,
                   bool block_rows) const {
        const SubBatch& sb = subs[k];
        PipeIn in{iv, sb.n, sb.rows, sb.row_lo, sb.nblk, d_off + sb.tab_at, d_sr + sb.tab_at,
                  block_rows ? d_sr + shard.size() + sb.tab_at : nullptr};
        in.block_local = local[k];
        in.ls.max_block = ls[k].max_block;  // the layout goes by the device tables below
        in.ls.tiles = ls[k].tiles;
        in.ls.chunks = ls[k].chunks;
        in.ls.wide = ls[k].wide;
        if (local[k] && !ls[k].dst.empty()) {
            in.sort_off = d_off + off.size() + sb.tab_at;
            in.sort_dst = d_off + 2 * off.size() + sb.tab_at;
            in.sort_idx = d_sr + 2 * shard.size() + sb.tab_at;
        }
        return in;
    }
};

// Region bits of a sub-batch of `rows` rows under the batch options (0: segments per (shard, row)).
uint32_t batch_region_bits(const rgl_batch_opts* o, uint32_t rows) {
    const uint32_t r = o ? o->region_bits : 0u;
    if (r == RGL_BATCH_NO_REGIONS || r == 0 || rows <= 1) return 0;
    return r;
}

// Region-ordered work needs the device-wide key sort (the block-local sort keeps block order).
void set_regions(PipeIn& in, uint32_t rb) {
    in.region_bits = rb;
    if (rb) in.block_local = 0;
}

int plan_batch(rgl_context* c, const rgl_batch* b, uint64_t sub, BatchPlan* P) {
    const uint64_t* bo = b->block_offsets;
    for (uint32_t i = 0; i < b->num_blocks; i++) {
        if (bo[i + 1] < bo[i]) return fail(RGL_ERR_INVALID_ARGUMENT, "block offsets must be non-decreasing");
        if (b->block_shards[i] >= c->idx->num_shards) return fail(RGL_ERR_INVALID_ARGUMENT, "shard id out of range");
        if (b->block_rows && b->block_rows[i] >= b->num_rows)
            return fail(RGL_ERR_INVALID_ARGUMENT, "block row >= num_rows");
    }
    SubBatch cur{};
    uint32_t rlo = 0xFFFFFFFFu, rhi = 0;
    bool open = false;
    auto close = [&]() {
        if (!open) return;
        P->off.push_back(cur.n);
        P->shard.push_back(0);  // keeps the three tables indexed alike
        P->row.push_back(0);
        cur.row_lo = b->block_rows ? rlo : 0;
        cur.rows = b->block_rows ? rhi - rlo + 1 : b->num_rows;
        P->max_n = std::max(P->max_n, cur.n);
        P->max_rows = std::max(P->max_rows, cur.rows);
        P->max_blk = std::max(P->max_blk, cur.nblk);
        P->subs.push_back(cur);
        open = false;
    };
    for (uint32_t i = 0; i < b->num_blocks; i++) {
        uint64_t at = bo[i], end = bo[i + 1];
        while (at < end) {
            if (!open) {
                cur = SubBatch{at, 0, 0, 0, (uint32_t)P->off.size(), 0};
                rlo = 0xFFFFFFFFu;
                rhi = 0;
                open = true;
            }
            const uint64_t take = std::min(end - at, sub - cur.n);
            P->off.push_back(cur.n);
            P->shard.push_back(b->block_shards[i]);
            P->row.push_back(b->block_rows ? b->block_rows[i] : 0);
            cur.nblk++;
            cur.n += take;
            if (b->block_rows) {
                rlo = std::min(rlo, b->block_rows[i]);
                rhi = std::max(rhi, b->block_rows[i]);
            }
            at += take;
            if (cur.n == sub) close();
        }
    }
    close();
    P->prepare(b->block_rows != nullptr);
    return RGL_OK;
}

Launch batch_launch(rgl_context* c, const rgl_batch_opts* o, rgl_query_opts* q) {
    *q = o ? o->query : rgl_query_opts{};
    if (o && (o->flags & RGL_BF_TUNED) && c->has_tuned) {
        if (!q->chunk) q->chunk = c->tuned.chunk;
        if (!q->ctas_per_sm) q->ctas_per_sm = c->tuned.ctas_per_sm;
        if (!q->pair_ratio) q->pair_ratio = c->tuned.pair_ratio;
    }
    return pick_launch(q);
}

// Enqueues a whole batch on the context stream: zero the outputs, one pipeline run per sub-batch,
// then the error word and the stats accumulator to pinned host memory.
int enqueue_batch(rgl_context* c, const rgl_batch* b, const BatchPlan& P, const uint64_t* d_off,
                  const uint32_t* d_sr, const rgl_query_opts* q, uint32_t* d_counts, unsigned long long* d_bp,
                  bool events, uint32_t* launches, const rgl_batch_opts* o) {
    cudaStream_t st = c->stream;
    const uint32_t D = c->idx->num_sources;
    uint32_t* d_small = c->small.as<uint32_t>();
    RGL_CUDA(cudaMemsetAsync(d_small, 0, 64, st));
    RGL_CUDA(cudaMemsetAsync(c->acc.p, 0, 64, st));
    RGL_CUDA(cudaMemsetAsync(d_counts, 0, (size_t)b->num_rows * D * 4, st));
    if (d_bp) RGL_CUDA(cudaMemsetAsync(d_bp, 0, (size_t)b->num_rows * D * 8, st));
    PipeMode m;
    m.zero_out = false;
    m.reset_err = false;
    m.events = events;
    m.acc = c->acc.as<unsigned long long>();
    uint32_t nl = 0;
    for (size_t k = 0; k < P.subs.size(); k++) {
        const SubBatch& sb = P.subs[k];
        PipeIn in = P.pipe_in(k, b->d_intervals + sb.begin, d_off, d_sr, b->block_rows != nullptr);
        set_regions(in, batch_region_bits(o, sb.rows));
        RGL_TRY(run_pipeline(c, in, q, d_counts + (uint64_t)sb.row_lo * D,
                             d_bp ? d_bp + (uint64_t)sb.row_lo * D : nullptr, nullptr, m));
        nl += c->last_launches;
    }
    RGL_CUDA(cudaMemcpyAsync(c->h_small, d_small, 4, cudaMemcpyDeviceToHost, st));
    RGL_CUDA(cudaMemcpyAsync(c->h_acc, c->acc.p, 64, cudaMemcpyDeviceToHost, st));
    *launches = nl;
    return RGL_OK;
}

void graph_drop(rgl_context* c) {
    if (c->gc.exec) cudaGraphExecDestroy(c->gc.exec);
    if (c->gc.graph) cudaGraphDestroy(c->gc.graph);
    c->gc.exec = nullptr;
    c->gc.graph = nullptr;
    c->gc.key.clear();
}

std::vector<uint64_t> batch_key(rgl_context* c, const rgl_batch* b, const rgl_batch_opts* o, const rgl_query_opts& q,
                                const Launch& L, const void* d_counts, const void* d_bp) {
    std::vector<uint64_t> k;
    k.reserve(17 + 3ull * b->num_blocks);
    k.push_back(b->num_rows);
    k.push_back(b->num_blocks);
    k.push_back((uint64_t)(uintptr_t)b->d_intervals);
    k.push_back((uint64_t)(uintptr_t)d_counts);
    k.push_back((uint64_t)(uintptr_t)d_bp);
    k.push_back(((uint64_t)L.chunk << 32) | L.ctas_per_sm);
    k.push_back(((uint64_t)L.pair_ratio << 32) | (o ? o->query.flags : 0));
    // as asked for: a default is more than the value it stands for (items sized by the run, a cost per run)
    k.push_back(((uint64_t)q.chunk << 32) | q.pair_ratio);
    k.push_back(o ? o->sub_batch : 0);
    k.push_back(o ? o->region_bits : 0);
    k.push_back(c->ws_sig);
    k.push_back(b->block_rows ? 1 : 0);
    for (uint32_t i = 0; i <= b->num_blocks; i++) k.push_back(b->block_offsets[i]);
    for (uint32_t i = 0; i < b->num_blocks; i++)
        k.push_back(((uint64_t)b->block_shards[i] << 32) | (b->block_rows ? b->block_rows[i] : 0));
    return k;
}

}  // namespace

namespace rgl {

cudaStream_t context_stream(rgl_context* c) { return c->stream; }

int context_reserve_rows(rgl_context* c, uint64_t max_intervals, uint32_t max_rows, uint32_t max_blocks) {
    RGL_CUDA(cudaSetDevice(c->idx->device));
    return ensure_workspace(c, max_intervals, max_rows, max_blocks);
}

int context_growth_bytes(rgl_context* c, uint64_t n, uint32_t rows, uint32_t nblk, uint64_t* bytes) {
    return size_workspace(c, n, rows, nblk, bytes);
}

// One batch whose intervals are already on the device, rows taken from the blocks (interval sids are
// ignored), as a single pipeline run: zero the num_rows x D outputs, sweep, error word to the host.
// Asynchronous on the context stream; the caller synchronises and then calls context_errors.
int enqueue_block_rows(rgl_context* c, uint32_t num_rows, uint32_t nblk, const uint32_t* shards, const uint32_t* rows,
                       const uint64_t* off, const rgl_interval* d_iv, const rgl_query_opts* q, uint32_t* d_counts,
                       unsigned long long* d_bp) {
    cudaStream_t st = c->stream;
    const uint32_t D = c->idx->num_sources;
    for (uint32_t i = 0; i < nblk; i++)
        if (shards[i] >= c->idx->num_shards || rows[i] >= num_rows)
            return fail(RGL_ERR_INVALID_ARGUMENT, "block shard or row out of range");
    const uint64_t n = nblk ? off[nblk] - off[0] : 0;
    RGL_TRY(ensure_workspace(c, n, 0, nblk));
    std::vector<uint64_t> rel(nblk + 1);
    for (uint32_t i = 0; i <= nblk; i++) rel[i] = off[i] - off[0];
    // device tables: offsets then the sort's segment-order offsets and destinations; shards, rows,
    // then the blocks' ranks in segment order
    LocalSort ls;
    const bool local = blocks_local(nblk, rel.data(), shards, rows, num_rows, 0, &ls);
    const bool perm = local && !ls.dst.empty();
    std::vector<uint64_t> ot(rel);
    if (perm) {
        ot.insert(ot.end(), ls.soff.begin(), ls.soff.end());
        ot.insert(ot.end(), ls.dst.begin(), ls.dst.end());
    }
    std::vector<uint32_t> sr(3ull * nblk + 3, 0);
    for (uint32_t i = 0; i < nblk; i++) {
        sr[i] = shards[i];
        sr[nblk + 1 + i] = rows[i];
        if (perm) sr[2 * (nblk + 1) + i] = ls.idx[i];
    }
    RGL_TRY(c->bt_off.ensure(ot.size() * 8 + 8));
    RGL_TRY(c->bt_shard.ensure(sr.size() * 4 + 4));
    RGL_CUDA(cudaMemcpyAsync(c->bt_off.p, ot.data(), ot.size() * 8, cudaMemcpyHostToDevice, st));
    RGL_CUDA(cudaMemcpyAsync(c->bt_shard.p, sr.data(), sr.size() * 4, cudaMemcpyHostToDevice, st));
    // the interval copies and table uploads above are ordered before the pipeline on this stream
    RGL_CUDA(cudaMemsetAsync(d_counts, 0, (size_t)num_rows * D * 4, st));
    if (d_bp) RGL_CUDA(cudaMemsetAsync(d_bp, 0, (size_t)num_rows * D * 8, st));
    PipeIn in{d_iv + off[0], n, num_rows, 0, nblk, c->bt_off.as<uint64_t>(), c->bt_shard.as<uint32_t>(),
              c->bt_shard.as<uint32_t>() + nblk + 1, 1};
    in.block_local = local;
    if (perm) {
        in.sort_off = c->bt_off.as<uint64_t>() + (nblk + 1);
        in.sort_dst = c->bt_off.as<uint64_t>() + 2 * (nblk + 1);
        in.sort_idx = c->bt_shard.as<uint32_t>() + 2 * (nblk + 1);
    }
    in.ls = std::move(ls);
    PipeMode m;
    m.zero_out = false;
    // the table uploads read pageable vectors that die here: an asynchronous copy from pageable
    // memory has staged its source before it returns
    return run_pipeline(c, in, q, d_counts, d_bp, nullptr, m);
}

// After the stream has been synchronised: the error bits of the last run.
int context_errors(rgl_context* c) { return finish(c, pick_launch(nullptr), nullptr); }

uint32_t context_last_launches(rgl_context* c) { return c->last_launches; }

}  // namespace rgl

extern "C" {

int rgl_context_create(rgl_index* index, void* stream, rgl_context** out) {
    clear_error();
    if (!index || !out) return fail(RGL_ERR_INVALID_ARGUMENT, "null argument");
    auto* c = new rgl_context();
    c->idx = index;
    c->device = index->device;
    index->refs.fetch_add(1);
    int s = RGL_OK;
    if (cudaSetDevice(index->device) != cudaSuccess) s = fail(RGL_ERR_DEVICE, "cudaSetDevice");
    if (s == RGL_OK) {
        if (stream) c->stream = reinterpret_cast<cudaStream_t>(stream);
        else if (cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess)
            s = fail(RGL_ERR_DEVICE, "cudaStreamCreate");
        else
            c->own_stream = true;
    }
    if (s == RGL_OK && (cudaStreamCreateWithFlags(&c->side, cudaStreamNonBlocking) != cudaSuccess ||
                        cudaEventCreateWithFlags(&c->ev_fork, cudaEventDisableTiming) != cudaSuccess ||
                        cudaEventCreateWithFlags(&c->ev_join, cudaEventDisableTiming) != cudaSuccess))
        s = fail(RGL_ERR_DEVICE, "side stream");
    if (s == RGL_OK) cudaDeviceGetAttribute(&c->num_sms, cudaDevAttrMultiProcessorCount, index->device);
    // shared-memory tallies of up to 160 KB (one row, D x 12 B); set once here so that no launch
    // path changes function attributes (graph capture included)
    if (s == RGL_OK) {
        const int mx = 160 * 1024;
        if (cudaFuncSetAttribute(k_sweep<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) != cudaSuccess ||
            cudaFuncSetAttribute(k_sweep<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) != cudaSuccess ||
            cudaFuncSetAttribute(k_sweep<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) != cudaSuccess ||
            cudaFuncSetAttribute(k_sweep<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) != cudaSuccess ||
            cudaFuncSetAttribute(k_pairs<true, true, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_pairs<false, true, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_pairs<true, true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) !=
                cudaSuccess ||
            cudaFuncSetAttribute(k_pairs<false, true, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx) !=
                cudaSuccess)
            s = fail(RGL_ERR_DEVICE, "cudaFuncSetAttribute");
    }
    for (int i = 0; i < 4 && s == RGL_OK; i++)
        if (cudaEventCreate(&c->ev[i]) != cudaSuccess) s = fail(RGL_ERR_DEVICE, "cudaEventCreate");
    // one page-locked allocation: the counter mirrors (256 bytes each), then the staging buffer
    if (s == RGL_OK && cudaMallocHost(&c->h_small, 512 + kHostIoBytes) != cudaSuccess) s = fail(RGL_ERR_OOM, "pinned");
    if (s == RGL_OK) {
        unsigned char* base = reinterpret_cast<unsigned char*>(c->h_small);
        c->h_acc = reinterpret_cast<unsigned long long*>(base + 256);
        c->h_io = base + 512;
    }
    if (s == RGL_OK) s = c->small.ensure(256);
    if (s != RGL_OK) {
        rgl_context_destroy(c);
        return s;
    }
    *out = c;
    return RGL_OK;
}

int rgl_context_destroy(rgl_context* c) {
    clear_error();
    if (!c) return RGL_OK;
    cudaSetDevice(c->device);
    if (c->stream) cudaStreamSynchronize(c->stream);
    if (c->side) cudaStreamSynchronize(c->side);
    DevBuf* bufs[] = {&c->iv, &c->blk_off, &c->blk_shard, &c->key_a, &c->key_b, &c->val_a, &c->val_b,
                      &c->ekey_a, &c->ekey_b, &c->starts, &c->ends, &c->shard, &c->row, &c->segnum, &c->seg_begin, &c->ps,
                      &c->pe, &c->emax, &c->lo, &c->cnt, &c->place, &c->rlo, &c->ranges, &c->rpos, &c->cub_tmp, &c->small,
                      &c->out_counts, &c->out_bp, &c->item_r0, &c->segtab, &c->tab2, &c->pc, &c->cr, &c->uhi, &c->rt,
                      &c->ulen, &c->rpair, &c->sums, &c->esums, &c->ppos, &c->psegs, &c->prow, &c->item_t0, &c->seg_need,
                      &c->item_hits, &c->item_base, &c->pairs, &c->bt_off, &c->bt_shard, &c->acc, &c->gc.t_off,
                      &c->gc.t_shard, &c->cub_tmp2, &c->sortplan, &c->sort_tab, &c->sort_rank};
    if (c->gc.exec) cudaGraphExecDestroy(c->gc.exec);
    if (c->gc.graph) cudaGraphDestroy(c->gc.graph);
    if (c->copy_stream) cudaStreamSynchronize(c->copy_stream);
    for (DevBuf* b : bufs) b->release();
    for (int i = 0; i < 2; i++) {
        c->stage[i].release();
        if (c->ev_copied[i]) cudaEventDestroy(c->ev_copied[i]);
        if (c->ev_used[i]) cudaEventDestroy(c->ev_used[i]);
    }
    if (c->copy_stream) cudaStreamDestroy(c->copy_stream);
    for (auto& e : c->ev)
        if (e) cudaEventDestroy(e);
    for (auto& e : c->tev) cudaEventDestroy(e);
    if (c->h_small) cudaFreeHost(c->h_small);
    if (c->own_stream && c->stream) cudaStreamDestroy(c->stream);
    if (c->side) cudaStreamDestroy(c->side);
    if (c->ev_fork) cudaEventDestroy(c->ev_fork);
    if (c->ev_join) cudaEventDestroy(c->ev_join);
    index_release(c->idx);
    delete c;
    (void)cudaGetLastError();
    return RGL_OK;
}

int rgl_context_reserve(rgl_context* c, uint64_t max_intervals, uint32_t max_rows) {
    clear_error();
    if (!c) return fail(RGL_ERR_INVALID_ARGUMENT, "null context");
    RGL_CUDA(cudaSetDevice(c->idx->device));
    return ensure_workspace(c, max_intervals, max_rows, 4096);
}

void* rgl_context_stream(rgl_context* c) { return c ? (void*)c->stream : nullptr; }

int rgl_context_sync(rgl_context* c) {
    if (!c) return fail(RGL_ERR_INVALID_ARGUMENT, "null context");
    RGL_CUDA(cudaStreamSynchronize(c->stream));
    return RGL_OK;
}

int rgl_query_counts_device(rgl_context* c, uint32_t num_rows, uint32_t num_shards, const uint32_t* shard_ids,
                            const uint64_t* shard_offsets, const rgl_interval* d_intervals,
                            const rgl_query_opts* opts, uint32_t* d_counts, uint64_t* d_overlap_bp,
                            rgl_query_stats* stats) {
    clear_error();
    if (!c || (num_shards && (!shard_ids || !shard_offsets))) return fail(RGL_ERR_INVALID_ARGUMENT, "null argument");
    if (!d_counts) return fail(RGL_ERR_INVALID_ARGUMENT, "counts buffer is required");
    RGL_CUDA(cudaSetDevice(c->idx->device));
    uint64_t n = num_shards ? shard_offsets[num_shards] - shard_offsets[0] : 0;
    if (n >= (1ull << 31)) return fail(RGL_ERR_INVALID_ARGUMENT, "at most 2^31-1 query intervals per call");
    for (uint32_t i = 0; i < num_shards; i++)
        if (shard_ids[i] >= c->idx->num_shards) return fail(RGL_ERR_INVALID_ARGUMENT, "shard id out of range");
    RGL_TRY(ensure_workspace(c, n, 0, num_shards));
    std::vector<uint64_t> off(num_shards + 1);
    for (uint32_t i = 0; i <= num_shards; i++) off[i] = shard_offsets[i] - shard_offsets[0];
    if (num_shards) {
        RGL_CUDA(cudaMemcpyAsync(c->blk_off.p, off.data(), off.size() * 8, cudaMemcpyHostToDevice, c->stream));
        RGL_CUDA(cudaMemcpyAsync(c->blk_shard.p, shard_ids, num_shards * 4ull, cudaMemcpyHostToDevice, c->stream));
        RGL_CUDA(cudaMemcpyAsync(c->iv.p, d_intervals + shard_offsets[0], n * sizeof(rgl_interval),
                                 cudaMemcpyDeviceToDevice, c->stream));
    }
    PipeIn in{c->iv.as<rgl_interval>(), n, num_rows, 0, num_shards, c->blk_off.as<uint64_t>(),
              c->blk_shard.as<uint32_t>(), nullptr};
    in.block_local = blocks_local(num_shards, off.data(), shard_ids, nullptr, num_rows, 0, &in.ls);
    RGL_TRY(run_pipeline(c, in, opts, d_counts, reinterpret_cast<unsigned long long*>(d_overlap_bp), stats));
    if (!stats) return RGL_OK;
    RGL_CUDA(cudaStreamSynchronize(c->stream));
    return finish(c, pick_launch(opts), stats);
}

int rgl_query_counts(rgl_context* c, const rgl_query_batch* b, const rgl_query_opts* opts, uint32_t* counts,
                     uint64_t* overlap_bp, rgl_query_stats* stats) {
    clear_error();
    if (!c || !b || !counts) return fail(RGL_ERR_INVALID_ARGUMENT, "null argument");
    RGL_CUDA(cudaSetDevice(c->idx->device));
    std::vector<uint32_t> ids;
    std::vector<const rgl_query_shard*> blocks;
    RGL_TRY(resolve_blocks(c, b, &ids, &blocks));
    uint64_t n = 0;
    std::vector<uint64_t> off(blocks.size() + 1, 0);
    for (size_t i = 0; i < blocks.size(); i++) {
        off[i] = n;
        n += blocks[i]->count;
    }
    off[blocks.size()] = n;
    if (n >= (1ull << 31)) return fail(RGL_ERR_INVALID_ARGUMENT, "at most 2^31-1 query intervals per call");
    const uint32_t rows = b->num_rows;
    const uint64_t cells = (uint64_t)rows * c->idx->num_sources;
    RGL_TRY(ensure_workspace(c, n, rows, (uint32_t)blocks.size()));
    cudaStream_t st = c->stream;
    PipeIn in{nullptr, n, rows, 0, (uint32_t)blocks.size(), nullptr, nullptr, nullptr};
    in.block_local = blocks_local((uint32_t)blocks.size(), off.data(), ids.data(), nullptr, rows, 0, &in.ls);
    // the outputs lie together on the device (overlaps, then counts), so that one copy brings both
    unsigned long long* d_bp = c->out_bp.as<unsigned long long>();
    uint32_t* d_counts = reinterpret_cast<uint32_t*>(d_bp + (overlap_bp ? cells : 0));
    const uint64_t out_bytes = cells * (overlap_bp ? 12 : 4);
    int s = upload_blocks(c, blocks, off, ids, &in, st);
    if (s == RGL_OK) s = run_pipeline(c, in, opts, d_counts, overlap_bp ? d_bp : nullptr, stats);
    if (s != RGL_OK) {
        cudaStreamSynchronize(st);  // the staging buffer may be in use
        return s;
    }
    const bool stage = cells && out_bytes <= kHostIoBytes;
    if (stage) {
        RGL_CUDA(cudaMemcpyAsync(c->h_io, c->out_bp.p, out_bytes, cudaMemcpyDeviceToHost, st));
    } else if (cells) {
        RGL_CUDA(cudaMemcpyAsync(counts, d_counts, cells * 4, cudaMemcpyDeviceToHost, st));
        if (overlap_bp) RGL_CUDA(cudaMemcpyAsync(overlap_bp, d_bp, cells * 8, cudaMemcpyDeviceToHost, st));
    }
    RGL_CUDA(cudaStreamSynchronize(st));
    if (stage) {
        if (overlap_bp) std::memcpy(overlap_bp, c->h_io, cells * 8);
        std::memcpy(counts, c->h_io + (overlap_bp ? cells * 8 : 0), cells * 4);
    }
    return finish(c, pick_launch(opts), stats);
}

int rgl_query_batch_device(rgl_context* c, const rgl_batch* b, const rgl_batch_opts* o, uint32_t* d_counts,
                           uint64_t* d_overlap_bp, rgl_batch_stats* stats) {
    clear_error();
    if (!c || !b || !d_counts) return fail(RGL_ERR_INVALID_ARGUMENT, "null argument");
    if (b->num_blocks && (!b->block_offsets || !b->block_shards || !b->d_intervals))
        return fail(RGL_ERR_INVALID_ARGUMENT, "incomplete batch");
    RGL_CUDA(cudaSetDevice(c->idx->device));
    const uint64_t sub = (o && o->sub_batch) ? std::min<uint64_t>(o->sub_batch, kMaxRunIntervals) : (1ull << 25);
    rgl_query_opts q;
    const Launch L = batch_launch(c, o, &q);
    const bool graph = o && (o->flags & RGL_BF_GRAPH);
    unsigned long long* d_bp = (d_overlap_bp && !(q.flags & RGL_QF_NO_OVERLAP))
                                   ? reinterpret_cast<unsigned long long*>(d_overlap_bp) : nullptr;
    cudaStream_t st = c->stream;
    BatchPlan P;
    std::vector<uint64_t> key;
    bool replay = false;
    if (graph) {
        key = batch_key(c, b, o, q, L, d_counts, d_bp);
        replay = c->gc.exec && key == c->gc.key;
    }
    if (!replay) {
        RGL_TRY(plan_batch(c, b, sub, &P));
        RGL_TRY(ensure_workspace(c, P.max_n, 0, P.max_blk));
    }
    if (stats) RGL_CUDA(cudaEventRecord(c->ev[0], st));
    uint32_t launches = 0, subs = 0, nodes = 0;
    if (replay) {
        RGL_CUDA(cudaGraphLaunch(c->gc.exec, st));
        launches = c->gc.launches;
        subs = c->gc.subs;
        nodes = c->gc.nodes;
    } else if (graph) {
        RGL_CUDA(cudaStreamSynchronize(st));  // the previous graph may still read its tables
        graph_drop(c);
        const std::vector<uint64_t> ot = P.off_table();
        RGL_TRY(c->gc.t_off.ensure(ot.size() * 8 + 8));
        const std::vector<uint32_t> sr = P.shard_rows();
        RGL_TRY(c->gc.t_shard.ensure(sr.size() * 4 + 4));
        RGL_CUDA(cudaMemcpy(c->gc.t_off.p, ot.data(), ot.size() * 8, cudaMemcpyHostToDevice));
        RGL_CUDA(cudaMemcpy(c->gc.t_shard.p, sr.data(), sr.size() * 4, cudaMemcpyHostToDevice));
        // the key is taken after the workspace is sized, so that a later reallocation invalidates it
        key = batch_key(c, b, o, q, L, d_counts, d_bp);
        RGL_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        int s = enqueue_batch(c, b, P, c->gc.t_off.as<uint64_t>(), c->gc.t_shard.as<uint32_t>(), &q, d_counts, d_bp,
                              false, &launches, o);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(st, &g);
        if (s != RGL_OK) {
            if (g) cudaGraphDestroy(g);
            return s;
        }
        if (e != cudaSuccess) return fail(RGL_ERR_DEVICE, std::string("stream capture: ") + cudaGetErrorString(e));
        cudaGraphExec_t x = nullptr;
        e = cudaGraphInstantiate(&x, g, 0);
        if (e != cudaSuccess) {
            cudaGraphDestroy(g);
            return fail(RGL_ERR_DEVICE, std::string("graph instantiate: ") + cudaGetErrorString(e));
        }
        size_t nn = 0;
        cudaGraphGetNodes(g, nullptr, &nn);
        c->gc.graph = g;
        c->gc.exec = x;
        c->gc.key = std::move(key);
        c->gc.nodes = nodes = (uint32_t)nn;
        c->gc.launches = launches;
        c->gc.subs = subs = (uint32_t)P.subs.size();
        RGL_CUDA(cudaGraphLaunch(x, st));
    } else {
        const std::vector<uint64_t> ot = P.off_table();
        RGL_TRY(c->bt_off.ensure(ot.size() * 8 + 8));
        const std::vector<uint32_t> sr = P.shard_rows();
        RGL_TRY(c->bt_shard.ensure(sr.size() * 4 + 4));
        RGL_CUDA(cudaMemcpyAsync(c->bt_off.p, ot.data(), ot.size() * 8, cudaMemcpyHostToDevice, st));
        RGL_CUDA(cudaMemcpyAsync(c->bt_shard.p, sr.data(), sr.size() * 4, cudaMemcpyHostToDevice, st));
        RGL_TRY(enqueue_batch(c, b, P, c->bt_off.as<uint64_t>(), c->bt_shard.as<uint32_t>(), &q, d_counts, d_bp, true,
                              &launches, o));
        subs = (uint32_t)P.subs.size();
    }
    c->last_n = 0;  // the single-call stats of finish() do not apply to a batch
    if (!stats) return RGL_OK;
    RGL_CUDA(cudaEventRecord(c->ev[2], st));
    RGL_CUDA(cudaStreamSynchronize(st));
    float ms = 0;
    RGL_CUDA(cudaEventElapsedTime(&ms, c->ev[0], c->ev[2]));
    std::memset(stats, 0, sizeof(*stats));
    stats->ranges = c->h_acc[0];
    stats->db_swept = c->h_acc[1];
    stats->rank_positions = c->h_acc[2];
    stats->pair_candidates = c->h_acc[3];
    stats->query_intervals = c->h_acc[4];
    stats->sub_batches = subs;
    stats->kernel_launches = launches;
    stats->graph_nodes = nodes;
    stats->graph_replayed = replay ? 1 : 0;
    stats->device_ms = ms;
    stats->chunk = L.chunk;
    stats->ctas_per_sm = L.ctas_per_sm;
    stats->pair_ratio = L.pair_ratio;
    return finish(c, L, nullptr);
}

int rgl_query_batch_host(rgl_context* c, const rgl_batch* b, const rgl_interval* h_intervals, const rgl_batch_opts* o,
                    uint32_t* counts, uint64_t* overlap_bp, rgl_batch_stats* stats) {
    clear_error();
    if (!c || !b || !counts) return fail(RGL_ERR_INVALID_ARGUMENT, "null argument");
    if (b->num_blocks && (!b->block_offsets || !b->block_shards || !h_intervals))
        return fail(RGL_ERR_INVALID_ARGUMENT, "incomplete batch");
    RGL_CUDA(cudaSetDevice(c->idx->device));
    const uint64_t sub = (o && o->sub_batch) ? std::min<uint64_t>(o->sub_batch, kMaxRunIntervals) : (1ull << 25);
    rgl_query_opts q;
    const Launch L = batch_launch(c, o, &q);
    const bool want_bp = overlap_bp && !(q.flags & RGL_QF_NO_OVERLAP);
    const uint32_t D = c->idx->num_sources;
    const uint64_t cells = (uint64_t)b->num_rows * D;
    BatchPlan P;
    RGL_TRY(plan_batch(c, b, sub, &P));
    RGL_TRY(ensure_workspace(c, P.max_n, b->num_rows, P.max_blk));
    for (int i = 0; i < 2; i++) {
        RGL_TRY(c->stage[i].ensure(std::max<uint64_t>(P.max_n, 1) * sizeof(rgl_interval)));
        if (!c->ev_copied[i]) RGL_CUDA(cudaEventCreateWithFlags(&c->ev_copied[i], cudaEventDisableTiming));
        if (!c->ev_used[i]) RGL_CUDA(cudaEventCreateWithFlags(&c->ev_used[i], cudaEventDisableTiming));
    }
    if (!c->copy_stream) RGL_CUDA(cudaStreamCreateWithFlags(&c->copy_stream, cudaStreamNonBlocking));
    cudaStream_t st = c->stream, cs = c->copy_stream;
    const std::vector<uint32_t> sr = P.shard_rows();
    const std::vector<uint64_t> ot = P.off_table();
    RGL_TRY(c->bt_off.ensure(ot.size() * 8 + 8));
    RGL_TRY(c->bt_shard.ensure(sr.size() * 4 + 4));
    if (stats) RGL_CUDA(cudaEventRecord(c->ev[0], st));
    RGL_CUDA(cudaMemcpyAsync(c->bt_off.p, ot.data(), ot.size() * 8, cudaMemcpyHostToDevice, st));
    RGL_CUDA(cudaMemcpyAsync(c->bt_shard.p, sr.data(), sr.size() * 4, cudaMemcpyHostToDevice, st));
    uint32_t* d_counts = c->out_counts.as<uint32_t>();
    unsigned long long* d_bp = want_bp ? c->out_bp.as<unsigned long long>() : nullptr;
    uint32_t* d_small = c->small.as<uint32_t>();
    RGL_CUDA(cudaMemsetAsync(d_small, 0, 64, st));
    RGL_CUDA(cudaMemsetAsync(c->acc.p, 0, 64, st));
    RGL_CUDA(cudaMemsetAsync(d_counts, 0, cells * 4, st));
    if (d_bp) RGL_CUDA(cudaMemsetAsync(d_bp, 0, cells * 8, st));
    PipeMode m;
    m.zero_out = false;
    m.reset_err = false;
    m.acc = c->acc.as<unsigned long long>();
    uint32_t launches = 0;
    const uint64_t* d_off = c->bt_off.as<uint64_t>();
    const uint32_t* d_sr = c->bt_shard.as<uint32_t>();
    for (size_t k = 0; k < P.subs.size(); k++) {
        const SubBatch& sb = P.subs[k];
        const int slot = (int)(k & 1);
        rgl_interval* stage = c->stage[slot].as<rgl_interval>();
        // the staging buffer is free once the sub-batch two back has been swept
        if (k >= 2) RGL_CUDA(cudaStreamWaitEvent(cs, c->ev_used[slot], 0));
        RGL_CUDA(cudaMemcpyAsync(stage, h_intervals + sb.begin, sb.n * sizeof(rgl_interval), cudaMemcpyHostToDevice, cs));
        RGL_CUDA(cudaEventRecord(c->ev_copied[slot], cs));
        RGL_CUDA(cudaStreamWaitEvent(st, c->ev_copied[slot], 0));
        PipeIn in = P.pipe_in(k, stage, d_off, d_sr, b->block_rows != nullptr);
        set_regions(in, batch_region_bits(o, sb.rows));
        RGL_TRY(run_pipeline(c, in, &q, d_counts + (uint64_t)sb.row_lo * D, d_bp ? d_bp + (uint64_t)sb.row_lo * D : nullptr,
                             nullptr, m));
        RGL_CUDA(cudaEventRecord(c->ev_used[slot], st));
        launches += c->last_launches;
    }
    RGL_CUDA(cudaMemcpyAsync(c->h_small, d_small, 4, cudaMemcpyDeviceToHost, st));
    RGL_CUDA(cudaMemcpyAsync(c->h_acc, c->acc.p, 64, cudaMemcpyDeviceToHost, st));
    if (cells) {
        RGL_CUDA(cudaMemcpyAsync(counts, d_counts, cells * 4, cudaMemcpyDeviceToHost, st));
        if (overlap_bp) {
            if (d_bp) RGL_CUDA(cudaMemcpyAsync(overlap_bp, d_bp, cells * 8, cudaMemcpyDeviceToHost, st));
            else std::memset(overlap_bp, 0, cells * 8);
        }
    }
    if (stats) RGL_CUDA(cudaEventRecord(c->ev[2], st));
    RGL_CUDA(cudaStreamSynchronize(st));
    c->last_n = 0;
    if (stats) {
        float ms = 0;
        RGL_CUDA(cudaEventElapsedTime(&ms, c->ev[0], c->ev[2]));
        std::memset(stats, 0, sizeof(*stats));
        stats->ranges = c->h_acc[0];
        stats->db_swept = c->h_acc[1];
        stats->rank_positions = c->h_acc[2];
        stats->pair_candidates = c->h_acc[3];
        stats->query_intervals = c->h_acc[4];
        stats->sub_batches = (uint32_t)P.subs.size();
        stats->kernel_launches = launches;
        stats->device_ms = ms;
        stats->chunk = L.chunk;
        stats->ctas_per_sm = L.ctas_per_sm;
        stats->pair_ratio = L.pair_ratio;
    }
    return finish(c, L, nullptr);
}

// Autotuner: times the batch's largest sub-batch over a grid of launch shapes (pair_ratio first at the default
// shape, then work-item size x CTAs per SM) and keeps the one whose whole run is the fastest.  Ratio 4 stands for the
// default, which is tried as such (see by_ranks), as is the default size (item_size): what wins as a default is kept as 0.
// The sweeps alone do not say which ratio is the fastest, since ranges swept by ranks have their ends sorted and
// tabled before: by the fastest sweeps 64 files of up to 1e5 intervals against 3.2e6 took 667 us (ratio 1) and 48 of up
// to 1e6 2,128 (ratio 2), by the fastest run 321 and 1,343, the default's.
int rgl_batch_autotune(rgl_context* c, const rgl_batch* b, uint64_t sub_batch, rgl_query_opts* best,
                       rgl_tune_trial* trials, uint32_t max_trials, uint32_t* num_trials) {
    clear_error();
    if (!c || !b || !best) return fail(RGL_ERR_INVALID_ARGUMENT, "null argument");
    RGL_CUDA(cudaSetDevice(c->idx->device));
    BatchPlan P;
    const uint64_t sub = sub_batch ? std::min<uint64_t>(sub_batch, kMaxRunIntervals) : (1ull << 25);
    RGL_TRY(plan_batch(c, b, sub, &P));
    if (P.subs.empty()) return fail(RGL_ERR_INVALID_ARGUMENT, "empty batch");
    size_t big = 0;
    for (size_t i = 1; i < P.subs.size(); i++)
        if (P.subs[i].n > P.subs[big].n) big = i;
    const SubBatch sb = P.subs[big];
    RGL_TRY(ensure_workspace(c, sb.n, sb.rows, sb.nblk));
    cudaStream_t st = c->stream;
    const std::vector<uint64_t> ot = P.off_table();
    RGL_TRY(c->bt_off.ensure(ot.size() * 8 + 8));
    const std::vector<uint32_t> sr = P.shard_rows();
    RGL_TRY(c->bt_shard.ensure(sr.size() * 4 + 4));
    RGL_CUDA(cudaMemcpyAsync(c->bt_off.p, ot.data(), ot.size() * 8, cudaMemcpyHostToDevice, st));
    RGL_CUDA(cudaMemcpyAsync(c->bt_shard.p, sr.data(), sr.size() * 4, cudaMemcpyHostToDevice, st));
    PipeIn in = P.pipe_in(big, b->d_intervals + sb.begin, c->bt_off.as<uint64_t>(), c->bt_shard.as<uint32_t>(),
                          b->block_rows != nullptr);
    set_regions(in, batch_region_bits(nullptr, sb.rows));
    const bool was_timing = c->timing;
    *best = rgl_query_opts{};
    rgl_query_opts keep{};
    uint32_t nt = 0;
    auto trial = [&](rgl_query_opts q, float* run_ms) -> int {
        float sweep_ms = 1e30f;
        *run_ms = 1e30f;
        for (int rep = 0; rep < 3; rep++) {
            c->timing = true;
            c->tev_used = 0;
            RGL_CUDA(cudaEventRecord(c->ev[0], st));
            RGL_TRY(run_pipeline(c, in, &q, c->out_counts.as<uint32_t>(), c->out_bp.as<unsigned long long>(), nullptr));
            RGL_CUDA(cudaEventRecord(c->ev[2], st));
            RGL_CUDA(cudaStreamSynchronize(st));
            float ms = 0;
            RGL_CUDA(cudaEventElapsedTime(&ms, c->tev[0], c->tev[1]));
            c->tev_used = 0;
            sweep_ms = std::min(sweep_ms, ms);
            RGL_CUDA(cudaEventElapsedTime(&ms, c->ev[0], c->ev[2]));
            *run_ms = std::min(*run_ms, ms);
        }
        const Launch L = pick_launch(&q);
        if (trials && nt < max_trials) trials[nt] = rgl_tune_trial{L.chunk, L.ctas_per_sm, L.pair_ratio, sweep_ms};
        nt++;
        return RGL_OK;
    };
    int s = RGL_OK;
    rgl_query_opts cur{};
    cur.flags = 0;
    float cur_ms = 1e30f;
    for (uint32_t pr : {1u, 2u, 4u, 8u}) {
        rgl_query_opts q = cur;
        q.pair_ratio = pr == pick_launch(nullptr).pair_ratio ? 0 : pr;
        float ms;
        if ((s = trial(q, &ms)) != RGL_OK) break;
        if (ms < cur_ms) {
            cur_ms = ms;
            keep = q;
        }
    }
    cur = keep;
    for (uint32_t ch : {512u, 1024u, 2048u, 4096u, 8192u}) {
        if (s != RGL_OK) break;
        for (uint32_t ct : {2u, 3u, 4u, 6u, 8u}) {
            rgl_query_opts q = cur;
            q.chunk = ch;
            q.ctas_per_sm = ct;
            float ms;
            if ((s = trial(q, &ms)) != RGL_OK) break;
            if (ms < cur_ms) {
                cur_ms = ms;
                keep = q;
            }
        }
    }
    c->timing = was_timing;
    if (s != RGL_OK) return s;
    const Launch L = pick_launch(&keep);
    *best = rgl_query_opts{L.chunk, L.ctas_per_sm, 256, 0, L.pair_ratio};  // what a tuned batch reports
    c->tuned = keep;
    c->has_tuned = true;
    if (num_trials) *num_trials = nt;
    RGL_CUDA(cudaStreamSynchronize(st));
    return finish(c, L, nullptr);
}

}  // extern "C"

namespace {
// The pairs of a batch: place(count, &pairs) says where they go (null: nowhere), once their number is known.
template <typename Place>
int query_pairs(rgl_context* c, const rgl_query_batch* b, uint64_t* out_count, Place place) {
    clear_error();
    if (!c || !b || !out_count) return fail(RGL_ERR_INVALID_ARGUMENT, "null argument");
    RGL_CUDA(cudaSetDevice(c->idx->device));
    *out_count = 0;
    std::vector<uint32_t> ids;
    std::vector<const rgl_query_shard*> blocks;
    RGL_TRY(resolve_blocks(c, b, &ids, &blocks));
    uint64_t n = 0;
    std::vector<uint64_t> off(blocks.size() + 1, 0);
    for (size_t i = 0; i < blocks.size(); i++) {
        off[i] = n;
        n += blocks[i]->count;
    }
    off[blocks.size()] = n;
    RGL_TRY(ensure_workspace(c, n, 0, (uint32_t)blocks.size()));
    cudaStream_t st = c->stream;
    // every candidate run becomes a pair run: a range is swept pair by pair when its candidates are
    // at most pair_ratio x its union, which no range exceeds at this ratio
    rgl_query_opts q{};
    q.pair_ratio = 0xFFFFFFFFu;
    PipeIn in{nullptr, n, b->num_rows, 0, (uint32_t)blocks.size(), nullptr, nullptr, nullptr};
    in.block_local = blocks_local((uint32_t)blocks.size(), off.data(), ids.data(), nullptr, b->num_rows, 0, &in.ls);
    PipeMode m;
    m.zero_out = false;
    m.no_sweep = true;
    int s = upload_blocks(c, blocks, off, ids, &in, st);
    if (s == RGL_OK) s = run_pipeline(c, in, &q, nullptr, nullptr, nullptr, m);
    if (s == RGL_OK)  // the pair work space total (small[12..13]) with the error word
        RGL_CUDA(cudaMemcpyAsync(c->h_small, c->small.p, 64, cudaMemcpyDeviceToHost, st));
    RGL_CUDA(cudaStreamSynchronize(st));
    RGL_TRY(s);
    RGL_TRY(finish(c, pick_launch(&q), nullptr));
    if (!n || !c->idx->num_slots) return RGL_OK;
    uint64_t positions = 0;
    std::memcpy(&positions, c->h_small + 12, 8);
    const uint32_t* Lp = c->small.as<uint32_t>() + 8;
    // items for every warp of the grid below where there are that many positions (2,048 each: 133 warps
    // walked the 272 thousand candidates of 1e5 queries, 118 us a pass)
    const uint64_t even = (positions / ((uint64_t)c->num_sms * 64) + 31) & ~31ull;
    const uint32_t chunk = (uint32_t)std::min<uint64_t>(2048, std::max<uint64_t>(64, even));
    const uint64_t items = (positions + chunk - 1) / chunk;
    if (!items) return RGL_OK;
    RGL_TRY(c->item_hits.ensure((items + 1) * 8));
    RGL_TRY(c->item_base.ensure((items + 1) * 8));
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, (uint64_t*)nullptr, (uint64_t*)nullptr, (int)(items + 1), st);
    RGL_TRY(c->cub_tmp.ensure(tb + 256));
    const unsigned grid = (unsigned)std::min<uint64_t>((items * 32 + 255) / 256, (uint64_t)c->num_sms * 16);
    RGL_CUDA(cudaMemsetAsync(c->item_hits.as<uint64_t>() + items, 0, 8, st));
    k_pair_list<false><<<grid, 256, 0, st>>>(c->ppos.as<uint64_t>(), Lp, c->psegs.as<PairSeg>(),
                                             c->prow.as<uint32_t>(), b->num_rows, c->idx->d_pos, c->idx->d_sid, items,
                                             chunk, c->item_hits.as<uint64_t>(), nullptr, nullptr);
    tb = c->cub_tmp.cap;
    RGL_CUDA(cub::DeviceScan::ExclusiveSum(c->cub_tmp.p, tb, c->item_hits.as<uint64_t>(), c->item_base.as<uint64_t>(),
                                           (int)(items + 1), st));
    uint64_t hits = 0;
    RGL_CUDA(cudaMemcpyAsync(&hits, c->item_base.as<uint64_t>() + items, 8, cudaMemcpyDeviceToHost, st));
    RGL_CUDA(cudaStreamSynchronize(st));
    *out_count = hits;
    if (!hits) return RGL_OK;
    rgl_pair* pairs = nullptr;
    RGL_TRY(place(hits, &pairs));
    if (!pairs) return RGL_OK;
    RGL_TRY(c->pairs.ensure(hits * sizeof(rgl_pair)));
    k_pair_list<true><<<grid, 256, 0, st>>>(c->ppos.as<uint64_t>(), Lp, c->psegs.as<PairSeg>(),
                                            c->prow.as<uint32_t>(), b->num_rows, c->idx->d_pos, c->idx->d_sid, items,
                                            chunk, nullptr, c->item_base.as<uint64_t>(), c->pairs.as<rgl_pair>());
    RGL_CUDA(cudaGetLastError());
    RGL_CUDA(cudaMemcpyAsync(pairs, c->pairs.p, hits * sizeof(rgl_pair), cudaMemcpyDeviceToHost, st));
    RGL_CUDA(cudaStreamSynchronize(st));
    return RGL_OK;
}
}  // namespace

extern "C" {

int rgl_query_pairs(rgl_context* c, const rgl_query_batch* b, uint64_t capacity, rgl_pair* pairs,
                    uint64_t* out_count) {
    return query_pairs(c, b, out_count, [&](uint64_t hits, rgl_pair** to) {
        if (pairs && capacity < hits)
            return fail(RGL_ERR_INVALID_ARGUMENT, "pair capacity too small (needs " + std::to_string(hits) + ")");
        *to = pairs;
        return (int)RGL_OK;
    });
}

int rgl_query_pairs_alloc(rgl_context* c, const rgl_query_batch* b, rgl_pair* (*alloc)(void*, uint64_t), void* user,
                          uint64_t* out_count) {
    if (!alloc) {
        clear_error();
        return fail(RGL_ERR_INVALID_ARGUMENT, "null argument");
    }
    return query_pairs(c, b, out_count, [&](uint64_t hits, rgl_pair** to) {
        *to = alloc(user, hits);
        return *to ? (int)RGL_OK : fail(RGL_ERR_OOM, "no room for " + std::to_string(hits) + " pairs");
    });
}

int rgl_context_check(rgl_context* c) {
    clear_error();
    if (!c) return fail(RGL_ERR_INVALID_ARGUMENT, "null context");
    RGL_CUDA(cudaStreamSynchronize(c->stream));
    return finish(c, pick_launch(nullptr), nullptr);
}

int rgl_context_set_timing(rgl_context* c, int on) {
    if (!c) return fail(RGL_ERR_INVALID_ARGUMENT, "null context");
    c->timing = on != 0;
    c->tev_used = 0;
    return RGL_OK;
}

int rgl_context_sweep_times(rgl_context* c, float* total_ms, uint32_t* launches) {
    if (!c || !total_ms || !launches) return fail(RGL_ERR_INVALID_ARGUMENT, "null argument");
    RGL_CUDA(cudaStreamSynchronize(c->stream));
    float tot = 0;
    for (size_t i = 0; i < c->tev_used; i++) {
        float ms = 0;
        RGL_CUDA(cudaEventElapsedTime(&ms, c->tev[2 * i], c->tev[2 * i + 1]));
        tot += ms;
    }
    *total_ms = tot;
    *launches = (uint32_t)c->tev_used;
    c->tev_used = 0;
    return RGL_OK;
}

int rgl_host_alloc(uint64_t bytes, void** out) {
    if (!out) return fail(RGL_ERR_INVALID_ARGUMENT, "null output");
    *out = nullptr;
    RGL_CUDA(cudaMallocHost(out, bytes ? bytes : 1));
    return RGL_OK;
}

int rgl_host_free(void* p) {
    if (p) RGL_CUDA(cudaFreeHost(p));
    return RGL_OK;
}

}  // extern "C"
