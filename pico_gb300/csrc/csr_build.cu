// Device CSR / virtual-graph builder.
//
// Replaces the reference's serial host builders: VirtualGraph::VirtualGraph +
// MakeUGraph (index2core/shared/virtual_graph.cpp:12-45, 96-192) and the
// std::set adjacency of Graph::readFile (peel/src/graph.cpp:103-131).  Steps,
// all on the GPU:
//   1. degree count (atomicAdd per endpoint; self-loops dropped, ids checked),
//   2. exclusive scan of degrees into int64 row offsets,
//   3. scatter of both directions of every edge into its row,
//   4. segmented row sort by neighbour id, with three size classes: <=32
//      entries (shuffle bitonic, up to four rows a warp), <=4096 (one to four
//      warps, register bitonic), larger (one CTA, a column bitmap or an LSD
//      radix through a global staging buffer),
//   5. optional unique per row, rescan and compaction.
// Steps 1 and 3 go through a partition by row ranges where that pays.  Rows in
// edge-list order (the order MakeUGraph produces) come from a stable radix sort
// of the entries by row instead of steps 1 to 4.
#include <algorithm>
#include <mutex>
#include <vector>

#include "kc_device.cuh"
#include "kc_internal.h"

namespace kc {

static int grid_for(uint64_t items, int threads, int sm_count) {
    uint64_t g = (items + threads - 1) / threads;
    uint64_t cap = (uint64_t)std::max(sm_count, 1) * 16;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

static int current_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 1;
}

// ---------------------------------------------------------------- scan ----
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

__device__ __forceinline__ unsigned long long block_excl_scan_u64(unsigned long long x,
                                                                  unsigned long long *warp_sums,
                                                                  unsigned long long &total) {
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long v = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        unsigned long long y = __shfl_up_sync(KC_FULL_MASK, v, d);
        if (lane >= (unsigned)d) v += y;
    }
    if (lane == 31) warp_sums[warp] = v;
    __syncthreads();
    if (warp == 0) {
        unsigned long long w = lane < (blockDim.x >> 5) ? warp_sums[lane] : 0ull;
        unsigned long long iv = w;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            unsigned long long y = __shfl_up_sync(KC_FULL_MASK, iv, d);
            if (lane >= (unsigned)d) iv += y;
        }
        if (lane < (blockDim.x >> 5)) warp_sums[lane] = iv - w;
        if (lane == 31) warp_sums[32] = iv;
    }
    __syncthreads();
    unsigned long long r = warp_sums[warp] + v - x;
    total = warp_sums[32];
    __syncthreads();
    return r;
}

__global__ void scan_tile_sums(const uint32_t *__restrict__ in, uint64_t n, unsigned long long *sums) {
    __shared__ unsigned long long ws[33];
    uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
    unsigned long long s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        uint64_t j = base + (uint64_t)i * SCAN_THREADS + threadIdx.x;
        if (j < n) s += in[j];
    }
    unsigned long long tot;
    block_excl_scan_u64(s, ws, tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void scan_sums_single(unsigned long long *sums, uint64_t count) {
    __shared__ unsigned long long ws[33];
    __shared__ unsigned long long carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint64_t base = 0; base < count; base += blockDim.x) {
        uint64_t j = base + threadIdx.x;
        unsigned long long x = j < count ? sums[j] : 0ull;
        unsigned long long tot;
        unsigned long long ex = block_excl_scan_u64(x, ws, tot);
        if (j < count) sums[j] = carry + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) sums[count] = carry;
}

__global__ void scan_tile_apply(const uint32_t *__restrict__ in, int64_t *__restrict__ out, uint64_t n,
                                const unsigned long long *sums) {
    // a word of padding per 32 keeps the threads' runs of 8 off each other's
    // banks, and the offsets leave through the same array, a warp's 32 at a time
    constexpr int PAD = SCAN_TILE + SCAN_TILE / 32;
    __shared__ unsigned long long ws[33];
    __shared__ unsigned long long tile[PAD];
    uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        const int k = i * SCAN_THREADS + threadIdx.x;
        const uint64_t j = base + k;
        tile[k + k / 32] = j < n ? in[j] : 0u;
    }
    __syncthreads();
    const int k0 = threadIdx.x * SCAN_ITEMS + threadIdx.x * SCAN_ITEMS / 32;
    unsigned long long loc[SCAN_ITEMS];
    unsigned long long s = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        loc[i] = s;
        s += tile[k0 + i];
    }
    unsigned long long tot;
    unsigned long long ex = block_excl_scan_u64(s, ws, tot);
    unsigned long long off = sums[blockIdx.x] + ex;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) tile[k0 + i] = off + loc[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        const int k = i * SCAN_THREADS + threadIdx.x;
        const uint64_t j = base + k;
        if (j < n) out[j] = (int64_t)tile[k + k / 32];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
        uint64_t tiles = gridDim.x;
        out[n] = (int64_t)sums[tiles];
    }
}

// out[0..n] = exclusive prefix of in[0..n), out[n] = total.
int exclusive_scan_u32_i64(const uint32_t *d_in, int64_t *d_out, uint64_t n, cudaStream_t s) {
    uint64_t tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    if (tiles == 0) {
        KC_CUDA(cudaMemsetAsync(d_out, 0, sizeof(int64_t), s));
        return KC_OK;
    }
    unsigned long long *sums = nullptr;
    KC_TRY(dalloc(&sums, tiles + 1, "scan sums"));
    scan_tile_sums<<<(unsigned)tiles, SCAN_THREADS, 0, s>>>(d_in, n, sums);
    scan_sums_single<<<1, 1024, 0, s>>>(sums, tiles);
    scan_tile_apply<<<(unsigned)tiles, SCAN_THREADS, 0, s>>>(d_in, d_out, n, sums);
    cudaError_t e = cudaGetLastError();
    cudaStreamSynchronize(s);
    dfree(sums);
    if (e != cudaSuccess) return fail(KC_ERR_CUDA, "scan launch: %s", cudaGetErrorString(e));
    return KC_OK;
}

// ------------------------------------------------------- count/scatter ----
__global__ void count_degrees(const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst, uint64_t m,
                              uint32_t n, uint32_t *deg, unsigned int *err) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t a = src[i], b = dst[i];
        if (a >= n || b >= n) {
            atomicCAS(err, 0u, 1u);
            continue;
        }
        if (a == b) continue;
        atomicAdd(&deg[a], 1u);
        atomicAdd(&deg[b], 1u);
    }
}

// cur: 64-bit row cursors preset to the row offsets, so one atomic gives an
// entry's position with no row-offset read (random 8-byte reads of rowptr
// were a third of this kernel's gathers: 8% of the C3 build measured).
__global__ void scatter_edges(const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst, uint64_t m,
                              uint32_t n, unsigned long long *cur, uint32_t *col) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t a = src[i], b = dst[i];
        if (a >= n || b >= n || a == b) continue;
        const unsigned long long pa = atomicAdd(&cur[a], 1ull);
        const unsigned long long pb = atomicAdd(&cur[b], 1ull);
        col[pa] = b;
        col[pb] = a;
    }
}

// ----------------------------------------------- partitioned count/scatter ----
// The degree count and the scatter above make two random L2 atomics and one
// random 4-byte write per entry (R-MAT 22: 1.90 + 3.15 ms, the atomics at 70 G/s).
// Where the order within a row is free, the entries are first partitioned by
// ranges of 2^shift rows ("buckets", at most PART_MAX_BUCKETS), so that counts,
// cursors and ranks can be kept in shared memory:
//   part_hist    entries per bucket (a shared-memory histogram per CTA);
//   part_plan    bucket bases, and the buckets cut into tiles of PART_TILE entries;
//   part_pairs   (row, column) pairs grouped by bucket: a tile of edges is
//                grouped in shared memory and written out bucket by bucket;
//   part_degrees row counts of every tile, added to the degrees (one atomic per
//                row of a tile; a bucket of one tile writes them), and where in
//                its row each tile's share begins;
//   part_rows    every tile sorts its columns by row in shared memory and writes
//                them out row by row.
// What bounds it is memory and the shared-memory atomics: the pairs are written
// once and read twice, each time with one atomic per entry (6 G/s per SM).
// R-MAT 22 (134 M entries): 0.12 + 0.62 + 0.21 + 0.60 ms and 0.03 ms of scans,
// where counting and scattering took 5.05 ms.
constexpr int PART_THREADS = 512;
// part_pairs groups 8,192 edges at a time: 8 pairs (two sectors) per bucket on
// average with 2,048 buckets, one CTA per SM.  Half as many edges, two CTAs per
// SM: whole builds of R-MAT 22 4.25 ms instead of 4.13, of a uniform random
// graph of 10^6 vertices and 16 M edges 1.15 instead of 1.05.
constexpr int PAIR_THREADS = 1024;
constexpr int PART_PER = 8;                                // edges per thread
constexpr uint32_t PART_EDGES = PAIR_THREADS * PART_PER;
constexpr uint32_t PART_TILE = 32768;                      // entries per tile of a bucket
constexpr uint32_t PART_MAX_BUCKETS = 4096;
constexpr int PART_MAX_SHIFT = 14;                         // 64 KB of row counters

struct PartPlan {
    uint64_t *base;    // [buckets + 1] first pair of each bucket
    uint64_t *cursor;  // [buckets]     next free pair while partitioning
    uint32_t *tile;    // [buckets + 1] first tile of each bucket
    uint32_t *off;     // [tiles << shift] where each tile's share of a row begins (unset where it has none)
    uint16_t *count;   // [tiles << shift] and how long it is (a tile has 32,768 entries)
    uint32_t buckets;
    int shift;
};

__global__ void __launch_bounds__(1024) part_hist(const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst,
                                                  uint64_t m, uint32_t n, PartPlan plan, unsigned int *err) {
    extern __shared__ uint32_t h[];
    for (uint32_t b = threadIdx.x; b < plan.buckets; b += blockDim.x) h[b] = 0;
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < m; i0 += 4 * stride) {
        uint32_t a[4], b[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint64_t i = i0 + k * stride;
            a[k] = i < m ? src[i] : 0u;
            b[k] = i < m ? dst[i] : 0u;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) {
            if (a[k] >= n || b[k] >= n) {
                if (i0 + k * stride < m) atomicCAS(err, 0u, 1u);
                continue;
            }
            if (a[k] == b[k]) continue;
            atomicAdd(&h[a[k] >> plan.shift], 1u);
            atomicAdd(&h[b[k] >> plan.shift], 1u);
        }
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < plan.buckets; b += blockDim.x)
        if (h[b]) atomicAdd(reinterpret_cast<unsigned long long *>(&plan.base[b]), (unsigned long long)h[b]);
}

// base: counts -> exclusive prefix; cursor: a copy; tile: prefix of the tile counts.
__global__ void __launch_bounds__(1024) part_plan(PartPlan plan) {
    __shared__ unsigned long long ws[33];
    constexpr uint32_t PER = PART_MAX_BUCKETS / 1024;
    unsigned long long c[PER], e = 0, t = 0;
    const uint32_t b0 = threadIdx.x * PER;
#pragma unroll
    for (uint32_t k = 0; k < PER; k++) {
        c[k] = b0 + k < plan.buckets ? plan.base[b0 + k] : 0ull;
        e += c[k];
        t += (c[k] + PART_TILE - 1) / PART_TILE;
    }
    unsigned long long etot, ttot;
    unsigned long long eat = block_excl_scan_u64(e, ws, etot);
    unsigned long long tat = block_excl_scan_u64(t, ws, ttot);
#pragma unroll
    for (uint32_t k = 0; k < PER; k++) {
        if (b0 + k < plan.buckets) {
            plan.base[b0 + k] = plan.cursor[b0 + k] = eat;
            plan.tile[b0 + k] = (uint32_t)tat;
        }
        eat += c[k];
        tat += (c[k] + PART_TILE - 1) / PART_TILE;
    }
    if (threadIdx.x == 0) {
        plan.base[plan.buckets] = etot;
        plan.tile[plan.buckets] = (uint32_t)ttot;
    }
}

// Shared memory: pairs of a tile, then per bucket the distance from a pair's
// place in the tile to its place in the output, and the bucket's count.
__global__ void __launch_bounds__(PAIR_THREADS) part_pairs(const uint32_t *__restrict__ src,
                                                           const uint32_t *__restrict__ dst, uint64_t m, uint32_t n,
                                                           PartPlan plan, uint2 *pairs) {
    extern __shared__ __align__(16) unsigned char part_sm[];
    uint2 *stage = reinterpret_cast<uint2 *>(part_sm);
    unsigned long long *delta = reinterpret_cast<unsigned long long *>(stage + 2 * PART_EDGES);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(delta + plan.buckets);
    __shared__ uint32_t wsum[PAIR_THREADS / 32];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t per = (plan.buckets + PAIR_THREADS - 1) / PAIR_THREADS;
    for (uint64_t t0 = (uint64_t)blockIdx.x * PART_EDGES; t0 < m; t0 += (uint64_t)gridDim.x * PART_EDGES) {
        for (uint32_t b = threadIdx.x; b < plan.buckets; b += PAIR_THREADS) cnt[b] = 0;
        uint32_t a[PART_PER], b[PART_PER];
#pragma unroll
        for (int k = 0; k < PART_PER; k++) {
            const uint64_t i = t0 + (uint64_t)k * PAIR_THREADS + threadIdx.x;
            a[k] = i < m ? src[i] : 0u;
            b[k] = i < m ? dst[i] : 0u;
        }
        __syncthreads();
        uint32_t rank[PART_PER];  // of both directions, 16 bits each (a tile has 16,384 pairs)
#pragma unroll
        for (int k = 0; k < PART_PER; k++) {
            rank[k] = 0;
            if (a[k] >= n || b[k] >= n || a[k] == b[k]) {
                a[k] = b[k] = 0;  // not an entry
            } else {
                rank[k] = atomicAdd(&cnt[a[k] >> plan.shift], 1u);
                rank[k] |= atomicAdd(&cnt[b[k] >> plan.shift], 1u) << 16;
            }
        }
        __syncthreads();
        // exclusive prefix of the counts; each bucket's pairs are reserved in
        // the output with one atomic
        constexpr uint32_t PER = PART_MAX_BUCKETS / PAIR_THREADS;
        const uint32_t b0 = threadIdx.x * per;
        uint32_t c[PER], own = 0;
        unsigned long long to[PER];
#pragma unroll
        for (uint32_t k = 0; k < PER; k++) {
            c[k] = k < per && b0 + k < plan.buckets ? cnt[b0 + k] : 0u;
            own += c[k];
        }
#pragma unroll
        for (uint32_t k = 0; k < PER; k++)
            to[k] = c[k] ? atomicAdd(reinterpret_cast<unsigned long long *>(&plan.cursor[b0 + k]), (unsigned long long)c[k]) : 0ull;
        uint32_t wtot;
        uint32_t at = warp_excl_scan(own, lane, wtot);
        if (lane == 0) wsum[warp] = wtot;
        __syncthreads();
        const uint32_t ws = lane < PAIR_THREADS / 32 ? wsum[lane] : 0u;
        at += __reduce_add_sync(KC_FULL_MASK, lane < warp ? ws : 0u);
        const uint32_t total = __reduce_add_sync(KC_FULL_MASK, ws);
#pragma unroll
        for (uint32_t k = 0; k < PER; k++)
            if (c[k]) {
                delta[b0 + k] = to[k] - at;
                cnt[b0 + k] = at;
                at += c[k];
            }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < PART_PER; k++)
            if (a[k] != b[k]) {
                stage[cnt[a[k] >> plan.shift] + (rank[k] & 0xffffu)] = make_uint2(a[k], b[k]);
                stage[cnt[b[k] >> plan.shift] + (rank[k] >> 16)] = make_uint2(b[k], a[k]);
            }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < total; i += PAIR_THREADS) {
            const uint2 q = stage[i];
            pairs[delta[q.x >> plan.shift] + i] = q;
        }
        __syncthreads();
    }
}

// The bucket of tile t, and its pairs [lo, hi).
__device__ __forceinline__ uint32_t part_tile(const PartPlan &plan, uint32_t t, uint64_t &lo, uint64_t &hi) {
    uint32_t b = 0, e = plan.buckets;  // last bucket with tile[b] <= t
    while (e - b > 1) {
        const uint32_t mid = (b + e) >> 1;
        if (plan.tile[mid] <= t) b = mid;
        else e = mid;
    }
    lo = plan.base[b] + (uint64_t)(t - plan.tile[b]) * PART_TILE;
    hi = min(plan.base[b + 1], lo + PART_TILE);
    return b;
}

__global__ void __launch_bounds__(PART_THREADS) part_degrees(const uint2 *__restrict__ pairs, PartPlan plan,
                                                             uint32_t n, uint32_t *deg) {
    extern __shared__ uint32_t rows_sm[];
    const uint32_t rows = 1u << plan.shift;
    const uint32_t tiles = plan.tile[plan.buckets];
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        uint64_t lo, hi;
        const uint32_t b = part_tile(plan, t, lo, hi);
        const bool alone = plan.tile[b + 1] - plan.tile[b] == 1;
        for (uint32_t i = threadIdx.x; i < rows; i += PART_THREADS) rows_sm[i] = 0;
        __syncthreads();
#pragma unroll 4
        for (uint64_t e = lo + threadIdx.x; e < hi; e += PART_THREADS) atomicAdd(&rows_sm[pairs[e].x & (rows - 1)], 1u);
        __syncthreads();
        const uint64_t r0 = (uint64_t)b << plan.shift;
        for (uint32_t i = threadIdx.x; i < rows && r0 + i < n; i += PART_THREADS) {
            const uint32_t c = rows_sm[i];
            const uint64_t at = ((uint64_t)t << plan.shift) + i;
            plan.count[at] = (uint16_t)c;
            if (!c) continue;
            if (alone) deg[r0 + i] = c;
            plan.off[at] = alone ? 0u : atomicAdd(&deg[r0 + i], c);
        }
        __syncthreads();
    }
}

// With up to PART_STAGE_ROWS rows per bucket a tile is put in row order in shared
// memory first (its columns, and the row of each), so that the entries of a row
// leave together: 16 on average with 2,048 rows, 7 to 8 sectors a warp instead
// of 32.  R-MAT 22 (134 M entries): 1.17 -> 0.60 ms; the direct form, one cursor
// per row in shared memory, stays for more rows, where the counters leave no
// room for a tile and its entries share few rows.
constexpr uint32_t PART_STAGE_ROWS = 4096;
constexpr size_t part_rows_smem(int shift) {
    return (1u << shift) <= PART_STAGE_ROWS ? (size_t)PART_TILE * 6 + ((size_t)8 << shift) : (size_t)4 << shift;
}
template <bool STAGE>
__global__ void __launch_bounds__(STAGE ? 1024 : PART_THREADS) part_rows(const uint2 *__restrict__ pairs, PartPlan plan,
                                                                         uint32_t n, const int64_t *__restrict__ rowptr,
                                                                         uint32_t *col) {
    extern __shared__ __align__(16) unsigned char part_sm[];
    constexpr uint32_t NT = STAGE ? 1024 : PART_THREADS;
    const uint32_t rows = 1u << plan.shift;
    uint32_t *cur = reinterpret_cast<uint32_t *>(part_sm);  // next place of each row
    // staged: distance from a place in the tile to the place in the bucket, per
    // row; the tile's columns and rows in row order
    uint32_t *delta = cur + rows, *stage = delta + rows;
    uint16_t *row_of = reinterpret_cast<uint16_t *>(stage + PART_TILE);
    __shared__ uint32_t wsum[NT / 32];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t tiles = plan.tile[plan.buckets];
    for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        uint64_t lo, hi;
        const uint32_t b = part_tile(plan, t, lo, hi);
        const uint64_t base = plan.base[b];  // the bucket's rows hold entries [base, base of the next)
        const uint64_t r0 = (uint64_t)b << plan.shift, t0 = (uint64_t)t << plan.shift;
        if constexpr (STAGE) {
            constexpr uint32_t PER = PART_STAGE_ROWS / NT;
            const uint32_t per = (rows + NT - 1) / NT, i0 = threadIdx.x * per;
            uint32_t c[PER], own = 0;
#pragma unroll
            for (uint32_t k = 0; k < PER; k++) {
                c[k] = k < per && i0 + k < rows && r0 + i0 + k < n ? plan.count[t0 + i0 + k] : 0u;
                own += c[k];
            }
            uint32_t wtot;
            uint32_t at = warp_excl_scan(own, lane, wtot);
            if (lane == 0) wsum[warp] = wtot;
            __syncthreads();
            at += __reduce_add_sync(KC_FULL_MASK, lane < warp ? wsum[lane] : 0u);
#pragma unroll
            for (uint32_t k = 0; k < PER; k++)
                if (c[k]) {
                    cur[i0 + k] = at;
                    delta[i0 + k] = (uint32_t)((uint64_t)rowptr[r0 + i0 + k] - base) + plan.off[t0 + i0 + k] - at;
                    at += c[k];
                }
            __syncthreads();
#pragma unroll 4
            for (uint64_t e = lo + threadIdx.x; e < hi; e += NT) {
                const uint2 q = pairs[e];
                const uint32_t r = q.x & (rows - 1), p = atomicAdd(&cur[r], 1u);
                stage[p] = q.y;
                row_of[p] = (uint16_t)r;
            }
            __syncthreads();
            const uint32_t len = (uint32_t)(hi - lo);
#pragma unroll 4
            for (uint32_t i = threadIdx.x; i < len; i += NT) col[base + (uint32_t)(delta[row_of[i]] + i)] = stage[i];
        } else {
            for (uint32_t i = threadIdx.x; i < rows && r0 + i < n; i += NT)
                if (plan.count[t0 + i]) cur[i] = (uint32_t)((uint64_t)rowptr[r0 + i] - base) + plan.off[t0 + i];
            __syncthreads();
#pragma unroll 4
            for (uint64_t e = lo + threadIdx.x; e < hi; e += NT) {
                const uint2 q = pairs[e];
                col[base + atomicAdd(&cur[q.x & (rows - 1)], 1u)] = q.y;
            }
        }
        __syncthreads();
    }
}

// Rows per bucket for n vertices (as a shift), or -1 where partitioning does not
// apply: fewer edges than PART_MIN_EDGES (the atomics' lines stay in L2 and the
// launches cost more; R-MAT 16, 1.05 M edges: 0.54 ms without, 0.52 with), more rows than the
// buckets cover, more than PART_MAX_ROWS rows per edge (the tiles' row counters
// then outweigh the edges: 2^26 vertices, 2^20 edges de-duplicated 2.5 ms with,
// 2.0 without; 2^22 edges sorted 1.7 with, 2.1 without), or more entries than a
// 32-bit offset within a bucket holds.
constexpr uint64_t PART_MIN_EDGES = 1u << 20, PART_MAX_ROWS = 16;
static int part_shift(uint64_t m, uint32_t n) {
    if (m < PART_MIN_EDGES || 2 * m >= 0xffffffffull || n > PART_MAX_ROWS * m) return -1;
    int shift = 6;
    while (shift < PART_MAX_SHIFT && ((n - 1) >> shift) + 1 > PART_MAX_BUCKETS / 2) shift++;
    return ((n - 1) >> shift) + 1 <= PART_MAX_BUCKETS ? shift : -1;
}

static int part_smem_limits() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    KC_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(KC_ERR_INVALID, "device %d out of range", dev);
    std::lock_guard<std::mutex> lk(mu);
    if (done[dev]) return KC_OK;
    const int rows = 4 << PART_MAX_SHIFT;
    KC_CUDA(cudaFuncSetAttribute(part_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(2 * PART_EDGES * sizeof(uint2) + PART_MAX_BUCKETS * 12)));
    KC_CUDA(cudaFuncSetAttribute(part_degrees, cudaFuncAttributeMaxDynamicSharedMemorySize, rows));
    KC_CUDA(cudaFuncSetAttribute(part_rows<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, rows));
    int most = 0;
    for (int shift = 0; 1u << shift <= PART_STAGE_ROWS; shift++) most = (int)part_rows_smem(shift);
    KC_CUDA(cudaFuncSetAttribute(part_rows<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    done[dev] = true;
    return KC_OK;
}

// ------------------------------------------------ edge-list row order ----
// Rows in the order of the edge list (both directions of line i at places 2 i
// and 2 i + 1 of the sequence): a stable LSD radix sort of the entries by row,
// two passes of up to 11 bits (one below 2^11 rows, three above 2^22), each
//   order_hist   digit counts of every CTA's stretch of the sequence,
//   order_scan   their prefixes over the stretches, and each digit's total,
//   order_place  entries to their places: a warp ranks its 256 entries of a
//                tile 32 at a time (lanes of one digit find each other), the
//                warps' counts are added up per digit, the tile is grouped by
//                digit in shared memory and written out run by run, and the
//                stretch's offsets move on from tile to tile.
// The first pass reads the edge list, the last writes columns and rows.  What
// bounds it is the chain of the ranking (a match and a shared-memory counter
// per 32 entries); writing each entry from where it was ranked instead of by
// runs made eight times the requests (R-MAT 18: 126 us a pass, 84 us now).
// Counting, scattering with atomics and sorting every row by line number took
// 1.24 ms of kernels on R-MAT 18 (4.2 M lines), these passes take 0.28 ms.
constexpr int ORDER_THREADS = 1024;
constexpr int ORDER_WARPS = ORDER_THREADS / 32;
constexpr int ORDER_STEPS = 8;                                    // of 32 entries, per warp and tile
constexpr uint32_t ORDER_TILE = ORDER_THREADS * ORDER_STEPS;      // entries
constexpr int ORDER_MAX_BITS = 11;

struct OrderPass {
    const uint32_t *src, *dst;  // first pass: the edge list
    const uint2 *in;            // later passes: (row, column) pairs
    uint64_t count;             // places of the sequence (first pass: 2 per line)
    uint64_t stretch;           // places per CTA, whole tiles
    uint32_t n;
    uint32_t row0, rows;        // first pass: entries of rows [row0, row0 + rows); pairs count rows from row0
    int shift, bits;
    uint32_t *hist;             // [CTAs][2^bits]
    uint32_t *total;            // [2^bits]
};

// Place e of the sequence; false where it holds no entry of these rows (a
// self-loop, a bad id, another row).
template <bool EDGES>
__device__ __forceinline__ bool order_entry(const OrderPass &P, uint64_t e, uint32_t &row, uint32_t &col) {
    if (e >= P.count) return false;
    if (EDGES) {
        const uint32_t a = P.src[e >> 1], b = P.dst[e >> 1];
        row = (e & 1 ? b : a) - P.row0;
        col = e & 1 ? a : b;
        return a != b && row < P.rows && col < P.n;  // the rows are below n
    }
    const uint2 q = P.in[e];
    row = q.x;
    col = q.y;
    return true;
}

template <bool EDGES>
__global__ void __launch_bounds__(ORDER_THREADS) order_hist(OrderPass P, unsigned int *err) {
    extern __shared__ uint32_t order_sm[];
    const uint32_t bins = 1u << P.bits;
    for (uint32_t d = threadIdx.x; d < bins; d += ORDER_THREADS) order_sm[d] = 0;
    __syncthreads();
    const uint64_t lo = blockIdx.x * P.stretch, hi = min(P.count, lo + P.stretch);
#pragma unroll 4
    for (uint64_t e = lo + threadIdx.x; e < hi; e += ORDER_THREADS) {
        uint32_t row = 0, col = 0;
        if (order_entry<EDGES>(P, e, row, col)) atomicAdd(&order_sm[(row >> P.shift) & (bins - 1)], 1u);
        else if (EDGES && err && (row >= P.n || col >= P.n)) atomicCAS(err, 0u, 1u);  // row0 is 0 where err is set
    }
    __syncthreads();
    for (uint32_t d = threadIdx.x; d < bins; d += ORDER_THREADS) P.hist[(uint64_t)blockIdx.x * bins + d] = order_sm[d];
}

// One lane per digit, 32 digits per CTA; the warps share the stretches.
__global__ void __launch_bounds__(1024) order_scan(OrderPass P, uint32_t ctas, unsigned long long *entries) {
    __shared__ uint32_t part[32][33];
    const uint32_t bins = 1u << P.bits;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t d = blockIdx.x * 32 + lane;
    const uint32_t per = (ctas + 31) / 32, c0 = warp * per, c1 = min(ctas, c0 + per);
    uint32_t sum = 0;
    if (d < bins)
        for (uint32_t c = c0; c < c1; c++) sum += P.hist[(uint64_t)c * bins + d];
    part[warp][lane] = sum;
    __syncthreads();
    uint32_t run = 0, all = 0;
    for (unsigned w = 0; w < 32; w++) {
        run += w < warp ? part[w][lane] : 0u;
        all += part[w][lane];
    }
    if (d < bins) {
        for (uint32_t c = c0; c < c1; c++) {
            const uint32_t x = P.hist[(uint64_t)c * bins + d];
            P.hist[(uint64_t)c * bins + d] = run;
            run += x;
        }
        if (warp == 0) P.total[d] = all;
    }
    if (warp == 0 && entries) {
        const uint32_t t = __reduce_add_sync(KC_FULL_MASK, d < bins ? all : 0u);  // at most 2^32 - 1 entries in all
        if (lane == 0 && t) atomicAdd(entries, (unsigned long long)t);
    }
}

// Shared memory: the tile's entries, per digit its first place in the tile, its
// next place in the output and the distance between the two, then a 16-bit
// count per warp and digit.
template <bool EDGES, bool LAST>
__global__ void __launch_bounds__(ORDER_THREADS) order_place(OrderPass P, uint2 *out, uint32_t *col_out,
                                                             uint32_t *row_out) {
    extern __shared__ __align__(16) uint32_t order_sm[];
    const uint32_t bins = 1u << P.bits;
    uint2 *stage = reinterpret_cast<uint2 *>(order_sm);
    uint32_t *first = order_sm + 2 * ORDER_TILE, *off = first + bins, *delta = off + bins;
    uint16_t *wc = reinterpret_cast<uint16_t *>(delta + bins);  // [warp][digit]
    __shared__ uint32_t wsum[ORDER_WARPS];
    constexpr uint32_t PER = (1u << ORDER_MAX_BITS) / ORDER_THREADS;  // digits per thread
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t d0 = threadIdx.x * PER;
    // CTA-wide exclusive prefix of one number per thread
    auto prefix = [&](uint32_t x, uint32_t &total) {
        uint32_t wtot;
        const uint32_t at = warp_excl_scan(x, lane, wtot);
        if (lane == 0) wsum[warp] = wtot;
        __syncthreads();
        const uint32_t ws = wsum[lane];  // 32 warps
        total = __reduce_add_sync(KC_FULL_MASK, ws);
        return at + __reduce_add_sync(KC_FULL_MASK, lane < warp ? ws : 0u);
    };
    // offsets: entries of smaller digits, and of this digit in earlier stretches
    uint32_t own = 0, all;
#pragma unroll
    for (uint32_t k = 0; k < PER; k++) own += d0 + k < bins ? P.total[d0 + k] : 0u;
    uint32_t at = prefix(own, all);
#pragma unroll
    for (uint32_t k = 0; k < PER; k++)
        if (d0 + k < bins) {
            off[d0 + k] = at + P.hist[(uint64_t)blockIdx.x * bins + d0 + k];
            at += P.total[d0 + k];
        }
    uint16_t *mine = wc + warp * bins;
    const uint64_t lo = blockIdx.x * P.stretch, hi = min(P.count, lo + P.stretch);
    for (uint64_t t0 = lo; t0 < hi; t0 += ORDER_TILE) {
        uint32_t row[ORDER_STEPS], col[ORDER_STEPS], rank[ORDER_STEPS];
        unsigned valid = 0;
#pragma unroll
        for (int k = 0; k < ORDER_STEPS; k++) {
            const uint64_t e = t0 + warp * (32 * ORDER_STEPS) + k * 32 + lane;
            row[k] = col[k] = 0;
            if (e < hi && order_entry<EDGES>(P, e, row[k], col[k])) valid |= 1u << k;
        }
        for (uint32_t d = lane; d < bins / 2; d += 32) reinterpret_cast<uint32_t *>(mine)[d] = 0;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < ORDER_STEPS; k++) {
            const bool on = (valid >> k) & 1u;
            const uint32_t d = on ? (row[k] >> P.shift) & (bins - 1) : bins;
            // lanes with the same digit, bit by bit (__match_any_sync: 13 us slower a pass)
            unsigned peers = __ballot_sync(KC_FULL_MASK, on);
            if (!on) peers = ~peers;
            for (int b = 0; b < P.bits; b++) {
                const unsigned vote = __ballot_sync(KC_FULL_MASK, (d >> b) & 1u);
                peers &= ((d >> b) & 1u) ? vote : ~vote;
            }
            const int leader = __ffs(peers) - 1;
            uint32_t before = 0;
            if (on && (int)lane == leader) {
                before = mine[d];
                mine[d] = (uint16_t)(before + __popc(peers));
            }
            __syncwarp();
            rank[k] = __shfl_sync(KC_FULL_MASK, before, leader) + __popc(peers & ((1u << lane) - 1u));
        }
        __syncthreads();
        // counts -> counts of the warps before; the digits' runs in the tile
        uint32_t runs[PER];
        own = 0;
#pragma unroll
        for (uint32_t k = 0; k < PER; k++) {
            runs[k] = 0;
            if (d0 + k >= bins) continue;
#pragma unroll 8
            for (int w = 0; w < ORDER_WARPS; w++) {
                const uint32_t c = wc[w * bins + d0 + k];
                wc[w * bins + d0 + k] = (uint16_t)runs[k];
                runs[k] += c;
            }
            own += runs[k];
        }
        uint32_t total;
        at = prefix(own, total);
#pragma unroll
        for (uint32_t k = 0; k < PER; k++)
            if (d0 + k < bins) {
                first[d0 + k] = at;
                delta[d0 + k] = off[d0 + k] - at;
                off[d0 + k] += runs[k];
                at += runs[k];
            }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < ORDER_STEPS; k++) {
            if (!((valid >> k) & 1u)) continue;
            const uint32_t d = (row[k] >> P.shift) & (bins - 1);
            stage[first[d] + mine[d] + rank[k]] = make_uint2(row[k], col[k]);
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < total; i += ORDER_THREADS) {
            const uint2 q = stage[i];
            const uint32_t to = delta[(q.x >> P.shift) & (bins - 1)] + i;
            if (LAST) {
                col_out[to] = q.y;
                row_out[to] = q.x;
            } else {
                out[to] = q;
            }
        }
        __syncthreads();
    }
}

// Degrees from the rows of the sorted entries: last place + 1 less first place.
__global__ void order_degrees(const uint32_t *__restrict__ rows, uint64_t nnz, uint32_t *deg) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nnz; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t r = rows[i];
        if (i == 0 || rows[i - 1] != r) atomicSub(&deg[r], (uint32_t)i);
        if (i + 1 == nnz || rows[i + 1] != r) atomicAdd(&deg[r], (uint32_t)(i + 1));
    }
}

static size_t order_smem(int bits) { return 8 * ORDER_TILE + ((size_t)12 << bits) + ((size_t)2 * ORDER_WARPS << bits); }

static int order_smem_limits() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    KC_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(KC_ERR_INVALID, "device %d out of range", dev);
    std::lock_guard<std::mutex> lk(mu);
    if (done[dev]) return KC_OK;
    const int most = (int)order_smem(ORDER_MAX_BITS);
    KC_CUDA(cudaFuncSetAttribute(order_place<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    KC_CUDA(cudaFuncSetAttribute(order_place<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    KC_CUDA(cudaFuncSetAttribute(order_place<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    KC_CUDA(cudaFuncSetAttribute(order_place<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    done[dev] = true;
    return KC_OK;
}

struct OrderBuild {
    Graph *g;
    const uint32_t *src, *dst;
    uint64_t m;
    uint64_t stretches;         // CTAs of a pass, at most: one per SM
    uint32_t *hist = nullptr, *deg = nullptr, *rows = nullptr;
    unsigned long long *state = nullptr;  // entries, error flag
    uint2 *buf[2] = {nullptr, nullptr};
    uint64_t done = 0;          // entries placed

    // the sort that used them has ended
    void free_sort() {
        dfree(rows);
        dfree(buf[0]);
        dfree(buf[1]);
        rows = nullptr;
        buf[0] = buf[1] = nullptr;
    }
    ~OrderBuild() {
        cudaStreamSynchronize(g->stream);
        free_sort();
        dfree(hist);
        dfree(deg);
        dfree(state);
    }
};

// Sorts the entries of rows [row0, row0 + rows) behind those already placed.
// All rows at once (row0 = 0, rows = n) also checks the ids and allocates the
// columns.  The sort takes 4 bytes per entry for the rows, 8 for the pairs (from
// 2^11 rows up) and 8 more above 2^22 rows, beside the 4 of the columns; where
// they are not free, the two halves of the rows follow one after the other, each
// reading the whole edge list.
static int order_range(OrderBuild &B, uint32_t row0, uint32_t rows) {
    Graph *g = B.g;
    cudaStream_t s = g->stream;
    const bool all = row0 == 0 && rows == g->n;
    int bits = 1;
    while (bits < 32 && ((uint64_t)rows - 1) >> bits) bits++;
    const int passes = (bits + ORDER_MAX_BITS - 1) / ORDER_MAX_BITS;
    const int digit = (bits + passes - 1) / passes;
    unsigned long long h[2] = {0, 0};
    // a list of self-loops alone leaves nothing to sort, and no tile to divide by
    for (int p = 0; p < passes && (p == 0 || h[0]); p++) {
        OrderPass P{};
        P.src = B.src;
        P.dst = B.dst;
        P.in = B.buf[(p + 1) & 1];
        P.count = p ? h[0] : 2 * B.m;
        P.n = g->n;
        P.row0 = row0;
        P.rows = rows;
        P.shift = p * digit;
        P.bits = std::min(digit, bits - P.shift);
        const uint64_t tiles = (P.count + ORDER_TILE - 1) / ORDER_TILE;
        const uint64_t per = (tiles + B.stretches - 1) / B.stretches;
        P.stretch = per * ORDER_TILE;
        const uint32_t ctas = (uint32_t)((tiles + per - 1) / per);
        P.hist = B.hist;
        P.total = B.hist + (B.stretches << ORDER_MAX_BITS);
        const size_t sm = order_smem(P.bits);
        const size_t hist_sm = (size_t)4 << P.bits;
        const uint32_t scan_ctas = ((1u << P.bits) + 31) / 32;
        const bool last = p + 1 == passes;
        uint32_t *col = g->col ? g->col + B.done : nullptr;
        if (p == 0) {
            if (!all) cudaMemsetAsync(B.state, 0, 16, s);
            order_hist<true><<<ctas, ORDER_THREADS, hist_sm, s>>>(P, all ? reinterpret_cast<unsigned int *>(B.state + 1) : nullptr);
            order_scan<<<scan_ctas, 1024, 0, s>>>(P, ctas, B.state);
            cudaMemcpyAsync(h, B.state, 16, cudaMemcpyDeviceToHost, s);
            cudaError_t e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) return fail(KC_ERR_CUDA, "degree count: %s", cudaGetErrorString(e));
            if (h[1]) return fail(KC_ERR_INVALID, "edge endpoint >= n (%u)", g->n);
            if (all) {
                g->nnz = h[0];
                KC_TRY(dalloc(&g->col, g->nnz + 1, "column ids"));
                col = g->col;
            }
            B.free_sort();  // of the rows before, which the wait above covers
            int rc = dalloc(&B.rows, h[0] + 1, "row ids");
            if (!rc && passes > 1) rc = dalloc(&B.buf[0], h[0] + 1, "ordered pairs");
            if (!rc && passes > 2) rc = dalloc(&B.buf[1], h[0] + 1, "ordered pairs");
            if (rc == KC_ERR_NOMEM && rows > 1) {
                clear_error();
                B.free_sort();
                KC_TRY(order_range(B, row0, rows / 2));
                return order_range(B, row0 + rows / 2, rows - rows / 2);
            }
            if (rc) return rc;
            if (last) order_place<true, true><<<ctas, ORDER_THREADS, sm, s>>>(P, nullptr, col, B.rows);
            else order_place<true, false><<<ctas, ORDER_THREADS, sm, s>>>(P, B.buf[0], nullptr, nullptr);
        } else {
            order_hist<false><<<ctas, ORDER_THREADS, hist_sm, s>>>(P, nullptr);
            order_scan<<<scan_ctas, 1024, 0, s>>>(P, ctas, nullptr);
            if (last) order_place<false, true><<<ctas, ORDER_THREADS, sm, s>>>(P, nullptr, col, B.rows);
            else order_place<false, false><<<ctas, ORDER_THREADS, sm, s>>>(P, B.buf[p & 1], nullptr, nullptr);
        }
    }
    if (h[0]) order_degrees<<<grid_for(h[0], 256, g->sm_count), 256, 0, s>>>(B.rows, h[0], B.deg + row0);
    B.done += h[0];
    return KC_OK;
}

// Builds g's rows in edge-list order (m > 0).
static int build_in_order(Graph *g, const uint32_t *d_src, const uint32_t *d_dst, uint64_t m, uint32_t n) {
    cudaStream_t s = g->stream;
    OrderBuild B;
    B.g = g;
    B.src = d_src;
    B.dst = d_dst;
    B.m = m;
    B.stretches = (uint64_t)g->sm_count;
    KC_TRY(order_smem_limits());
    KC_TRY(dalloc(&B.hist, (B.stretches + 1) << ORDER_MAX_BITS, "digit counts"));
    KC_TRY(dalloc(&B.state, 2, "entry count"));
    KC_TRY(dalloc(&B.deg, (uint64_t)n + 1, "degrees"));
    // ahead of the larger one, so that the first kernel follows it at once
    cudaMemsetAsync(B.state, 0, 16, s);
    cudaMemsetAsync(B.deg, 0, ((uint64_t)n + 1) * 4, s);
    KC_TRY(order_range(B, 0, n));
    KC_TRY(exclusive_scan_u32_i64(B.deg, g->rowptr, n, s));
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(KC_ERR_CUDA, "ordered rows: %s", cudaGetErrorString(e));
    return KC_OK;
}

// ------------------------------------------------------ segmented sort ----
// Rows are sorted by size class: up to 8, 16 and 32 entries four, two and one
// to a warp (shuffle bitonic networks); 33..4096 entries padded to P = 2^k
// (k = 6..12) and sorted in registers, by one to four warps a row; longer rows
// one CTA per row, with a bitmap where repeated entries are dropped anyway and
// an LSD radix sort elsewhere.
constexpr uint32_t CLASS_B_MAX = 4096;
constexpr int SORT_SHORT = 3;     // classes of at most 32 entries
constexpr int SORT_BUCKETS = 11;  // 0..2: <= 8, 16, 32; 3..9: P = 64..4096; 10: > 4096
constexpr int CLASSIFY_THREADS = 512;

__device__ __forceinline__ int sort_bucket(int64_t len) {
    if (len < 2) return -1;
    if (len <= 8) return 0;
    if (len > (int64_t)CLASS_B_MAX) return SORT_BUCKETS - 1;
    return 29 - __clz((int)len - 1);  // 9..16 -> 1, 17..32 -> 2, 33..64 -> 3, ..
}

// Pass 1 (cursor == nullptr): rows per bucket into counts.  Pass 2: each row
// id goes to list[cursor[bucket]++] (cursors start at the buckets' offsets).
// The CTA counts in shared memory and makes one atomic per bucket: all of it
// in pass 1, per 512 rows in pass 2 (one per warp and bucket took 0.17 ms a
// pass on 4.2 M rows, 0.02 ms now).
__global__ void __launch_bounds__(CLASSIFY_THREADS) classify_rows(const int64_t *__restrict__ rowptr, uint32_t n,
                                                                  unsigned long long *counts,
                                                                  unsigned long long *cursor, uint32_t *list) {
    __shared__ unsigned int cnt[SORT_BUCKETS];
    __shared__ unsigned long long base[SORT_BUCKETS];
    if (threadIdx.x < SORT_BUCKETS) cnt[threadIdx.x] = 0;
    __syncthreads();
    for (uint64_t v0 = blockIdx.x * (uint64_t)CLASSIFY_THREADS; v0 < n; v0 += (uint64_t)gridDim.x * CLASSIFY_THREADS) {
        const uint64_t v = v0 + threadIdx.x;
        const int cls = v < n ? sort_bucket(rowptr[v + 1] - rowptr[v]) : -1;
        const unsigned lane = threadIdx.x & 31;
        const unsigned peers = __match_any_sync(KC_FULL_MASK, cls);
        const int leader = __ffs(peers) - 1;
        unsigned rank = 0;
        if (cls >= 0 && (int)lane == leader) rank = atomicAdd(&cnt[cls], (unsigned)__popc(peers));
        if (!cursor) continue;
        rank = __shfl_sync(KC_FULL_MASK, rank, leader) + __popc(peers & ((1u << lane) - 1u));
        __syncthreads();
        if (threadIdx.x < SORT_BUCKETS) {
            const unsigned c = cnt[threadIdx.x];
            cnt[threadIdx.x] = 0;
            base[threadIdx.x] = c ? atomicAdd(&cursor[threadIdx.x], (unsigned long long)c) : 0ull;
        }
        __syncthreads();
        if (cls >= 0) list[base[cls] + rank] = (uint32_t)v;
    }
    __syncthreads();
    if (!cursor && threadIdx.x < SORT_BUCKETS && cnt[threadIdx.x])
        atomicAdd(&counts[threadIdx.x], (unsigned long long)cnt[threadIdx.x]);
}

// Class A: rows of at most G = 8, 16 or 32 entries, 32 / G of them per warp,
// bitonic networks over shuffles (one row per warp whatever its length: 0.37 ms
// on R-MAT 22, 0.14 ms now).
template <int G>
__global__ void sort_rows_short(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ rows,
                                uint64_t nrows, uint32_t *key) {
    const unsigned gl = threadIdx.x & (G - 1);
    const uint64_t first = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) / G;
    const uint64_t step = (uint64_t)gridDim.x * blockDim.x / G;
    const uint64_t turns = (nrows + step - 1) / step;  // the same for every lane of a warp
    for (uint64_t t = 0; t < turns; t++) {
        const uint64_t r = first + t * step;
        int64_t start = 0;
        uint32_t len = 0;
        if (r < nrows) {
            const uint32_t v = rows[r];
            start = rowptr[v];
            len = (uint32_t)(rowptr[v + 1] - start);
        }
        uint32_t k = gl < len ? key[start + gl] : 0xffffffffu;
#pragma unroll
        for (int size = 2; size <= G; size <<= 1) {
#pragma unroll
            for (int stride = size >> 1; stride > 0; stride >>= 1) {
                const uint32_t pk = __shfl_xor_sync(KC_FULL_MASK, k, stride);
                const bool up = (gl & size) == 0 || size == G;
                const bool lower = (gl & stride) == 0;
                k = lower == up ? min(k, pk) : max(k, pk);
            }
        }
        if (gl < len) key[start + gl] = k;
    }
}

// Class B: rows of P/2 < len <= P = 32 R W entries, padded to P with the
// largest key, in the registers of W warps: a bitonic network in which lane l
// of warp w holds entries (32 w + l) R + j, so that strides below R are
// compares within a lane, strides below 32 R shuffles, and only the widest
// strides of rows above 1,024 entries go through shared memory (1 and 3 steps
// of 66 and 78).  A phase that sorts downwards on a lane runs upwards on
// complemented keys.  Keys are loaded in any order and stored in row order
// through shared memory.  What bounds it is the instructions of the compares;
// the network in shared memory that it replaces paid two reads, two writes and
// a barrier a step (R-MAT 22, 134 M entries, rows of 33..4,096: 2.66 ms, now
// 0.77 ms).
constexpr int SORT_THREADS = 256;

// The compares of one phase (entries at distance top, top / 2, .. 1, all within
// a warp's 32 R entries).  up(j): whether entry j of a lane sorts upwards.
template <int R, typename Up>
__device__ __forceinline__ void sort_phase(uint32_t (&k)[R], int top, unsigned lane, Up up) {
#pragma unroll
    for (int stride = 16 * R; stride > 0; stride >>= 1) {
        if (stride > top) continue;
        if (stride >= R) {
            const bool lower = (lane & (stride / R)) == 0;
#pragma unroll
            for (int j = 0; j < R; j++) {
                const uint32_t pk = __shfl_xor_sync(KC_FULL_MASK, k[j], stride / R);
                k[j] = lower ? min(k[j], pk) : max(k[j], pk);
            }
        } else {
#pragma unroll
            for (int j = 0; j < R; j++)
                if (!(j & stride)) {
                    const uint32_t lo = min(k[j], k[j | stride]), hi = max(k[j], k[j | stride]);
                    k[j] = up(j) ? lo : hi;
                    k[j | stride] = up(j) ? hi : lo;
                }
        }
    }
}

template <int R, int W>
__global__ void __launch_bounds__(SORT_THREADS) sort_rows_reg(const int64_t *__restrict__ rowptr,
                                                              const uint32_t *__restrict__ rows, uint64_t nrows,
                                                              uint32_t *key) {
    constexpr int OWN = 32 * R;  // entries of a warp
    constexpr int RPC = SORT_THREADS / 32 / W;  // rows per CTA
    __shared__ uint32_t sk[SORT_THREADS / 32][OWN + R];
    const unsigned lane = threadIdx.x & 31, wib = threadIdx.x >> 5, w = wib % W;
    for (uint64_t g = (uint64_t)blockIdx.x * RPC; g < nrows; g += (uint64_t)gridDim.x * RPC) {
        const uint64_t r = g + wib / W;
        int64_t start = 0;
        uint32_t len = 0;
        if (r < nrows) {
            const uint32_t v = rows[r];
            start = rowptr[v] + (int64_t)w * OWN;
            const int64_t left = rowptr[v + 1] - start;
            len = left <= 0 ? 0u : left < OWN ? (uint32_t)left : (uint32_t)OWN;
        }
        uint32_t k[R];
#pragma unroll
        for (int j = 0; j < R; j++) {
            const uint32_t e = j * 32 + lane;
            k[j] = e < len ? key[start + e] : 0xffffffffu;
        }
        // entries whose index has the bit `size` sort downwards in that phase
#pragma unroll
        for (int size = 2; size <= OWN; size <<= 1) {
            uint32_t flip = 0;
            if (size < OWN && size >= R) flip = (lane & (size / R)) ? 0xffffffffu : 0u;
            if (size == OWN) flip = W > 1 && (w & 1) ? 0xffffffffu : 0u;
#pragma unroll
            for (int j = 0; j < R; j++) k[j] ^= flip;
            sort_phase<R>(k, size / 2, lane, [&](int j) { return size >= R || !(j & size); });
#pragma unroll
            for (int j = 0; j < R; j++) k[j] ^= flip;
        }
        if constexpr (W > 1) {
#pragma unroll 1
            for (int ws = 2; ws <= W; ws <<= 1) {  // phases of 2, 4, .. W warps
                const uint32_t flip = ws < W && (w & ws) ? 0xffffffffu : 0u;
#pragma unroll
                for (int j = 0; j < R; j++) k[j] ^= flip;
#pragma unroll 1
                for (int d = ws / 2; d > 0; d >>= 1) {
                    const unsigned other = wib ^ d;
                    const bool lower = (w & d) == 0;
                    __syncthreads();
#pragma unroll
                    for (int j = 0; j < R; j++) sk[wib][j * 32 + lane] = k[j];
                    __syncthreads();
#pragma unroll
                    for (int j = 0; j < R; j++) {
                        const uint32_t pk = sk[other][j * 32 + lane];
                        k[j] = lower ? min(k[j], pk) : max(k[j], pk);
                    }
                }
                sort_phase<R>(k, OWN / 2, lane, [](int) { return true; });
#pragma unroll
                for (int j = 0; j < R; j++) k[j] ^= flip;
            }
            __syncthreads();
        }
#pragma unroll
        for (int j = 0; j < R; j++) {
            const uint32_t i = lane * R + j;
            sk[wib][i + i / 32] = k[j];
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < R; j++) {
            const uint32_t e = j * 32 + lane;
            if (e < len) key[start + e] = sk[wib][e + j];
        }
        __syncwarp();
    }
}

// Long rows that will be de-duplicated: the columns of a row set bits in a
// shared-memory bitmap, which is then read back in order.  A row takes as
// many passes as the columns need bitmaps; the slots freed by repeated
// entries are filled with the row's last column, so the row stays sorted and
// the de-duplication drops them.  Results of several passes wait in tk.  What
// bounds it is clearing and reading the bitmap (about 4,500 clocks a pass);
// the radix sort below takes about 7 clocks an entry of an SM, so rows of at
// least BITMAP_ROW entries per pass go this way (R-MAT 22, rows above 4,096:
// 2.42 ms by radix, 0.80 ms here).  Where a row's columns are crowded, a few
// threads hold them all, and 1,664 columns written by one thread after the other
// outlast the rest of the pass: their warps write them together, 32 words at a
// time (whole builds: ten cliques of 4,200 consecutive vertices 23.4 -> 6.4 ms,
// 9.8 with the radix sort alone; a clique of 5,000 3.16 -> 1.21, 2.52; R-MAT 22
// the same).
constexpr int BITMAP_THREADS = 1024;
constexpr uint32_t BITMAP_OWN = 52;  // words per thread: 16-byte reads 52 words apart meet no bank twice
constexpr uint32_t BITMAP_WORDS = BITMAP_THREADS * BITMAP_OWN;  // 208 KB: 1,703,936 columns a pass
constexpr uint32_t BITMAP_ROW = 512;

__global__ void __launch_bounds__(BITMAP_THREADS) sort_rows_bitmap(const int64_t *__restrict__ rowptr,
                                                                   const uint32_t *__restrict__ rows, uint64_t nrows,
                                                                   uint32_t n, uint32_t min_len, uint32_t *key,
                                                                   uint32_t *tk) {
    extern __shared__ __align__(16) uint32_t bits[];
    __shared__ uint32_t wsum[BITMAP_THREADS / 32];
    __shared__ uint32_t last_sh;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t cols = BITMAP_WORDS * 32;
    uint4 *mine = reinterpret_cast<uint4 *>(bits + threadIdx.x * BITMAP_OWN);
#pragma unroll
    for (uint32_t i = 0; i < BITMAP_OWN / 4; i++) mine[i] = make_uint4(0, 0, 0, 0);
    for (uint64_t r = blockIdx.x; r < nrows; r += gridDim.x) {
        const uint32_t v = rows[r];
        const int64_t start = rowptr[v];
        const uint32_t len = (uint32_t)(rowptr[v + 1] - start);
        if (len < min_len) continue;
        uint32_t *out = n > cols ? tk + start : key + start;
        uint32_t off = 0;  // columns written
        const uint32_t few = 64 + len / 256;  // four times a thread's share, and what a warp's help costs
        for (uint64_t c0 = 0; c0 < n; c0 += cols) {
            __syncthreads();  // the bitmap is clear
#pragma unroll 4
            for (uint32_t j = threadIdx.x; j < len; j += BITMAP_THREADS) {
                const uint64_t c = (uint64_t)key[start + j] - c0;  // wraps below c0
                if (c < cols) atomicOr(&bits[c >> 5], 1u << (c & 31));
            }
            __syncthreads();
            // every thread takes its own words: count, then write from its offset
            uint32_t own = 0;
#pragma unroll
            for (uint32_t i = 0; i < BITMAP_OWN / 4; i++) {
                const uint4 q = mine[i];
                own += __popc(q.x) + __popc(q.y) + __popc(q.z) + __popc(q.w);
            }
            uint32_t wtot;
            uint32_t at = off + warp_excl_scan(own, lane, wtot);
            if (lane == 0) wsum[warp] = wtot;
            __syncthreads();
            const uint32_t ws = wsum[lane];  // 32 warps
            at += __reduce_add_sync(KC_FULL_MASK, lane < warp ? ws : 0u);
            off += __reduce_add_sync(KC_FULL_MASK, ws);
            // a thread with far more columns than most has its warp write them
            for (unsigned many = __ballot_sync(KC_FULL_MASK, own > few); many; many &= many - 1) {
                const int l = __ffs(many) - 1;
                const uint32_t w0 = (threadIdx.x - lane + l) * BITMAP_OWN;
                uint32_t to = __shfl_sync(KC_FULL_MASK, at, l);
                for (uint32_t i = lane; i - lane < BITMAP_OWN; i += 32) {
                    const uint32_t word = i < BITMAP_OWN ? bits[w0 + i] : 0u;
                    uint32_t all;
                    uint32_t p = to + warp_excl_scan((uint32_t)__popc(word), lane, all);
                    to += all;
                    for (uint32_t b = word; b; b &= b - 1) {
                        const uint32_t c = (uint32_t)c0 + (w0 + i) * 32 + __ffs(b) - 1;
                        out[p++] = c;
                        if (p == off) last_sh = c;
                    }
                    if (i < BITMAP_OWN) bits[w0 + i] = 0;
                }
            }
            if (own && own <= few) {
                const uint32_t col0 = (uint32_t)c0 + threadIdx.x * BITMAP_OWN * 32;
                for (uint32_t i = 0; i < BITMAP_OWN / 4; i++) {
                    const uint4 q = mine[i];
                    if (!(q.x | q.y | q.z | q.w)) continue;
                    const uint32_t word[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int t = 0; t < 4; t++)
                        for (uint32_t b = word[t]; b; b &= b - 1) {
                            const uint32_t c = col0 + (4 * i + t) * 32 + __ffs(b) - 1;
                            out[at++] = c;
                            if (at == off) last_sh = c;  // the last of this pass (the row's, after the last pass)
                        }
                    mine[i] = make_uint4(0, 0, 0, 0);
                }
            }
        }
        __syncthreads();
        const uint32_t last = last_sh;
        for (uint32_t j = off + threadIdx.x; j < len; j += BITMAP_THREADS) key[start + j] = last;
        if (out != key + start)
            for (uint32_t j = threadIdx.x; j < off; j += BITMAP_THREADS) key[start + j] = out[j];
    }
}

// Class C: one CTA per long row, LSD radix sort with 8-bit digits, stable from
// pass to pass.  Ping-pongs between the row and the same range of the staging
// array tk, one pass per digit, and copies back after an odd pass count.
constexpr int RADIX_THREADS = 256;
constexpr int RADIX_WARPS = RADIX_THREADS / 32;

__global__ void __launch_bounds__(RADIX_THREADS) sort_rows_radix(const int64_t *__restrict__ rowptr,
                                                                 const uint32_t *__restrict__ rows, uint64_t nrows,
                                                                 uint32_t *key, uint32_t *tk, int passes,
                                                                 uint32_t below) {
    __shared__ uint32_t hist[256];
    __shared__ uint32_t base[256];
    __shared__ uint32_t wcnt[RADIX_WARPS][256];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (uint64_t r = blockIdx.x; r < nrows; r += gridDim.x) {
        uint32_t v = rows[r];
        int64_t start = rowptr[v];
        uint32_t len = (uint32_t)(rowptr[v + 1] - start);
        if (len >= below) continue;  // sorted by sort_rows_bitmap
        uint32_t *ik = key + start;
        uint32_t *ok = tk + start;
        for (int pass = 0; pass < passes; pass++) {
            int shift = 8 * pass;
            for (int i = threadIdx.x; i < 256; i += RADIX_THREADS) hist[i] = 0;
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < len; j += RADIX_THREADS) atomicAdd(&hist[(ik[j] >> shift) & 255u], 1u);
            __syncthreads();
            if (warp == 0) {
                uint32_t loc[8];
                uint32_t s = 0;
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    loc[i] = s;
                    s += hist[lane * 8 + i];
                }
                uint32_t tot;
                uint32_t ex = warp_excl_scan(s, lane, tot);
#pragma unroll
                for (int i = 0; i < 8; i++) base[lane * 8 + i] = ex + loc[i];
            }
            __syncthreads();
            for (uint32_t tile = 0; tile < len; tile += RADIX_THREADS) {
                for (int i = threadIdx.x; i < RADIX_WARPS * 256; i += RADIX_THREADS) (&wcnt[0][0])[i] = 0;
                __syncthreads();
                uint32_t j = tile + threadIdx.x;
                bool valid = j < len;
                uint32_t kk = valid ? ik[j] : 0u;
                uint32_t d = valid ? ((kk >> shift) & 255u) : 256u;
                unsigned int peers = __match_any_sync(KC_FULL_MASK, d);
                uint32_t rank = __popc(peers & ((1u << lane) - 1u));
                if (valid && rank == 0) wcnt[warp][d] = __popc(peers);
                __syncthreads();
                if (valid) {
                    uint32_t before = 0;
                    for (unsigned w = 0; w < warp; w++) before += wcnt[w][d];
                    ok[base[d] + before + rank] = kk;
                }
                __syncthreads();
                for (int dd = threadIdx.x; dd < 256; dd += RADIX_THREADS) {
                    uint32_t t = 0;
                    for (int w = 0; w < RADIX_WARPS; w++) t += wcnt[w][dd];
                    base[dd] += t;
                }
                __syncthreads();
            }
            uint32_t *t0 = ik; ik = ok; ok = t0;
            __syncthreads();
        }
        if (passes & 1) {
            // result sits in the staging range: copy back into the row
            for (uint32_t j = threadIdx.x; j < len; j += RADIX_THREADS) key[start + j] = tk[start + j];
        }
        __syncthreads();
    }
}

static void launch_reg(int logp, const int64_t *rowptr, const uint32_t *rows, uint64_t nrows, uint32_t *key, int sms,
                       cudaStream_t s) {
    const uint64_t rpc = logp <= 10 ? SORT_THREADS / 32 : (SORT_THREADS / 32) >> (logp - 10);
    const int gr = (int)std::max<uint64_t>(1, std::min<uint64_t>((nrows + rpc - 1) / rpc, (uint64_t)sms * 8));
    switch (logp) {
    case 6: sort_rows_reg<2, 1><<<gr, SORT_THREADS, 0, s>>>(rowptr, rows, nrows, key); break;
    case 7: sort_rows_reg<4, 1><<<gr, SORT_THREADS, 0, s>>>(rowptr, rows, nrows, key); break;
    case 8: sort_rows_reg<8, 1><<<gr, SORT_THREADS, 0, s>>>(rowptr, rows, nrows, key); break;
    case 9: sort_rows_reg<16, 1><<<gr, SORT_THREADS, 0, s>>>(rowptr, rows, nrows, key); break;
    case 10: sort_rows_reg<32, 1><<<gr, SORT_THREADS, 0, s>>>(rowptr, rows, nrows, key); break;
    case 11: sort_rows_reg<32, 2><<<gr, SORT_THREADS, 0, s>>>(rowptr, rows, nrows, key); break;
    default: sort_rows_reg<32, 4><<<gr, SORT_THREADS, 0, s>>>(rowptr, rows, nrows, key); break;
    }
}

// Raises sort_rows_bitmap's dynamic shared-memory limit, once per device.
static int bitmap_smem_limit() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    KC_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(KC_ERR_INVALID, "device %d out of range", dev);
    std::lock_guard<std::mutex> lk(mu);
    if (done[dev]) return KC_OK;
    KC_CUDA(cudaFuncSetAttribute(sort_rows_bitmap, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(BITMAP_WORDS * 4)));
    done[dev] = true;
    return KC_OK;
}

// Sorts every row of g->col.  dedup: repeated entries will be dropped.
static int sort_rows(Graph *g, bool dedup, cudaStream_t s) {
    uint32_t *key = g->col;
    const uint32_t n = g->n;
    if (n == 0 || g->nnz == 0) return KC_OK;
    const int sms = current_sms();
    uint32_t *list = nullptr;
    unsigned long long *counts = nullptr;
    KC_TRY(dalloc(&list, (uint64_t)n, "row class list"));
    if (dalloc(&counts, 2 * SORT_BUCKETS, "row class counts") != KC_OK) { dfree(list); return KC_ERR_NOMEM; }
    unsigned long long *cursor = counts + SORT_BUCKETS;
    cudaMemsetAsync(counts, 0, SORT_BUCKETS * sizeof(unsigned long long), s);
    const int cg = (int)std::min<uint64_t>(((uint64_t)n + CLASSIFY_THREADS - 1) / CLASSIFY_THREADS, (uint64_t)sms * 4);
    classify_rows<<<cg, CLASSIFY_THREADS, 0, s>>>(g->rowptr, n, counts, nullptr, nullptr);
    unsigned long long h[SORT_BUCKETS], off[SORT_BUCKETS + 1];
    cudaMemcpyAsync(h, counts, sizeof(h), cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { dfree(list); dfree(counts); return fail(KC_ERR_CUDA, "classify: %s", cudaGetErrorString(e)); }
    off[0] = 0;
    for (int c = 0; c < SORT_BUCKETS; c++) off[c + 1] = off[c] + h[c];
    cudaMemcpyAsync(cursor, off, SORT_BUCKETS * sizeof(unsigned long long), cudaMemcpyHostToDevice, s);
    classify_rows<<<cg, CLASSIFY_THREADS, 0, s>>>(g->rowptr, n, nullptr, cursor, list);
    for (int c = 0; c < SORT_SHORT; c++) {
        if (!h[c]) continue;
        const int gr = grid_for(h[c] * (8u << c), 256, sms);
        const uint32_t *rows = list + off[c];
        if (c == 0) sort_rows_short<8><<<gr, 256, 0, s>>>(g->rowptr, rows, h[c], key);
        else if (c == 1) sort_rows_short<16><<<gr, 256, 0, s>>>(g->rowptr, rows, h[c], key);
        else sort_rows_short<32><<<gr, 256, 0, s>>>(g->rowptr, rows, h[c], key);
    }
    for (int c = SORT_SHORT; c < SORT_BUCKETS - 1; c++)
        if (h[c]) launch_reg(c + 3, g->rowptr, list + off[c], h[c], key, sms, s);
    uint32_t *tk = nullptr;
    int rc = KC_OK;
    const unsigned long long hc = h[SORT_BUCKETS - 1];
    if (hc) {
        int bits = 1;
        while (bits < 32 && (n >> bits) != 0) bits++;
        int passes = (bits + 7) / 8;
        // rows from this length on go through the bitmap
        const uint64_t maps = ((uint64_t)n + BITMAP_WORDS * 32 - 1) / (BITMAP_WORDS * 32);
        const uint32_t bitmap_from = dedup ? (uint32_t)std::min<uint64_t>(maps * BITMAP_ROW, 0xffffffffu) : 0xffffffffu;
        const bool all_bitmap = bitmap_from <= CLASS_B_MAX + 1;
        if (!all_bitmap || maps > 1) rc = dalloc(&tk, g->nnz, "row sort staging keys");
        if (rc == KC_OK && dedup) rc = bitmap_smem_limit();
        if (rc == KC_OK) {
            const uint32_t *lc = list + off[SORT_BUCKETS - 1];
            if (dedup)
                sort_rows_bitmap<<<(unsigned)std::min<unsigned long long>(hc, (unsigned long long)sms), BITMAP_THREADS,
                                   BITMAP_WORDS * 4, s>>>(g->rowptr, lc, hc, n, bitmap_from, key, tk);
            if (!all_bitmap)
                sort_rows_radix<<<(unsigned)std::min<unsigned long long>(hc, (unsigned long long)sms * 4), RADIX_THREADS, 0, s>>>(
                    g->rowptr, lc, hc, key, tk, passes, bitmap_from);
        }
    }
    e = cudaGetLastError();
    cudaError_t e2 = cudaStreamSynchronize(s);
    dfree(tk);
    dfree(list);
    dfree(counts);
    if (rc != KC_OK) return rc;
    if (e != cudaSuccess || e2 != cudaSuccess)
        return fail(KC_ERR_CUDA, "row sort: %s", cudaGetErrorString(e != cudaSuccess ? e : e2));
    return KC_OK;
}

// ----------------------------------------------------------- unique -------
// De-duplication of sorted rows, entry-parallel: an entry is kept when it
// starts its row or differs from its predecessor.  Row starts are first set
// in a bitmap over the entries (one thread per row), so a tile of UQ_TILE
// entries (UQ_PER consecutive entries per thread) reads them with its entries
// whatever the number of rows, empty ones included, that start in it.  Pass 1
// counts the kept entries of each tile; a scan gives each tile its output
// offset; pass 2 writes the kept entries and saves, per thread, its kept mask
// and the kept count before it in the tile; a pass over the rows then gives
// each row its new offset from those.
constexpr unsigned UQ_THREADS = 256;
constexpr unsigned UQ_PER = 16;
constexpr unsigned UQ_TILE = UQ_THREADS * UQ_PER;

__global__ void mark_row_starts(const int64_t *__restrict__ rowptr, uint32_t n, uint32_t *startbits) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        const int64_t r = rowptr[v];
        if (rowptr[v + 1] > r) atomicOr(&startbits[r >> 5], 1u << (r & 31));
    }
}

// This thread's UQ_PER entries of the tile [t0, t0 + len), four 16-byte loads
// (col is aligned, t0 a multiple of UQ_TILE), and their kept mask (bit i: entry
// t0 + threadIdx.x * UQ_PER + i).
__device__ __forceinline__ unsigned uq_mask(const uint32_t *__restrict__ col, const uint32_t *__restrict__ startbits,
                                            uint64_t t0, unsigned len, uint32_t (&x)[UQ_PER]) {
    unsigned mask = 0;
    const unsigned o0 = threadIdx.x * UQ_PER;
    if (o0 < len) {
        const uint64_t e0 = t0 + o0;  // a multiple of UQ_PER: the bits lie in one word
        const unsigned sb = (startbits[e0 >> 5] >> (e0 & 31)) & ((1u << UQ_PER) - 1u);
        uint32_t prev = e0 > 0 ? col[e0 - 1] : 0u;
        if (o0 + UQ_PER <= len) {
#pragma unroll
            for (unsigned q = 0; q < UQ_PER / 4; q++) {
                const uint4 y = __ldcs(reinterpret_cast<const uint4 *>(col + e0) + q);
                x[4 * q] = y.x;
                x[4 * q + 1] = y.y;
                x[4 * q + 2] = y.z;
                x[4 * q + 3] = y.w;
            }
        } else {
#pragma unroll
            for (unsigned i = 0; i < UQ_PER; i++) x[i] = o0 + i < len ? col[e0 + i] : 0u;
        }
#pragma unroll
        for (unsigned i = 0; i < UQ_PER; i++) {
            if (o0 + i < len && (((sb >> i) & 1u) || x[i] != prev)) mask |= 1u << i;
            prev = x[i];
        }
    }
    return mask;
}

__global__ void __launch_bounds__(UQ_THREADS) unique_tiles_count(const uint32_t *__restrict__ col,
                                                                  const uint32_t *__restrict__ startbits, uint64_t nnz,
                                                                  uint32_t *tile_cnt) {
    __shared__ uint32_t wsum[UQ_THREADS / 32];
    const uint64_t tiles = (nnz + UQ_TILE - 1) / UQ_TILE;
    for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint64_t t0 = t * UQ_TILE;
        const unsigned len = (unsigned)(nnz - t0 < (uint64_t)UQ_TILE ? nnz - t0 : (uint64_t)UQ_TILE);
        uint32_t x[UQ_PER];
        const unsigned c = __reduce_add_sync(KC_FULL_MASK, (unsigned)__popc(uq_mask(col, startbits, t0, len, x)));
        if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = c;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned tot = 0;
            for (unsigned w = 0; w < UQ_THREADS / 32; w++) tot += wsum[w];
            tile_cnt[t] = tot;
        }
        __syncthreads();
    }
}

// The kept entries of a tile are gathered in shared memory and written as one
// run (each thread writing its own 64 bytes: 0.67 ms on 134 M entries, 0.24 ms now).
__global__ void __launch_bounds__(UQ_THREADS) unique_tiles_write(const uint32_t *__restrict__ col,
                                                                  const uint32_t *__restrict__ startbits, uint64_t nnz,
                                                                  const int64_t *__restrict__ tile_off, uint32_t *ncol,
                                                                  uint16_t *tmask, uint16_t *tpre) {
    __shared__ uint32_t wsum[UQ_THREADS / 32];
    __shared__ uint32_t kept[UQ_TILE];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t tiles = (nnz + UQ_TILE - 1) / UQ_TILE;
    for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
        const uint64_t t0 = t * UQ_TILE;
        const unsigned len = (unsigned)(nnz - t0 < (uint64_t)UQ_TILE ? nnz - t0 : (uint64_t)UQ_TILE);
        uint32_t x[UQ_PER];
        const unsigned mask = uq_mask(col, startbits, t0, len, x);
        unsigned wt;
        const unsigned ex = warp_excl_scan((unsigned)__popc(mask), lane, wt);
        if (lane == 0) wsum[warp] = wt;
        __syncthreads();
        unsigned before = ex, total = 0;
#pragma unroll
        for (unsigned w = 0; w < UQ_THREADS / 32; w++) {
            before += w < warp ? wsum[w] : 0u;
            total += wsum[w];
        }
        tmask[t * UQ_THREADS + threadIdx.x] = (uint16_t)mask;
        tpre[t * UQ_THREADS + threadIdx.x] = (uint16_t)before;
        unsigned k = before;
#pragma unroll
        for (unsigned i = 0; i < UQ_PER; i++)
            if ((mask >> i) & 1u) kept[k++] = x[i];
        __syncthreads();
        const int64_t base = tile_off[t];
        for (unsigned i = threadIdx.x; i < total; i += UQ_THREADS) ncol[base + i] = kept[i];
        __syncthreads();
    }
}

// New offset of every row: the kept entries before its old start.
__global__ void unique_rows(const int64_t *__restrict__ rowptr, uint32_t n, uint64_t nnz,
                            const int64_t *__restrict__ tile_off, const uint16_t *__restrict__ tmask,
                            const uint16_t *__restrict__ tpre, int64_t *nrow) {
    const uint64_t tiles = (nnz + UQ_TILE - 1) / UQ_TILE;
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v <= n; v += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = (uint64_t)rowptr[v];
        if (r >= nnz) {
            nrow[v] = tile_off[tiles];
            continue;
        }
        const uint64_t t = r / UQ_TILE;
        const unsigned o = (unsigned)(r % UQ_TILE);
        const uint64_t th = t * UQ_THREADS + o / UQ_PER;
        nrow[v] = tile_off[t] + tpre[th] + __popc((unsigned)tmask[th] & ((1u << (o % UQ_PER)) - 1u));
    }
}

// ------------------------------------------------------- graph stats ------
__global__ void degree_stats(const int64_t *__restrict__ rowptr, uint32_t n, uint32_t *maxdeg,
                             unsigned long long *vnodes) {
    __shared__ uint32_t mx_sh;
    __shared__ unsigned long long vn_sh;
    if (threadIdx.x == 0) {
        mx_sh = 0;
        vn_sh = 0;
    }
    __syncthreads();
    uint32_t mx = 0;
    unsigned long long vn = 0;
#pragma unroll 4
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t d = (uint64_t)(rowptr[v + 1] - rowptr[v]);
        mx = max(mx, (uint32_t)d);
        vn += (d + 31) / 32;
    }
    mx = __reduce_max_sync(KC_FULL_MASK, mx);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vn += __shfl_xor_sync(KC_FULL_MASK, vn, o);
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&mx_sh, mx);
        atomicAdd(&vn_sh, vn);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(maxdeg, mx_sh);
        atomicAdd(vnodes, vn_sh);
    }
}

int graph_finish(Graph *g) {
    cudaStream_t s = g->stream;
    uint32_t *md = nullptr;
    KC_TRY(dalloc(&md, 4, "graph stats"));
    unsigned long long *vn = reinterpret_cast<unsigned long long *>(md + 2);
    cudaMemsetAsync(md, 0, 16, s);
    // few CTAs: each ends with two atomics on the same two words
    if (g->n) degree_stats<<<std::min(grid_for(g->n, 256, g->sm_count), std::max(g->sm_count, 1) * 4), 256, 0, s>>>(g->rowptr, g->n, md, vn);
    uint32_t h[4];
    cudaMemcpyAsync(h, md, 16, cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    dfree(md);
    if (e != cudaSuccess) return fail(KC_ERR_CUDA, "graph stats: %s", cudaGetErrorString(e));
    g->max_deg = h[0];
    unsigned long long vv;
    memcpy(&vv, &h[2], 8);
    g->num_vnodes = vv;
    return KC_OK;
}

// ------------------------------------------------------------ build -------
int build_csr_from_edges(Graph *g, const uint32_t *d_src, const uint32_t *d_dst, uint64_t m, uint32_t n,
                         uint32_t flags) {
    cudaStream_t s = g->stream;
    const int sms = g->sm_count;
    const bool keep_order = (flags & (KC_EDGES_DEDUP | KC_EDGES_SORT_ROWS)) == 0;
    if (keep_order && 2 * m > 0xffffffffull)
        return fail(KC_ERR_UNSUPPORTED, "edge-list row order needs 2*m < 2^32 (m=%llu); pass KC_EDGES_SORT_ROWS",
                    (unsigned long long)m);
    g->n = n;
    if (keep_order && m && n) {
        KC_TRY(dalloc(&g->rowptr, (uint64_t)n + 1, "row offsets"));
        KC_TRY(build_in_order(g, d_src, d_dst, m, n));
        return graph_finish(g);
    }
    uint32_t *deg = nullptr, *err = nullptr;
    KC_TRY(dalloc(&deg, (uint64_t)n + 1, "degrees"));
    int rc = dalloc(&err, 1, "error flag");
    if (rc) { dfree(deg); return rc; }
    rc = dalloc(&g->rowptr, (uint64_t)n + 1, "row offsets");
    if (rc) { dfree(deg); dfree(err); return rc; }
    cudaMemsetAsync(deg, 0, ((uint64_t)n + 1) * 4, s);
    cudaMemsetAsync(err, 0, 4, s);
    // partitioned where the order within a row is free and there is room for
    // the pairs (16 bytes per edge) and the tiles' row shares, 6 bytes x (2 m /
    // PART_TILE + buckets) x rows per bucket: 1.1 bytes per edge on R-MAT 22, up to
    // 102 where rows outnumber edges by PART_MAX_ROWS
    PartPlan plan{};
    uint2 *pairs = nullptr;
    plan.shift = part_shift(m, n);
    if (plan.shift >= 0) {
        plan.buckets = ((n - 1) >> plan.shift) + 1;
        rc = dalloc(&plan.base, 3ull * (plan.buckets + 1), "partition plan");
        if (!rc) rc = dalloc(&pairs, 2 * m, "partitioned edges");
        const uint64_t shares = (2 * m / PART_TILE + plan.buckets) << plan.shift;
        if (!rc) rc = dalloc(&plan.off, shares, "row shares of the tiles");
        if (!rc) rc = dalloc(&plan.count, shares, "row shares of the tiles");
        if (!rc) rc = part_smem_limits();
        if (rc) {
            dfree(plan.base);
            dfree(pairs);
            dfree(plan.off);
            dfree(plan.count);
            plan.shift = -1;
            pairs = nullptr;
            if (rc != KC_ERR_NOMEM) { dfree(deg); dfree(err); return rc; }
            clear_error();
        }
    }
    bool part = plan.shift >= 0;
    auto release_part = [&]() {
        if (part) {
            dfree(plan.base);
            dfree(pairs);
            dfree(plan.off);
            dfree(plan.count);
        }
    };
    const int part_grid = sms * 2;
    const size_t row_smem = part ? (size_t)4 << plan.shift : 0;
    const int row_grid = sms * (row_smem <= 32768 ? 4 : 3);  // 512 threads of 32 registers, up to 64 KB of counters
    if (part) {
        plan.cursor = plan.base + plan.buckets + 1;
        plan.tile = reinterpret_cast<uint32_t *>(plan.cursor + plan.buckets);
        cudaMemsetAsync(plan.base, 0, 8ull * (plan.buckets + 1), s);
        part_hist<<<part_grid, 1024, plan.buckets * 4, s>>>(d_src, d_dst, m, n, plan, err);
        part_plan<<<1, 1024, 0, s>>>(plan);
    } else if (m) {
        count_degrees<<<grid_for(m, 256, sms), 256, 0, s>>>(d_src, d_dst, m, n, deg, err);
    }
    uint32_t herr = 0;
    cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { dfree(deg); dfree(err); release_part(); return fail(KC_ERR_CUDA, "degree count: %s", cudaGetErrorString(e)); }
    if (herr) { dfree(deg); dfree(err); release_part(); return fail(KC_ERR_INVALID, "edge endpoint >= n (%u)", n); }
    if (part) {
        part_pairs<<<(unsigned)std::min<uint64_t>((m + PART_EDGES - 1) / PART_EDGES, (uint64_t)sms), PAIR_THREADS,
                     2 * PART_EDGES * sizeof(uint2) + plan.buckets * 12, s>>>(d_src, d_dst, m, n, plan, pairs);
        part_degrees<<<row_grid, PART_THREADS, row_smem, s>>>(pairs, plan, n, deg);
    }
    rc = exclusive_scan_u32_i64(deg, g->rowptr, n, s);
    if (rc) { dfree(deg); dfree(err); release_part(); return rc; }
    int64_t nnz = 0;
    cudaMemcpy(&nnz, g->rowptr + n, 8, cudaMemcpyDeviceToHost);
    g->nnz = (uint64_t)nnz;
    rc = dalloc(&g->col, g->nnz + 1, "column ids");
    if (rc == KC_ERR_NOMEM && part) {
        // the partition holds twice the columns: without it they may fit, and
        // the edges are scattered by the row offsets that it gave
        release_part();
        part = false;
        clear_error();
        rc = dalloc(&g->col, g->nnz + 1, "column ids");
    }
    if (rc) { dfree(deg); dfree(err); release_part(); return rc; }
    unsigned long long *cur = nullptr;  // row fill cursors, starting at the row offsets
    if (part && (1u << plan.shift) <= PART_STAGE_ROWS) {
        part_rows<true><<<sms, 1024, part_rows_smem(plan.shift), s>>>(pairs, plan, n, g->rowptr, g->col);
    } else if (part) {
        part_rows<false><<<row_grid, PART_THREADS, row_smem, s>>>(pairs, plan, n, g->rowptr, g->col);
    } else if (m) {
        rc = dalloc(&cur, (uint64_t)n + 1, "row cursors");
        if (rc) { dfree(deg); dfree(err); release_part(); return rc; }
        cudaMemcpyAsync(cur, g->rowptr, ((uint64_t)n + 1) * 8, cudaMemcpyDeviceToDevice, s);
        scatter_edges<<<grid_for(m, 256, sms), 256, 0, s>>>(d_src, d_dst, m, n, cur, g->col);
    }
    e = cudaStreamSynchronize(s);
    dfree(cur);
    release_part();
    if (e != cudaSuccess) { dfree(deg); dfree(err); return fail(KC_ERR_CUDA, "scatter: %s", cudaGetErrorString(e)); }
    rc = sort_rows(g, (flags & KC_EDGES_DEDUP) != 0, s);
    if (rc) { dfree(deg); dfree(err); return rc; }
    if ((flags & KC_EDGES_DEDUP) && g->nnz) {
        int64_t *nrow = nullptr, *toff = nullptr;
        uint32_t *ncol = nullptr, *tcnt = nullptr, *sbits = nullptr;
        uint16_t *tmask = nullptr, *tpre = nullptr;
        const uint64_t tiles = (g->nnz + UQ_TILE - 1) / UQ_TILE;
        auto release = [&]() {
            dfree(tcnt);
            dfree(toff);
            dfree(sbits);
            dfree(tmask);
            dfree(tpre);
        };
        rc = dalloc(&nrow, (uint64_t)n + 1, "dedup row offsets");
        if (rc == KC_OK) rc = dalloc(&tcnt, tiles, "dedup tile counts");
        if (rc == KC_OK) rc = dalloc(&toff, tiles + 1, "dedup tile offsets");
        if (rc == KC_OK) rc = dalloc(&sbits, tiles * (UQ_TILE / 32), "row-start bitmap");
        if (rc == KC_OK) rc = dalloc(&tmask, tiles * UQ_THREADS, "dedup masks");
        if (rc == KC_OK) rc = dalloc(&tpre, tiles * UQ_THREADS, "dedup prefixes");
        if (rc) { release(); dfree(nrow); dfree(deg); dfree(err); return rc; }
        cudaMemsetAsync(sbits, 0, tiles * (UQ_TILE / 32) * sizeof(uint32_t), s);
        mark_row_starts<<<grid_for(n, 256, sms), 256, 0, s>>>(g->rowptr, n, sbits);
        const int ug = (int)std::min<uint64_t>(tiles, (uint64_t)sms * 8);
        unique_tiles_count<<<ug, UQ_THREADS, 0, s>>>(g->col, sbits, g->nnz, tcnt);
        rc = exclusive_scan_u32_i64(tcnt, toff, tiles, s);
        int64_t nn = 0;
        if (rc == KC_OK) {
            cudaMemcpy(&nn, toff + tiles, 8, cudaMemcpyDeviceToHost);
            rc = dalloc(&ncol, (uint64_t)nn + 1, "dedup column ids");
        }
        if (rc) { release(); dfree(nrow); dfree(deg); dfree(err); return rc; }
        unique_tiles_write<<<ug, UQ_THREADS, 0, s>>>(g->col, sbits, g->nnz, toff, ncol, tmask, tpre);
        unique_rows<<<grid_for((uint64_t)n + 1, 256, sms), 256, 0, s>>>(g->rowptr, n, g->nnz, toff, tmask, tpre, nrow);
        e = cudaStreamSynchronize(s);
        release();
        dfree(g->rowptr);
        dfree(g->col);
        g->rowptr = nrow;
        g->col = ncol;
        g->nnz = (uint64_t)nn;
        if (e != cudaSuccess) { dfree(deg); dfree(err); return fail(KC_ERR_CUDA, "unique: %s", cudaGetErrorString(e)); }
    }
    dfree(deg);
    dfree(err);
    return graph_finish(g);
}

// ---------------------------------------------------------- validate ------
__device__ __forceinline__ unsigned long long pair_hash(uint32_t a, uint32_t b) {
    unsigned long long z = ((unsigned long long)a << 32 | b) + 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// Symmetry as multiset equality of {(min,max)} over entries above and below
// the diagonal: counts and a commutative hash sum must agree.
__global__ void validate_kernel(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ col, uint32_t n,
                                unsigned long long *acc) {
    const unsigned lane = threadIdx.x & 31;
    uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    unsigned long long bad = 0, hlo = 0, hhi = 0, clo = 0, chi = 0;
    for (uint64_t v = warp; v < n; v += nwarps) {
        for (int64_t j = rowptr[v] + lane; j < rowptr[v + 1]; j += 32) {
            uint32_t u = col[j];
            if (u >= n || u == v) { bad++; continue; }
            if (u > v) { hlo += pair_hash((uint32_t)v, u); clo++; }
            else { hhi += pair_hash(u, (uint32_t)v); chi++; }
        }
    }
    atomicAdd(&acc[0], bad);
    atomicAdd(&acc[1], hlo);
    atomicAdd(&acc[2], hhi);
    atomicAdd(&acc[3], clo);
    atomicAdd(&acc[4], chi);
}

int graph_validate(Graph *g, uint64_t *bad) {
    unsigned long long *acc = nullptr;
    KC_TRY(dalloc(&acc, 5, "validate"));
    cudaMemsetAsync(acc, 0, 40, g->stream);
    if (g->n) validate_kernel<<<grid_for((uint64_t)g->n * 32, 256, g->sm_count), 256, 0, g->stream>>>(g->rowptr, g->col, g->n, acc);
    unsigned long long h[5];
    cudaMemcpyAsync(h, acc, 40, cudaMemcpyDeviceToHost, g->stream);
    cudaError_t e = cudaStreamSynchronize(g->stream);
    dfree(acc);
    if (e != cudaSuccess) return fail(KC_ERR_CUDA, "validate: %s", cudaGetErrorString(e));
    uint64_t b = h[0];
    b += h[3] > h[4] ? h[3] - h[4] : h[4] - h[3];
    if (h[3] == h[4] && h[1] != h[2]) b += 1;
    *bad = b;
    return KC_OK;
}

// ---------------------------------------------------- virtual layout ------
__global__ void vlayout_kernel(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ col, uint32_t n,
                               uint32_t *node_pointer, uint32_t *edge_list) {
    const unsigned lane = threadIdx.x & 31;
    uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t v = warp; v < n; v += nwarps) {
        int64_t s = rowptr[v], e = rowptr[v + 1];
        uint64_t slot = (uint64_t)s + v;
        if (lane == 0) {
            node_pointer[v] = (uint32_t)slot;
            edge_list[slot] = (uint32_t)(e - s);
        }
        for (int64_t j = s + lane; j < e; j += 32) edge_list[slot + 1 + (j - s)] = col[j];
    }
}

__global__ void vparts_count(const int64_t *__restrict__ rowptr, uint32_t n, uint32_t part_size, uint32_t *k) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x)
        k[v] = (uint32_t)(((uint64_t)(rowptr[v + 1] - rowptr[v]) + part_size - 1) / part_size);
}

__global__ void vparts_fill(const int64_t *__restrict__ pstart, const uint32_t *__restrict__ k, uint32_t n,
                            uint32_t *parts) {
    for (uint64_t v = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; v < n; v += (uint64_t)gridDim.x * blockDim.x) {
        int64_t p = pstart[v];
        for (uint32_t j = 0; j < k[v]; j++) {
            parts[2 * (p + j)] = (uint32_t)v;
            parts[2 * (p + j) + 1] = j;
        }
    }
}

int virtual_layout(Graph *g, uint32_t part_size, uint32_t *h_node_pointer, uint32_t *h_edge_list,
                   uint32_t *h_parts, uint64_t *num_parts) {
    if (part_size == 0) return fail(KC_ERR_INVALID, "part_size must be > 0");
    cudaStream_t s = g->stream;
    const uint32_t n = g->n;
    uint32_t *k = nullptr;
    int64_t *pstart = nullptr;
    KC_TRY(dalloc(&k, (uint64_t)n + 1, "vnode counts"));
    int rc = dalloc(&pstart, (uint64_t)n + 1, "vnode offsets");
    if (rc) { dfree(k); return rc; }
    if (n) vparts_count<<<grid_for(n, 256, g->sm_count), 256, 0, s>>>(g->rowptr, n, part_size, k);
    rc = exclusive_scan_u32_i64(k, pstart, n, s);
    int64_t np = 0;
    if (rc == KC_OK) cudaMemcpy(&np, pstart + n, 8, cudaMemcpyDeviceToHost);
    *num_parts = (uint64_t)np;
    if (rc || (!h_parts && !h_node_pointer && !h_edge_list)) { dfree(k); dfree(pstart); return rc; }
    if (g->nnz + n > 0xffffffffull) { dfree(k); dfree(pstart); return fail(KC_ERR_UNSUPPORTED, "layout offsets exceed uint32"); }
    uint32_t *dnp = nullptr, *del = nullptr, *dparts = nullptr;
    rc = dalloc(&dnp, (uint64_t)n + 1, "nodePointer");
    if (!rc) rc = dalloc(&del, g->nnz + n + 1, "edgeList");
    if (!rc) rc = dalloc(&dparts, 2ull * (uint64_t)np + 2, "partNodePointer");
    if (!rc) {
        if (n) {
            vlayout_kernel<<<grid_for((uint64_t)n * 32, 256, g->sm_count), 256, 0, s>>>(g->rowptr, g->col, n, dnp, del);
            vparts_fill<<<grid_for(n, 256, g->sm_count), 256, 0, s>>>(pstart, k, n, dparts);
        }
        if (h_node_pointer) cudaMemcpyAsync(h_node_pointer, dnp, (uint64_t)n * 4, cudaMemcpyDeviceToHost, s);
        if (h_edge_list) cudaMemcpyAsync(h_edge_list, del, (g->nnz + n) * 4, cudaMemcpyDeviceToHost, s);
        if (h_parts) cudaMemcpyAsync(h_parts, dparts, 2ull * np * 4, cudaMemcpyDeviceToHost, s);
        cudaError_t e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) rc = fail(KC_ERR_CUDA, "virtual layout: %s", cudaGetErrorString(e));
    }
    dfree(dnp);
    dfree(del);
    dfree(dparts);
    dfree(k);
    dfree(pstart);
    return rc;
}

}  // namespace kc
