// Exact core maintenance for batches of edge insertions and deletions.
//
// The reference has no edge-update path (its "dyn" drivers only use dynamic
// work queues); this subsystem is new.  Core numbers stay exact:
//   * the CSR is rewritten in one streaming pass per change set: the sorted
//     change lists become edits of the column array (entries that go, entries
//     that come before a position), and binary searches among the few edits
//     near an entry give its new place;
//   * deletions: cores only decrease, so the old cores are upper bounds; the
//     h-index iteration restarts from them with the endpoints of the deleted
//     edges active and converges to the new cores (only vertices whose
//     neighbourhood changed are revisited);
//   * insertions are split into matchings (greedy edge colouring on the
//     host).  Inserting a matching M raises a core by at most one: the
//     (k+1)-core of G+M minus M has minimum degree >= k, so it lies in the
//     k-core of G.  A vertex can rise only if it is reachable from a
//     lower-core endpoint of an edge of M through vertices of its own old core
//     (otherwise its component together with the (k+1)-core of G would already
//     be a (k+1)-core of G).  Those vertices are found by a BFS, raised to
//     min(core + 1, degree), and the h-index iteration settles them;
//   * batches above a size threshold (a larger one for batches of deletions
//     only) are applied in one rewrite and followed by a full decomposition,
//     which is cheaper than many rounds.
#include <algorithm>
#include <chrono>
#include <cstring>
#include <vector>

#include "kc_device.cuh"
#include "kc_internal.h"

namespace kc {

static int grid_of(const Graph *g, uint64_t items) {
    uint64_t b = (items + 255) / 256;
    uint64_t cap = (uint64_t)std::max(g->sm_count, 1) * 16;
    return (int)std::max<uint64_t>(1, std::min(b, cap));
}

// Entries of the ascending a[0..len) below x.
template <class T>
__device__ __forceinline__ uint64_t count_below(const T *__restrict__ a, uint64_t len, T x) {
    uint64_t lo = 0, hi = len;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (__ldg(&a[mid]) < x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// The same by a warp, 32 probes at a time: three dependent reads for lists of
// up to 32,768 edits instead of fifteen, which is what a CTA of the rewrite
// waits for before it can start.
template <class T>
__device__ __forceinline__ uint64_t warp_count_below(const T *__restrict__ a, uint64_t len, T x) {
    const unsigned lane = threadIdx.x & 31;
    uint64_t lo = 0, hi = len;
    while (hi - lo > 32) {
        const uint64_t step = (hi - lo + 31) / 32, p = lo + lane * step + step - 1;  // the last entry of part `lane`
        lo += step * __popc(__ballot_sync(KC_FULL_MASK, p < hi && __ldg(&a[p]) < x));
        if (lo > hi) lo = hi;
        if (hi - lo > step) hi = lo + step;
    }
    const uint64_t p = lo + lane;
    return lo + __popc(__ballot_sync(KC_FULL_MASK, p < hi && __ldg(&a[p]) < x));
}

// ------------------------------------------------------------ change lists ----
// A change list is its directed entries (row << 32 | column, both directions of
// every listed edge) in ascending order; self-loops and padding are ~0 and come
// last.  Index 0 below is the deletions, 1 the insertions.
constexpr int CH_TILE = 2048;  // entries sorted by one CTA
// Up to this many entries a list is sorted by tiles that rank their entries in
// each other; longer ones go through the CSR builder, whose passes over all
// vertices and dozens of launches then weigh less than the ranking, which
// grows with the square.  Two updates of R-MAT 18 / 20 / 22, tiles against
// builder: 130,000 entries 4.17 / 7.48 / 9.67 against 4.52 / 7.80 / 10.30 ms,
// 260,000 entries the same within 2%, 520,000 entries (18, 22) 6.60 / 15.4
// against 4.89 / 13.9 ms.
constexpr uint64_t CH_TILED_MAX = 1ull << 17;

struct ChangeLists {
    const uint32_t *src[2], *dst[2];
    uint64_t m[2];           // listed edges
    unsigned tiles[2];       // of CH_TILE entries
    unsigned long long *run[2], *keys[2];  // [tiles * CH_TILE] sorted tiles, the sorted list
};

// What the rewrite of the CSR reports back.
struct RewriteOut {
    unsigned long long edits[2];  // directed entries deleted, inserted
    unsigned long long vnodes;    // of the new graph, as graph_finish counts them
    unsigned int max_deg, err;
};

// Entries of one tile, in ascending order (bitonic in shared memory: 66 steps
// of one exchange per thread, bound by their barriers; 17 us at any length up
// to a wave of tiles).
__global__ void __launch_bounds__(CH_TILE / 2) change_tiles(ChangeLists L, uint32_t n, RewriteOut *out) {
    __shared__ unsigned long long key[CH_TILE];
    const int w = blockIdx.x >= L.tiles[0];
    const uint64_t t0 = (uint64_t)(blockIdx.x - (w ? L.tiles[0] : 0u)) * CH_TILE;
    bool bad = false;
    for (unsigned i = threadIdx.x; i < CH_TILE; i += blockDim.x) {
        const uint64_t e = t0 + i;
        unsigned long long k = ~0ull;
        if (e < 2 * L.m[w]) {
            const uint32_t u = L.src[w][e >> 1], v = L.dst[w][e >> 1];
            if (u >= n || v >= n) bad = true;
            else if (u != v) k = (e & 1) ? ((unsigned long long)v << 32 | u) : ((unsigned long long)u << 32 | v);
        }
        key[i] = k;
    }
    if (__syncthreads_or(bad) && threadIdx.x == 0) out->err = 1;
    for (unsigned size = 2; size <= CH_TILE; size <<= 1)
        for (unsigned stride = size >> 1; stride > 0; stride >>= 1) {
            const unsigned i = 2 * threadIdx.x - (threadIdx.x & (stride - 1));
            const unsigned long long x = key[i], y = key[i + stride];
            if ((x > y) == ((i & size) == 0)) {
                key[i] = y;
                key[i + stride] = x;
            }
            __syncthreads();
        }
    for (unsigned i = threadIdx.x; i < CH_TILE; i += blockDim.x) L.run[w][t0 + i] = key[i];
}

// Merges the tiles: an entry's place in the list is its place in its own tile
// plus its rank in every other one (equal entries keep the order of their
// tiles).  The searches of different tiles do not depend on each other, so four
// run at a time: 14 us for ten tiles.  Both kernels stand for the CSR build of
// a change list, 125 us of passes over 4 M vertices.
__global__ void __launch_bounds__(256) change_ranks(ChangeLists L) {
    constexpr unsigned PER = CH_TILE / 256;
    unsigned b = blockIdx.x;
    const int w = b >= L.tiles[0] * PER;
    if (w) b -= L.tiles[0] * PER;
    const unsigned t = b / PER, tiles = L.tiles[w];
    const unsigned i = (b % PER) * 256 + threadIdx.x;
    const unsigned long long *run = L.run[w];
    const unsigned long long x = run[(uint64_t)t * CH_TILE + i];
    uint64_t rank = i;
    constexpr int Q = 4;
    for (unsigned o = 0; o < tiles; o += Q) {
        unsigned pos[Q] = {};
#pragma unroll
        for (unsigned step = CH_TILE / 2; step > 0; step >>= 1)
#pragma unroll
            for (int q = 0; q < Q; q++) {
                if (o + q >= tiles) continue;
                const unsigned long long y = __ldg(&run[(uint64_t)(o + q) * CH_TILE + pos[q] + step - 1]);
                if (y < x || (y == x && o + q < t)) pos[q] += step;
            }
#pragma unroll
        for (int q = 0; q < Q; q++) {
            if (o + q >= tiles || o + q == t) continue;
            const unsigned long long y = __ldg(&run[(uint64_t)(o + q) * CH_TILE + pos[q]]);  // pos <= CH_TILE - 1
            rank += pos[q] + (y < x || (y == x && o + q < t) ? 1u : 0u);
        }
    }
    L.keys[w][rank] = x;
}

// The entries of a change list that the CSR builder sorted (one warp per 32
// rows: most of them are empty).
__global__ void list_keys(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ col, uint32_t n,
                          unsigned long long *keys) {
    const unsigned lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t v0 = blockIdx.x * (uint64_t)blockDim.x + (threadIdx.x & ~31u); v0 < n; v0 += stride) {
        const uint64_t v = v0 + lane;
        const int64_t a = v < n ? rowptr[v] : 0, z = v < n ? rowptr[v + 1] : 0;
        unsigned rows = __ballot_sync(KC_FULL_MASK, z > a);
        while (rows) {
            const int l = __ffs(rows) - 1;
            rows &= rows - 1;
            const int64_t ra = __shfl_sync(KC_FULL_MASK, a, l), rz = __shfl_sync(KC_FULL_MASK, z, l);
            for (int64_t e = ra + lane; e < rz; e += 32) keys[e] = (unsigned long long)(v0 + l) << 32 | col[e];
        }
    }
}

// ------------------------------------------------------------- the rewrite ----
// Sorted change lists turn into edits of the column array: positions of entries
// that go, ascending, and positions before which an entry comes, ascending with
// their keys.  The rewrite needs nothing per row: an old entry at e moves to
// e - (deletions before e) + (insertions at or before e), and insertion k at
// position p lands on p - (deletions before p) + k.
struct Edits {
    const unsigned long long *keys[2];
    uint64_t len[2];
    unsigned blocks[2];   // of 256 entries
    int64_t *found[2];    // [len] position of every entry's edit, -1: none
    uint32_t *count;      // [blocks[0] + blocks[1]] edits per block
    const int64_t *base;  // prefix of count, or null: the few counts are added up where they are needed
    int64_t *pos[2];      // the edits
    unsigned long long *ikey;
};

// Which entries change the graph: a deletion that is in its row and not among
// the insertions, an insertion that is not in its row; each once.
__global__ void __launch_bounds__(256) plan_edits(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ col,
                                                  Edits E) {
    const int w = blockIdx.x >= E.blocks[0];
    const uint64_t j = (uint64_t)(blockIdx.x - (w ? E.blocks[0] : 0u)) * 256 + threadIdx.x;
    bool edit = false;
    if (j < E.len[w]) {
        const unsigned long long k = E.keys[w][j];
        int64_t at = -1;
        if (k != ~0ull && (j == 0 || E.keys[w][j - 1] != k)) {
            const int64_t r0 = rowptr[k >> 32];
            const uint64_t len = (uint64_t)(rowptr[(k >> 32) + 1] - r0);
            const uint32_t x = (uint32_t)k;
            const uint64_t p = count_below(col + r0, len, x);
            const bool there = p < len && col[r0 + p] == x;
            if (w) {
                edit = !there;
            } else if (there) {
                const uint64_t q = count_below(E.keys[1], E.len[1], k);
                edit = !(q < E.len[1] && E.keys[1][q] == k);  // deleted and inserted: it stays
            }
            if (edit) at = r0 + (int64_t)p;
        }
        E.found[w][j] = at;
    }
    const int c = __syncthreads_count(edit);
    if (threadIdx.x == 0) E.count[blockIdx.x] = (uint32_t)c;
}

__global__ void __launch_bounds__(256) place_edits(Edits E, RewriteOut *out) {
    __shared__ unsigned part[8];
    __shared__ unsigned long long before;
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int w = blockIdx.x >= E.blocks[0];
    const unsigned first = w ? E.blocks[0] : 0u;
    if (threadIdx.x == 0) before = E.base ? (unsigned long long)(E.base[blockIdx.x] - E.base[first]) : 0ull;
    __syncthreads();
    if (!E.base) {
        unsigned s = 0;
        for (unsigned b = first + threadIdx.x; b < blockIdx.x; b += 256) s += E.count[b];
        s = __reduce_add_sync(KC_FULL_MASK, s);
        if (lane == 0 && s) atomicAdd(&before, (unsigned long long)s);
    }
    const uint64_t j = (uint64_t)(blockIdx.x - first) * 256 + threadIdx.x;
    const int64_t at = j < E.len[w] ? E.found[w][j] : -1;
    const unsigned m = __ballot_sync(KC_FULL_MASK, at >= 0);
    if (lane == 0) part[warp] = __popc(m);
    __syncthreads();
    unsigned long long o = before + __popc(m & ((1u << lane) - 1u));
    for (unsigned i = 0; i < warp; i++) o += part[i];
    if (at >= 0) {
        E.pos[w][o] = at;
        if (w) E.ikey[o] = E.keys[1][j];
    }
    if (threadIdx.x == 255 && blockIdx.x == first + E.blocks[w] - 1) out->edits[w] = o + (at >= 0 ? 1 : 0);
}

// New row offsets, and the new graph's largest degree and virtual-node count
// from the same pass.  Each CTA looks up the edits of its rows once; a thread
// searches them for its nine rows side by side (the hubs' tile holds most of
// the edits, and one search after the other there outlasts the other tiles).
constexpr unsigned ROW_TILE = 2048;
__global__ void __launch_bounds__(256) shift_rows(const int64_t *__restrict__ rowptr, uint32_t n,
                                                  const int64_t *__restrict__ dpos,
                                                  const unsigned long long *__restrict__ ikey, RewriteOut *out,
                                                  int64_t *nrow) {
    __shared__ int64_t off[ROW_TILE + 1];
    __shared__ uint64_t cut[4];
    __shared__ unsigned long long vn_sum;
    __shared__ unsigned md_max;
    const uint64_t v0 = (uint64_t)blockIdx.x * ROW_TILE;
    const uint64_t v1 = v0 + ROW_TILE < n ? v0 + ROW_TILE : n;
    const unsigned rows = (unsigned)(v1 - v0);
    constexpr unsigned PER = ROW_TILE / 256 + 1;
    int64_t old[PER];  // on their way while the edits are looked up
#pragma unroll
    for (unsigned j = 0; j < PER; j++) {
        const unsigned i = j * 256 + threadIdx.x;
        if (i <= rows) old[j] = rowptr[v0 + i];
    }
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < 4) {
        const uint64_t v = warp & 1 ? v1 : v0;
        const uint64_t c = warp < 2 ? warp_count_below(dpos, out->edits[0], rowptr[v])
                                    : warp_count_below(ikey, out->edits[1], (unsigned long long)v << 32);
        if (lane == 0) cut[warp] = c;
    }
    if (threadIdx.x == 128) {
        vn_sum = 0;
        md_max = 0;
    }
    __syncthreads();
    const uint64_t d0 = cut[0], dn = cut[1] - d0, i0 = cut[2], in = cut[3] - i0;
    uint64_t gone[PER] = {}, come[PER] = {};
    for (uint64_t step = dn ? 1ull << (63 - __clzll((long long)dn)) : 0; step; step >>= 1)
#pragma unroll
        for (unsigned j = 0; j < PER; j++)
            if (gone[j] + step <= dn && j * 256 + threadIdx.x <= rows && __ldg(&dpos[d0 + gone[j] + step - 1]) < old[j])
                gone[j] += step;
    for (uint64_t step = in ? 1ull << (63 - __clzll((long long)in)) : 0; step; step >>= 1)
#pragma unroll
        for (unsigned j = 0; j < PER; j++)
            if (come[j] + step <= in && (__ldg(&ikey[i0 + come[j] + step - 1]) >> 32) < v0 + j * 256 + threadIdx.x)
                come[j] += step;
#pragma unroll
    for (unsigned j = 0; j < PER; j++) {
        const unsigned i = j * 256 + threadIdx.x;
        if (i > rows) continue;
        off[i] = old[j] - (int64_t)(d0 + gone[j]) + (int64_t)(i0 + come[j]);
        if (i < rows || v1 == n) nrow[v0 + i] = off[i];
    }
    __syncthreads();
    unsigned md = 0;
    unsigned long long vn = 0;
    for (unsigned i = threadIdx.x; i < rows; i += 256) {
        const uint64_t d = (uint64_t)(off[i + 1] - off[i]);
        md = max(md, (unsigned)d);
        vn += (d + 31) / 32;
    }
    md = __reduce_max_sync(KC_FULL_MASK, md);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vn += __shfl_xor_sync(KC_FULL_MASK, vn, o);
    if (lane == 0) {
        atomicMax(&md_max, md);
        atomicAdd(&vn_sum, vn);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicMax(&out->max_deg, md_max);
        atomicAdd(&out->vnodes, vn_sum);
    }
}

// The new column array.  A CTA takes a tile of old entries and looks up the
// edits in it; its warps narrow them to chunks of 512 entries, and a chunk
// without edits (with 10^4 edges on 128 M entries all but one in seven) is a
// plain copy with sixteen loads in flight per lane.  Bound by memory: the two
// arrays do not share alignment, so accesses stay 4 bytes wide per lane and the
// rate comes from 40 warps per SM: 128 M entries with 20,000 edits in 165 us
// (6.2 TB/s; 172 us with four CTAs per SM, 202 us with the tile's edits looked
// up by one thread each).  Runs of unchanged rows copied apart from the changed
// rows, which warps merged entry by entry, took 260 + 95 us.
constexpr uint64_t MOVE_TILE = 8192;
constexpr unsigned MOVE_CHUNK = 512;
__global__ void __launch_bounds__(256, 5) move_entries(const uint32_t *__restrict__ col, uint64_t nnz,
                                                    const int64_t *__restrict__ dpos, const int64_t *__restrict__ ipos,
                                                    const unsigned long long *__restrict__ ikey,
                                                    const RewriteOut *__restrict__ out, uint32_t *ncol) {
    __shared__ uint64_t cut[4];
    const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint64_t t0 = (uint64_t)blockIdx.x * MOVE_TILE;
    const bool last = t0 + MOVE_TILE >= nnz;
    const uint64_t t1 = last ? nnz : t0 + MOVE_TILE;
    if (warp < 4) {
        const uint64_t len = out->edits[warp >> 1];
        const uint64_t c = warp == 3 && last ? len  // those behind the last entry too
                                             : warp_count_below(warp < 2 ? dpos : ipos, len, (int64_t)(warp & 1 ? t1 : t0));
        if (lane == 0) cut[warp] = c;
    }
    __syncthreads();
    const uint64_t d0 = cut[0], d1 = cut[1], i0 = cut[2], i1 = cut[3];
    for (uint64_t k = i0 + threadIdx.x; k < i1; k += 256) {
        const int64_t p = ipos[k];
        ncol[(uint64_t)p - d0 - count_below(dpos + d0, d1 - d0, p) + k] = (uint32_t)ikey[k];
    }
    for (uint64_t c = t0 + warp * MOVE_CHUNK; c < t1; c += 8 * MOVE_CHUNK) {
        const uint64_t ce = c + MOVE_CHUNK < t1 ? c + MOVE_CHUNK : t1;
        const uint64_t a = d0 + count_below(dpos + d0, d1 - d0, (int64_t)c);
        const uint64_t an = d0 + count_below(dpos + d0, d1 - d0, (int64_t)ce) - a;
        const uint64_t b = i0 + count_below(ipos + i0, i1 - i0, (int64_t)c);
        const uint64_t bn = i0 + count_below(ipos + i0, i1 - i0, (int64_t)ce) - b;
        uint32_t x[MOVE_CHUNK / 32];
#pragma unroll
        for (unsigned i = 0; i < MOVE_CHUNK / 32; i++) {
            const uint64_t e = c + i * 32 + lane;
            if (e < ce) x[i] = __ldcs(&col[e]);
        }
        if (an == 0 && bn == 0) {
#pragma unroll
            for (unsigned i = 0; i < MOVE_CHUNK / 32; i++) {
                const uint64_t e = c + i * 32 + lane;
                if (e < ce) ncol[e - a + b] = x[i];
            }
        } else {
#pragma unroll
            for (unsigned i = 0; i < MOVE_CHUNK / 32; i++) {
                const uint64_t e = c + i * 32 + lane;
                if (e >= ce) continue;
                const uint64_t g = count_below(dpos + a, an, (int64_t)e);
                if (g < an && dpos[a + g] == (int64_t)e) continue;
                ncol[e - a - g + b + count_below(ipos + b, bn, (int64_t)e + 1)] = x[i];
            }
        }
    }
}

// Rows sorted and without repeated neighbours (required by the merge).
// Counts entries that are not strictly above their predecessor in the same
// row.  Each CTA checks one tile of entries; the row starts falling in the
// tile are marked in shared memory first, so hub rows split over many CTAs.
constexpr uint64_t CHECK_TILE = 8192;
__global__ void rows_simple(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ col, uint32_t n,
                            uint64_t nnz, unsigned long long *bad) {
    __shared__ uint32_t starts[CHECK_TILE / 32];
    __shared__ uint32_t first_row;
    unsigned long long b = 0;
    for (uint64_t t0 = blockIdx.x * CHECK_TILE; t0 < nnz; t0 += (uint64_t)gridDim.x * CHECK_TILE) {
        const uint64_t t1 = t0 + CHECK_TILE < nnz ? t0 + CHECK_TILE : nnz;
        for (unsigned i = threadIdx.x; i < CHECK_TILE / 32; i += blockDim.x) starts[i] = 0;
        if (threadIdx.x == 0) {
            // the last row starting at or before t0
            uint32_t lo = 0, hi = n;
            while (lo < hi) {
                const uint32_t mid = (lo + hi + 1) >> 1;
                if ((uint64_t)rowptr[mid] <= t0) lo = mid;
                else hi = mid - 1;
            }
            first_row = lo;
        }
        __syncthreads();
        for (uint64_t v = first_row + threadIdx.x; v < n && (uint64_t)rowptr[v] < t1; v += blockDim.x) {
            const uint64_t r = (uint64_t)rowptr[v];
            if (r >= t0) atomicOr(&starts[(r - t0) >> 5], 1u << ((r - t0) & 31));
        }
        __syncthreads();
        for (uint64_t e = t0 + threadIdx.x; e < t1; e += blockDim.x) {
            const uint64_t o = e - t0;
            const bool is_start = (starts[o >> 5] >> (o & 31)) & 1u;
            if (!is_start && e > 0) b += col[e] <= col[e - 1];
        }
        __syncthreads();
    }
    if (b) atomicAdd(bad, b);
}

// Roots of a matching: the endpoint(s) with the smaller old core.
__global__ void matching_roots(const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst, uint64_t m,
                               const uint32_t *__restrict__ core, uint32_t *visited, uint32_t *out,
                               unsigned long long *out_len) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t a = src[i], b = dst[i];
        const uint32_t ca = core[a], cb = core[b];
        const uint32_t k = min(ca, cb);
        const uint32_t ends[2] = {a, b};
        const uint32_t cs[2] = {ca, cb};
        for (int t = 0; t < 2; t++) {
            if (cs[t] != k) continue;
            const uint32_t v = ends[t];
            const unsigned bit = 1u << (v & 31);
            if (atomicOr(&visited[v >> 5], bit) & bit) continue;
            out[atomicAdd(out_len, 1ull)] = v;
        }
    }
}

// Entries [e0, e1) of the row of a frontier vertex of old core k: neighbours of
// the same old core that are not yet visited go to the next frontier and to the
// candidate list (one warp).
__device__ __forceinline__ void subcore_entries(const uint32_t *__restrict__ col, const uint32_t *__restrict__ core,
                                                int64_t e0, int64_t e1, uint32_t k, unsigned lane, uint32_t *visited,
                                                uint32_t *next, unsigned long long *next_len, uint32_t *cand,
                                                unsigned long long *cand_len) {
    constexpr int U = 4;
    for (int64_t e = e0 + lane; e < e1; e += 32 * U) {
        uint32_t u[U], c[U];
#pragma unroll
        for (int i = 0; i < U; i++) u[i] = e + 32 * i < e1 ? col[e + 32 * i] : 0u;
#pragma unroll
        for (int i = 0; i < U; i++) c[i] = e + 32 * i < e1 ? core[u[i]] : ~k;
#pragma unroll
        for (int i = 0; i < U; i++) {
            if (c[i] != k) continue;
            const unsigned bit = 1u << (u[i] & 31);
            if (__ldcg(&visited[u[i] >> 5]) & bit) continue;
            if (atomicOr(&visited[u[i] >> 5], bit) & bit) continue;
            next[atomicAdd(next_len, 1ull)] = u[i];
            cand[atomicAdd(cand_len, 1ull)] = u[i];
        }
    }
}

// One BFS level over edges joining vertices of equal old core, one warp per
// frontier vertex.  Rows above BFS_CHUNK entries are listed chunk by chunk for
// subcore_chunks: endpoints of inserted edges are often hubs, whose rows one
// warp walked at two dependent reads per 32 entries (updates of 100 / 400 edges,
// half insertions: R-MAT 22 5.59 / 7.14 -> 3.60 / 5.20 ms, R-MAT 18 2.22 / 4.09
// -> 1.89 / 3.55).
constexpr uint32_t BFS_CHUNK = 1024;
__global__ void subcore_bfs(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ col,
                            const uint32_t *__restrict__ core, const uint32_t *__restrict__ front, uint64_t flen,
                            uint32_t *visited, uint32_t *next, unsigned long long *next_len, uint32_t *cand,
                            unsigned long long *cand_len, unsigned long long *chunks, unsigned long long *chunks_len) {
    const unsigned lane = threadIdx.x & 31;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t i = warp; i < flen; i += nw) {
        const uint32_t v = front[i];
        const uint32_t k = core[v];  // on its way with the offsets
        const int64_t e0 = rowptr[v], e1 = rowptr[v + 1];
        if (e1 - e0 > BFS_CHUNK) {
            const unsigned long long n = (unsigned long long)(e1 - e0 + BFS_CHUNK - 1) / BFS_CHUNK;
            unsigned long long at = 0;
            if (lane == 0) at = atomicAdd(chunks_len, n);
            at = __shfl_sync(KC_FULL_MASK, at, 0);
            for (unsigned long long c = lane; c < n; c += 32) chunks[at + c] = (unsigned long long)v << 32 | c;
            continue;
        }
        subcore_entries(col, core, e0, e1, k, lane, visited, next, next_len, cand, cand_len);
    }
}

__global__ void subcore_chunks(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ col,
                               const uint32_t *__restrict__ core, const unsigned long long *__restrict__ chunks,
                               const unsigned long long *__restrict__ chunks_len, uint32_t *visited, uint32_t *next,
                               unsigned long long *next_len, uint32_t *cand, unsigned long long *cand_len) {
    const unsigned lane = threadIdx.x & 31;
    const uint64_t warp = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    const uint64_t n = *chunks_len;
    for (uint64_t i = warp; i < n; i += nw) {
        const uint32_t v = (uint32_t)(chunks[i] >> 32);
        const int64_t e0 = rowptr[v] + (int64_t)(uint32_t)chunks[i] * BFS_CHUNK;
        const int64_t e1 = min(rowptr[v + 1], e0 + (int64_t)BFS_CHUNK);
        subcore_entries(col, core, e0, e1, core[v], lane, visited, next, next_len, cand, cand_len);
    }
}

// Raise candidates by one (at most to their degree): new upper bounds.
__global__ void raise_bounds(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ list, uint64_t len,
                             uint32_t *core) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < len; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t v = list[i];
        const uint32_t d = (uint32_t)(rowptr[v + 1] - rowptr[v]);
        core[v] = min(core[v] + 1u, d);
    }
}

// Endpoints of an edge list as a vertex list (duplicates allowed).
__global__ void endpoints(const uint32_t *__restrict__ src, const uint32_t *__restrict__ dst, uint64_t m,
                          uint32_t *out) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        out[2 * i] = src[i];
        out[2 * i + 1] = dst[i];
    }
}

// Scratch arrays of one call, freed when the call returns (after the call's
// stream has finished with them, so an early error return cannot free memory
// that a launched kernel still uses).
struct Scratch {
    cudaStream_t stream = nullptr;
    std::vector<void *> ptrs;
    template <class T>
    int get(T **p, uint64_t count, const char *what) {
        int rc = dalloc(p, std::max<uint64_t>(count, 1), what);
        if (!rc) ptrs.push_back(*p);
        return rc;
    }
    ~Scratch() {
        if (stream && !ptrs.empty()) cudaStreamSynchronize(stream);
        for (void *p : ptrs) dfree(p);
    }
};

// Rewrites g's CSR: minus the edges of `del`, plus the edges of `ins` (both
// undirected edge lists on the device; either may be empty).  Counts the
// undirected edges actually deleted / inserted.  The graph stays as it was
// until the rewrite is known to have succeeded; the host waits once, at its end.
static int apply_changes(Graph *g, const uint32_t *d_isrc, const uint32_t *d_idst, uint64_t mi, const uint32_t *d_dsrc,
                         const uint32_t *d_ddst, uint64_t md, uint64_t *n_del, uint64_t *n_ins) {
    cudaStream_t s = g->stream;
    const uint32_t n = g->n;
    const uint64_t m[2] = {md, mi};
    const uint32_t *src[2] = {d_dsrc, d_isrc}, *dst[2] = {d_ddst, d_idst};
    // long lists: sorted by the builder, like any graph
    Graph lists[2];
    ChangeLists L{};
    Edits E{};
    for (int w = 0; w < 2; w++) {
        E.len[w] = 2 * m[w];
        if (2 * m[w] <= CH_TILED_MAX) {
            L.src[w] = src[w];
            L.dst[w] = dst[w];
            L.m[w] = m[w];
            L.tiles[w] = (unsigned)((2 * m[w] + CH_TILE - 1) / CH_TILE);
            continue;
        }
        Graph &q = lists[w];
        q.device = g->device;
        q.sm_count = g->sm_count;
        // borrows g's stream only while it is built (its destructor would
        // otherwise destroy it)
        q.stream = s;
        const int rc = build_csr_from_edges(&q, src[w], dst[w], m[w], n, KC_EDGES_DEDUP);
        q.stream = nullptr;
        if (rc) return rc;
        E.len[w] = q.nnz;
    }
    for (int w = 0; w < 2; w++) E.blocks[w] = (unsigned)((E.len[w] + 255) / 256);
    const unsigned blocks = E.blocks[0] + E.blocks[1];
    // one allocation for everything of the lists' size: the report, per list
    // the sorted tiles (later the edits found), the keys and the edits, the
    // counts and their prefix
    uint64_t cap[2], words = sizeof(RewriteOut) / 8;
    for (int w = 0; w < 2; w++) {
        cap[w] = std::max<uint64_t>((uint64_t)L.tiles[w] * CH_TILE, E.len[w]);
        words += 3 * cap[w];
    }
    words += cap[1] + ((uint64_t)blocks + 1) / 2 + blocks + 2;
    Scratch sc;
    sc.stream = s;
    unsigned long long *w8 = nullptr;
    KC_TRY(sc.get(&w8, words, "change lists"));
    RewriteOut *out = reinterpret_cast<RewriteOut *>(w8);
    unsigned long long *next = w8 + sizeof(RewriteOut) / 8;
    for (int w = 0; w < 2; w++) {
        L.run[w] = next;
        L.keys[w] = next + cap[w];
        E.keys[w] = L.keys[w];
        E.found[w] = reinterpret_cast<int64_t *>(L.run[w]);
        E.pos[w] = reinterpret_cast<int64_t *>(next + 2 * cap[w]);
        next += 3 * cap[w];
    }
    E.ikey = next;
    next += cap[1];
    int64_t *base = reinterpret_cast<int64_t *>(next);
    next += blocks + 1;
    E.count = reinterpret_cast<uint32_t *>(next);
    KC_CUDA(cudaMemsetAsync(out, 0, sizeof(RewriteOut), s));
    const unsigned tiles = L.tiles[0] + L.tiles[1];
    if (tiles) {
        change_tiles<<<tiles, CH_TILE / 2, 0, s>>>(L, n, out);
        change_ranks<<<tiles * (CH_TILE / 256), 256, 0, s>>>(L);
    }
    for (int w = 0; w < 2; w++)
        if (lists[w].nnz)
            list_keys<<<grid_of(g, n), 256, 0, s>>>(lists[w].rowptr, lists[w].col, n, L.keys[w]);
    if (blocks) {
        plan_edits<<<blocks, 256, 0, s>>>(g->rowptr, g->col, E);
        if (blocks > 2 * CH_TILED_MAX / 256) {
            KC_TRY(exclusive_scan_u32_i64(E.count, base, blocks, s));
            E.base = base;
        }
        place_edits<<<blocks, 256, 0, s>>>(E, out);
    }
    int64_t *rp_new = nullptr;
    uint32_t *col_new = nullptr;
    KC_TRY(dalloc(&rp_new, (uint64_t)n + 1, "row offsets"));
    int rc = dalloc(&col_new, g->nnz + E.len[1] + 1, "column ids");
    if (rc) {
        cudaStreamSynchronize(s);
        dfree(rp_new);
        return rc;
    }
    shift_rows<<<(unsigned)(((uint64_t)n + ROW_TILE - 1) / ROW_TILE + (n == 0)), 256, 0, s>>>(
        g->rowptr, n, E.pos[0], E.ikey, out, rp_new);
    move_entries<<<(unsigned)((g->nnz + MOVE_TILE - 1) / MOVE_TILE + (g->nnz == 0)), 256, 0, s>>>(
        g->col, g->nnz, E.pos[0], E.pos[1], E.ikey, out, col_new);
    RewriteOut h{};
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, out, sizeof(h), cudaMemcpyDeviceToHost, s);
    const cudaError_t es = cudaStreamSynchronize(s);
    if (e == cudaSuccess) e = es;
    if (e != cudaSuccess) rc = fail(KC_ERR_CUDA, "CSR merge: %s", cudaGetErrorString(e));
    else if (h.err) rc = fail(KC_ERR_INVALID, "edge endpoint >= n (%u)", n);
    if (rc) {
        dfree(rp_new);
        dfree(col_new);
        return rc;
    }
    dfree(g->rowptr);
    dfree(g->col);
    g->rowptr = rp_new;
    g->col = col_new;
    g->nnz = g->nnz - h.edits[0] + h.edits[1];
    g->max_deg = h.max_deg;
    g->num_vnodes = h.vnodes;
    *n_del = h.edits[0] / 2;
    *n_ins = h.edits[1] / 2;
    return KC_OK;
}

static int ensure_maint(Graph *g) {
    if (!g->mfront[0]) {
        const uint64_t n = g->n;
        KC_TRY(dalloc(&g->mfront[0], n + 1, "bfs frontier"));
        KC_TRY(dalloc(&g->mfront[1], n + 1, "bfs frontier"));
        KC_TRY(dalloc(&g->mcand, n + 1, "candidates"));
        KC_TRY(dalloc(&g->mvisit, (n + 31) / 32 + 1, "bfs visited"));
        KC_TRY(dalloc(&g->mcount, 4, "bfs counters"));
    }
    return KC_OK;
}

// Subcore candidates of one inserted matching (already in the CSR); returns
// their number, the list in g->mcand.
static int subcore_candidates(Graph *g, const uint32_t *d_src, const uint32_t *d_dst, uint64_t m, uint64_t *count) {
    cudaStream_t s = g->stream;
    KC_TRY(ensure_maint(g));
    unsigned long long *lens = g->mcount;  // [0] frontier a, [1] frontier b, [2] candidates, [3] chunks of long rows
    Scratch sc;
    sc.stream = s;
    unsigned long long *chunks = nullptr;
    KC_TRY(sc.get(&chunks, 2 * (g->nnz / BFS_CHUNK) + 1, "bfs chunks"));
    KC_CUDA(cudaMemsetAsync(g->mvisit, 0, (((uint64_t)g->n + 31) / 32) * 4, s));
    KC_CUDA(cudaMemsetAsync(lens, 0, 32, s));
    matching_roots<<<grid_of(g, m), 256, 0, s>>>(d_src, d_dst, m, g->core, g->mvisit, g->mfront[0], &lens[0]);
    unsigned long long flen = 0;
    KC_CUDA(cudaMemcpyAsync(&flen, &lens[0], 8, cudaMemcpyDeviceToHost, s));
    KC_CUDA(cudaStreamSynchronize(s));
    // the roots are candidates too
    KC_CUDA(cudaMemcpyAsync(g->mcand, g->mfront[0], flen * 4, cudaMemcpyDeviceToDevice, s));
    unsigned long long total = flen;
    KC_CUDA(cudaMemcpyAsync(&lens[2], &total, 8, cudaMemcpyHostToDevice, s));
    int cur = 0;
    // without a long row there is nothing to list, and a search of many levels (a
    // path, a mesh) would pay a clearing and a launch on each: an edge put back
    // into a path of 20,000 vertices 446 -> 303 ms, into a ring of 200,000 joined
    // to ten on either side 278 -> 171
    const bool long_rows = g->max_deg > BFS_CHUNK;
    for (uint32_t level = 0; flen > 0; level++) {
        if (level > g->n) return fail(KC_ERR_CAPACITY, "subcore search did not terminate");
        const int nxt = cur ^ 1;
        KC_CUDA(cudaMemsetAsync(&lens[nxt], 0, 8, s));
        if (long_rows) KC_CUDA(cudaMemsetAsync(&lens[3], 0, 8, s));
        subcore_bfs<<<grid_of(g, flen * 32), 256, 0, s>>>(g->rowptr, g->col, g->core, g->mfront[cur], flen, g->mvisit,
                                                          g->mfront[nxt], &lens[nxt], g->mcand, &lens[2], chunks,
                                                          &lens[3]);
        if (long_rows)
            subcore_chunks<<<grid_of(g, 1u << 20), 256, 0, s>>>(g->rowptr, g->col, g->core, chunks, &lens[3], g->mvisit,
                                                                g->mfront[nxt], &lens[nxt], g->mcand, &lens[2]);
        KC_CUDA(cudaMemcpyAsync(&flen, &lens[nxt], 8, cudaMemcpyDeviceToHost, s));
        KC_CUDA(cudaStreamSynchronize(s));
        cur = nxt;
    }
    KC_CUDA(cudaMemcpyAsync(&total, &lens[2], 8, cudaMemcpyDeviceToHost, s));
    KC_CUDA(cudaStreamSynchronize(s));
    *count = total;
    return KC_OK;
}

int graph_update(Graph *g, const uint32_t *ins_src, const uint32_t *ins_dst, uint64_t n_ins, const uint32_t *del_src,
                 const uint32_t *del_dst, uint64_t n_del, kc_update_stats *st) {
    cudaStream_t s = g->stream;
    const auto t0 = std::chrono::steady_clock::now();
    kc_update_stats out;
    memset(&out, 0, sizeof(out));
    const uint32_t n = g->n;
    // deletions alone need no matching rounds: the h-index iteration from the
    // old cores beats a full decomposition up to a few hundred thousand edges
    // (R-MAT 22: 10^3 0.45 vs 5.6 ms, 10^4 0.99 vs 5.6, 10^5 5.3 vs 6.3, 5 x 10^5
    // 8.1 vs 6.8; R-MAT 20: 5 x 10^5 3.7 vs 4.1, 10^6 4.5 vs 4.0)
    const bool incremental = n_ins + n_del <= (uint64_t)g->tune.update_incremental_max ||
                             (n_ins == 0 && n_del <= (uint64_t)g->tune.update_deletion_incremental_max);
    // The incremental path applies the deletions before it colours the
    // insertions on the host (which indexes per-vertex arrays), so it checks
    // every id first; the full path builds both change lists on the device,
    // which rejects ids >= n before the graph is rewritten.
    if (incremental) {
        for (uint64_t i = 0; i < n_ins; i++)
            if (ins_src[i] >= n || ins_dst[i] >= n) return fail(KC_ERR_INVALID, "inserted edge endpoint >= n");
        for (uint64_t i = 0; i < n_del; i++)
            if (del_src[i] >= n || del_dst[i] >= n) return fail(KC_ERR_INVALID, "deleted edge endpoint >= n");
    }
    if (!g->simple_checked) {
        unsigned long long *bad = nullptr;
        KC_TRY(dalloc(&bad, 1, "row check"));
        cudaMemsetAsync(bad, 0, 8, s);
        if (n && g->nnz) {
            const uint64_t tiles = (g->nnz + CHECK_TILE - 1) / CHECK_TILE;
            rows_simple<<<(int)std::min<uint64_t>(tiles, (uint64_t)g->sm_count * 16), 256, 0, s>>>(g->rowptr, g->col, n,
                                                                                                   g->nnz, bad);
        }
        unsigned long long hb = 0;
        cudaMemcpyAsync(&hb, bad, 8, cudaMemcpyDeviceToHost, s);
        cudaError_t e = cudaStreamSynchronize(s);
        dfree(bad);
        if (e != cudaSuccess) return fail(KC_ERR_CUDA, "row check: %s", cudaGetErrorString(e));
        if (hb) return fail(KC_ERR_UNSUPPORTED, "updates need sorted rows without parallel edges (build with KC_EDGES_DEDUP)");
        g->simple_checked = true;
    }
    if (!g->core_valid) KC_TRY(peel_run(g, s, false, nullptr));
    Scratch sc;
    sc.stream = s;
    uint32_t *d_del_s = nullptr, *d_del_d = nullptr;
    if (n_del) {
        KC_TRY(sc.get(&d_del_s, n_del, "deleted edges"));
        KC_TRY(sc.get(&d_del_d, n_del, "deleted edges"));
        KC_CUDA(cudaMemcpyAsync(d_del_s, del_src, n_del * 4, cudaMemcpyHostToDevice, s));
        KC_CUDA(cudaMemcpyAsync(d_del_d, del_dst, n_del * 4, cudaMemcpyHostToDevice, s));
    }
    if (!incremental) {
        uint32_t *d_is = nullptr, *d_id = nullptr;
        if (n_ins) {
            KC_TRY(sc.get(&d_is, n_ins, "inserted edges"));
            KC_TRY(sc.get(&d_id, n_ins, "inserted edges"));
            KC_CUDA(cudaMemcpyAsync(d_is, ins_src, n_ins * 4, cudaMemcpyHostToDevice, s));
            KC_CUDA(cudaMemcpyAsync(d_id, ins_dst, n_ins * 4, cudaMemcpyHostToDevice, s));
        }
        uint64_t nd = 0, ni = 0;
        KC_TRY(apply_changes(g, d_is, d_id, n_ins, d_del_s, d_del_d, n_del, &nd, &ni));
        KC_TRY(peel_run(g, s, false, nullptr));
        out.deleted = nd;
        out.inserted = ni;
        out.recomputed = 1;
    } else {
        if (n_del) {
            uint64_t nd = 0, ni = 0;
            KC_TRY(apply_changes(g, nullptr, nullptr, 0, d_del_s, d_del_d, n_del, &nd, &ni));
            out.deleted = nd;
            if (nd) {
                uint32_t *ends = nullptr;
                KC_TRY(sc.get(&ends, 2 * n_del, "deleted endpoints"));
                endpoints<<<grid_of(g, n_del), 256, 0, s>>>(d_del_s, d_del_d, n_del, ends);
                kc_stats hs;
                memset(&hs, 0, sizeof(hs));
                KC_TRY(hindex_run_from(g, ends, 2 * n_del, s, &hs));
                out.sweeps += hs.iterations;
            }
        }
        if (n_ins) {
            // greedy edge colouring: every colour class is a matching
            std::vector<uint32_t> color(n_ins), used;
            if (g->color_count.size() != n) g->color_count.assign(n, 0);
            uint32_t rounds = 0;
            for (uint64_t i = 0; i < n_ins; i++) {
                const uint32_t a = ins_src[i], b = ins_dst[i];
                if (a == b) {
                    color[i] = 0xffffffffu;
                    continue;
                }
                const uint32_t c = std::max(g->color_count[a], g->color_count[b]);
                color[i] = c;
                if (!g->color_count[a]) used.push_back(a);
                if (!g->color_count[b]) used.push_back(b);
                g->color_count[a] = g->color_count[b] = c + 1;
                rounds = std::max(rounds, c + 1);
            }
            for (uint32_t v : used) g->color_count[v] = 0;
            std::vector<uint64_t> cstart(rounds + 1, 0);
            for (uint64_t i = 0; i < n_ins; i++)
                if (color[i] != 0xffffffffu) cstart[color[i] + 1]++;
            for (uint32_t r = 0; r < rounds; r++) cstart[r + 1] += cstart[r];
            std::vector<uint32_t> hs_(cstart[rounds]), hd_(cstart[rounds]);
            std::vector<uint64_t> fill(cstart.begin(), cstart.end() - 1);
            for (uint64_t i = 0; i < n_ins; i++) {
                if (color[i] == 0xffffffffu) continue;
                const uint64_t p = fill[color[i]]++;
                hs_[p] = ins_src[i];
                hd_[p] = ins_dst[i];
            }
            uint32_t *d_is = nullptr, *d_id = nullptr;
            KC_TRY(sc.get(&d_is, hs_.size(), "inserted edges"));
            KC_TRY(sc.get(&d_id, hd_.size(), "inserted edges"));
            if (!hs_.empty()) {
                KC_CUDA(cudaMemcpyAsync(d_is, hs_.data(), hs_.size() * 4, cudaMemcpyHostToDevice, s));
                KC_CUDA(cudaMemcpyAsync(d_id, hd_.data(), hd_.size() * 4, cudaMemcpyHostToDevice, s));
            }
            for (uint32_t r = 0; r < rounds; r++) {
                const uint64_t m = cstart[r + 1] - cstart[r];
                if (!m) continue;
                uint64_t nd = 0, ni = 0;
                KC_TRY(apply_changes(g, d_is + cstart[r], d_id + cstart[r], m, nullptr, nullptr, 0, &nd, &ni));
                out.inserted += ni;
                out.rounds++;
                if (!ni) continue;
                uint64_t cands = 0;
                KC_TRY(subcore_candidates(g, d_is + cstart[r], d_id + cstart[r], m, &cands));
                out.candidates += cands;
                if (!cands) continue;
                raise_bounds<<<grid_of(g, cands), 256, 0, s>>>(g->rowptr, g->mcand, cands, g->core);
                kc_stats hs;
                memset(&hs, 0, sizeof(hs));
                KC_TRY(hindex_run_from(g, g->mcand, cands, s, &hs));
                out.sweeps += hs.iterations;
            }
        }
    }
    KC_CUDA(cudaStreamSynchronize(s));
    g->core_valid = true;
    out.ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    if (st) *st = out;
    return KC_OK;
}

}  // namespace kc
