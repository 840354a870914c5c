// Batched k-core decomposition of many independent graphs in one pass.
//
// The reference decomposes one graph per process (each driver's main()); a
// batch of graphs there is a loop of whole program runs.  Here a batch is a
// segmented CSR -- graph i owns vertices [vbase[i], vbase[i+1]) of one packed
// CSR and its rows reference only its own vertices -- decomposed by
// persistent kernels in which each CTA takes whole graphs from a work list
// (largest first) and peels them entirely on the SM:
//   * residual degrees and the claim bitmap of the graph live in shared memory
//     (uint16 degrees when the graph's maximum degree allows, else uint32);
//     graphs too large for shared memory use the same code on global memory;
//   * a level starts with one scan that claims every unclaimed vertex with
//     residual degree <= L (its core number is L) and queues its row in
//     chunk-sized items; warps then expand the queued rows, concatenated, and
//     decrement unclaimed neighbours with shared-memory atomics; the decrement
//     that takes a neighbour from L+1 to L claims it and queues its row for
//     the next round, so cascades need no rescan; the smallest residual degree
//     left above L is the next level (empty levels are skipped);
//   * CTA barriers (__syncthreads) replace the reference's host round trips.
// Graphs are split into size classes, each with its own kernel
// configuration, launched on forked streams; the sequence can be captured
// once as a CUDA graph and replayed.  kc_batch_autotune times a few
// configurations on the batch itself and keeps the fastest.
#include <algorithm>
#include <cstring>
#include <mutex>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include "kc_device.cuh"
#include "kc_internal.h"

namespace kc {

constexpr unsigned BATCH_MIN_CHUNK = 128;
constexpr unsigned NO_LVL = 0xffffffffu;
constexpr int BATCH_U = 8;  // row entries in flight per lane
constexpr int BATCH_GROUPS = 4;  // 8-vertex groups a thread scans per step
// Offset of a row entry within its graph: graphs in shared memory have fewer
// than 2^31 entries (larger ones go to the global-memory class).
template <bool SMEM>
struct OffOf {
    using type = uint32_t;
};
template <>
struct OffOf<false> {
    using type = int64_t;
};

struct BatchArgs {
    const int64_t *rowptr;
    const uint32_t *col;
    uint32_t *core;
    const uint32_t *vbase;
    const uint32_t *order;  // graph indices of this class, largest first
    uint32_t count;
    unsigned long long *F;            // row-chunk queue scratch (packed-graph sized)
    const unsigned long long *fbase;  // per-graph offset into F
    unsigned int *next;               // work counter of this class
    uint32_t *gdeg;                   // global-memory residual degrees (packed ids)
    uint8_t *gclaimed;                // global-memory claim flags (packed ids)
    uint32_t chunk;
    uint32_t smem_n;                  // vertex capacity of the shared-memory arrays
    unsigned long long *gtrace;       // per graph: start ns, end ns, SM id (or nullptr)
    unsigned q_cap;                   // row ranges per ring (two rings in shared memory)
    unsigned id_cap;                  // scanned claims in the shared-memory id list (at least 32)
};

// Whether vertex v has been claimed (SMEM: claim bitmap in shared memory,
// otherwise one flag byte per vertex in global memory).
template <bool SMEM>
__device__ __forceinline__ bool is_claimed(const uint32_t *bits, const uint8_t *flags, uint32_t v) {
    return SMEM ? ((bits[v >> 5] >> (v & 31)) & 1u) != 0u : flags[v] != 0;
}

// 1 << d, 0 for d >= 32.
__device__ __forceinline__ unsigned bit_or_zero(unsigned d) {
    unsigned r;
    asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(d));
    return r;
}

// One CTA per graph.  What bounds it is the chain of dependent steps -- row
// offsets, row entries, shared-memory decrements, barrier -- of every cascade
// round of every level, and with many warps the instructions issued, so the
// kernel spends as few of both as it can:
//   * a claim also sets the top bit of the vertex's residual degree, so that
//     the scan sees claimed vertices as large.  (The claim bits alone decide
//     what is claimed: a caller's asymmetric rows can wear the top bit down.)
//   * a level's scan takes the degrees 8 vertices per thread straight from
//     shared memory: one 16-byte load and a packed minimum; only groups with a
//     vertex at or below L are looked at one by one;
//   * scan claims go to a small id list; the next step reads their row offsets
//     all at once and queues row ranges of at most `chunk` entries; the claims
//     made while expanding read their own row offsets at once and queue ranges
//     the same way, so long rows spread over the warps of the next round;
//   * a round's items are shared out evenly over the warps; a warp walks its
//     items' entries as one sequence, 32 x BATCH_U at a time.  The owner of an
//     entry is counted: the items that start within a window of 32 entries set
//     one bit each (one reduction), an entry's owner is the number of starts
//     at or before it.  A round of at most one item per warp, which long chains
//     and the ends of most cascades consist of, hands nothing out, scans nothing
//     and looks no owner up, and its short rows are one window (a path of 40,000
//     vertices 35.7 -> 19.7 ms, the mix 8.6 -> 7.9, 256 small graphs 0.31 ->
//     0.25, R-MAT 20,011 / 320,000 without allocation 0.78 -> 0.65; the same
//     branch as a condition ahead of the loop, not an if and else, leaves the
//     mix at 8.8);
//   * one barrier per round (the counters of three rounds rotate);
//   * queues live in shared memory (ids: id_cap, two rings of q_cap ranges for
//     the round read and the round filled); what does not fit goes to the
//     graph's part of F in global memory.
// Measured against the kernel with alive lists, claim bits probed per scanned
// vertex and items handed out 32 to a warp: 4,096-graph mix (1.8 B row entries)
// 38.0 -> 8.6 ms, 256 graphs of up to 3,162 vertices 0.96 -> 0.29 ms.  On
// Erdos-Renyi graphs alone an SM walks 1.95 G row entries/s, 2.6 instructions
// each, the issue slots 62% busy.
// WIDE: 16-bit degrees up to 65,534 and no mark; the scan takes claimed vertices
// out by the claim bits of the group, a byte beside its degrees.
template <typename DegT, bool SMEM, bool WIDE = false>
__global__ void __launch_bounds__(1024, 1) batch_peel(BatchArgs A) {
    static_assert(!WIDE || (SMEM && sizeof(DegT) == 2), "wide degrees are 16-bit ones in shared memory");
    using Off = typename OffOf<SMEM>::type;  // entry offset within the graph
    // degrees are below it
    constexpr unsigned MARK = WIDE ? 0xffffu : 1u << (8 * sizeof(DegT) - 1);
    extern __shared__ __align__(16) unsigned char smem[];
    // cnt[r % 3]: items of round r; head[r % 3]: next item to take in round r
    __shared__ unsigned int gi_sh, idcnt, cnt[3], head[3], minlev[2];
    const unsigned tid = threadIdx.x, lane = tid & 31, nthreads = blockDim.x, nwarps = nthreads >> 5;
    const unsigned le = 0xffffffffu >> (31 - lane);  // this lane and those before it
    DegT *deg = reinterpret_cast<DegT *>(smem);
    uint32_t *bits = reinterpret_cast<uint32_t *>(smem + A.smem_n * sizeof(DegT));
    uint8_t *flags = nullptr;
    unsigned long long *ring =
        reinterpret_cast<unsigned long long *>(smem + A.smem_n * sizeof(DegT) + ((A.smem_n / 8 + 15) & ~15u));
    uint32_t *ids = reinterpret_cast<uint32_t *>(ring + 2 * A.q_cap);
    const unsigned q_cap = A.q_cap, id_cap = A.id_cap, chunk = A.chunk;
    if (tid < 3) cnt[tid] = head[tid] = 0;
    if (tid == 0) idcnt = 0;
    unsigned r = 0;  // running round number (never reset: the counters rotate across levels and graphs)
    for (;;) {
        __syncthreads();  // the previous graph's last reads of minlev are done
        if (tid == 0) {
            gi_sh = atomicAdd(A.next, 1u);
            minlev[0] = minlev[1] = NO_LVL;
        }
        __syncthreads();
        const unsigned idx = gi_sh;
        if (idx >= A.count) return;
        const uint32_t gi = A.order[idx];
        if (A.gtrace && tid == 0) {
            unsigned smid;
            asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
            A.gtrace[3ull * gi] = global_ns();
            A.gtrace[3ull * gi + 2] = smid;
        }
        const uint32_t v0 = A.vbase[gi];
        const uint32_t n = A.vbase[gi + 1] - v0;
        const int64_t *rp = A.rowptr + v0;
        const int64_t e0 = rp[0];  // the graph's entries start here
        const uint32_t *colv = A.col + e0;
        unsigned long long *F = A.F + A.fbase[gi];
        if (!SMEM) {
            // 8-vertex groups start aligned: every graph has 8 spare entries
            const uint64_t o = ((uint64_t)v0 + 8ull * gi + 7ull) & ~7ull;
            deg = reinterpret_cast<DegT *>(A.gdeg + o);
            flags = A.gclaimed + o;
        }
        const uint32_t groups = (n + 7) / 8;
        unsigned my_min = NO_LVL;
        for (uint32_t v = tid; v < groups * 8; v += nthreads) {
            uint32_t d = MARK;  // past the last vertex
            if (v < n) {
                d = (uint32_t)(rp[v + 1] - rp[v]);
                my_min = min(my_min, d);
            }
            deg[v] = (DegT)d;
            if (!SMEM) flags[v] = 0;
        }
        if (SMEM)
            for (uint32_t w = tid; w < (n + 31) / 32; w += nthreads) bits[w] = 0u;
        my_min = __reduce_min_sync(KC_FULL_MASK, my_min);
        if (lane == 0 && my_min != NO_LVL) atomicMin(&minlev[1], my_min);
        __syncthreads();
        unsigned L = minlev[1];  // the first level is the smallest degree
        // Queues the rows of the lanes' vertices v (take) as ranges of at most
        // chunk entries -- start << 24 | length, start relative to e0 -- for
        // round rr, whose list starts at F[fb] where the ring is full
        // (warp-wide call).
        auto enqueue = [&](bool take, uint32_t v, unsigned rr, unsigned fb) {
            uint32_t k = 0;
            int64_t r0 = 0, r1 = 0;
            if (take) {
                r0 = rp[v] - e0;
                r1 = rp[v + 1] - e0;
                k = (uint32_t)((r1 - r0 + chunk - 1) / chunk);
            }
            unsigned tot, ex;
            if (__any_sync(KC_FULL_MASK, k > 1)) {
                ex = warp_excl_scan(k, lane, tot);
            } else {  // one range each
                const unsigned m = __ballot_sync(KC_FULL_MASK, k != 0);
                ex = __popc(m & (le >> 1));
                tot = __popc(m);
            }
            unsigned base = 0;
            if (lane == 0 && tot) base = atomicAdd(&cnt[rr % 3], tot);
            base = __shfl_sync(KC_FULL_MASK, base, 0) + ex;
            unsigned long long *slot = ring + (rr & 1) * q_cap;
            for (uint32_t j = 0; j < k; j++, base++) {
                const int64_t s0 = r0 + (int64_t)j * chunk;
                const int64_t l = min((int64_t)chunk, r1 - s0);
                const unsigned long long it = ((unsigned long long)s0 << 24) | (unsigned long long)l;
                if (base < q_cap) slot[base] = it;
                else __stcg(&F[fb + base], it);
            }
        };
        for (unsigned lev = 0; L != NO_LVL; lev++) {  // levels
            my_min = NO_LVL;
            // ---- scan: claim every vertex at or below L ----
            unsigned min2 = 0xffffffffu;  // 16-bit degrees: packed minima of the vertices left
            for (uint32_t b = 0; b < groups; b += BATCH_GROUPS * nthreads) {
                unsigned claims = 0;  // bit 8 g + j: vertex j of the thread's g-th group
#pragma unroll
                for (int g = 0; g < BATCH_GROUPS; g++) {
                    const uint32_t c = b + g * nthreads + tid;
                    if (c >= groups) continue;
                    uint4 *p = reinterpret_cast<uint4 *>(deg) + c * (sizeof(DegT) / 2);
                    uint4 x = SMEM ? p[0] : __ldcg(p);
                    if constexpr (WIDE) {
                        const unsigned gone = reinterpret_cast<const uint8_t *>(bits)[c];
                        auto two = [&](int j) { return ((gone >> j) & 1u) * 0xffffu | ((gone >> (j + 1)) & 1u) * 0xffff0000u; };
                        x.x |= two(0);
                        x.y |= two(2);
                        x.z |= two(4);
                        x.w |= two(6);
                    }
                    unsigned low = 0;  // vertices at or below L
                    if constexpr (sizeof(DegT) == 2) {
                        unsigned gm = __vimin3_u16x2(x.x, x.y, __vimin3_u16x2(x.z, x.w, x.w));
                        if (min(gm & 0xffffu, gm >> 16) <= L) {
                            uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                            for (int j = 0; j < 8; j++) {
                                if (((w[j / 2] >> (16 * (j & 1))) & 0xffffu) <= L) {
                                    low |= 1u << j;
                                    w[j / 2] |= MARK << (16 * (j & 1));
                                }
                            }
                            if (!WIDE) p[0] = make_uint4(w[0], w[1], w[2], w[3]);
                            gm = __vimin3_u16x2(w[0], w[1], __vimin3_u16x2(w[2], w[3], w[3]));
                        }
                        min2 = __vimin3_u16x2(min2, gm, gm);
                    } else {
                        uint4 y = SMEM ? p[1] : __ldcg(p + 1);
                        uint32_t d[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            if (d[j] <= L) {
                                low |= 1u << j;
                                d[j] |= MARK;
                            }
                            my_min = min(my_min, d[j]);
                        }
                        if (low) {
                            p[0] = make_uint4(d[0], d[1], d[2], d[3]);
                            p[1] = make_uint4(d[4], d[5], d[6], d[7]);
                        }
                    }
                    if (low) {
                        if (SMEM) {
                            low &= ~(unsigned)reinterpret_cast<const uint8_t *>(bits)[c];
                            atomicOr(&bits[c >> 2], low << (8 * (c & 3)));
                        } else {
                            for (unsigned t = low; t; t &= t - 1) {
                                uint8_t *f = &flags[8 * (size_t)c + __ffs(t) - 1];
                                if (*f) low &= ~(t & (0u - t));
                                else *f = 1;
                            }
                        }
                        claims |= low << (8 * g);
                    }
                }
                if (!__any_sync(KC_FULL_MASK, claims != 0)) continue;
                if (L == 0 && lev == 0) {
                    // vertices without a row: nothing to queue
                    for (; claims; claims &= claims - 1) {
                        const unsigned j = __ffs(claims) - 1;
                        A.core[v0 + 8 * (b + (j >> 3) * nthreads + tid) + (j & 7)] = 0;
                    }
                    continue;
                }
                unsigned tot;
                unsigned pos = warp_excl_scan(__popc(claims), lane, tot);
                unsigned base = 0;
                if (lane == 0) base = atomicAdd(&idcnt, tot);
                pos += __shfl_sync(KC_FULL_MASK, base, 0);
                while (__any_sync(KC_FULL_MASK, claims != 0)) {
                    const unsigned j = __ffs(claims) - 1;  // garbage without a claim left
                    const uint32_t v = 8 * (b + (j >> 3) * nthreads + tid) + (j & 7);
                    const bool on = claims != 0, listed = pos < id_cap;
                    if (on) A.core[v0 + v] = L;
                    if (on && listed) ids[pos] = v;
                    // the id list is full: read the row offsets here
                    if (__any_sync(KC_FULL_MASK, on && !listed)) enqueue(on && !listed, v, r, 0u);
                    pos++;
                    claims &= claims - 1;
                }
            }
            if (sizeof(DegT) == 2) my_min = min(min2 & 0xffffu, min2 >> 16);
            if (my_min >= MARK) my_min = NO_LVL;
            __syncthreads();
            if (tid == 0) minlev[(lev + 1) & 1] = NO_LVL;  // every thread read it before this barrier
            const unsigned nid = min(idcnt, id_cap);
            if (nid) {
                for (unsigned b = 0; b < nid; b += nthreads) {
                    const bool on = b + tid < nid;
                    enqueue(on, on ? ids[b + tid] : 0u, r, 0u);
                }
                __syncthreads();
                if (tid == 0) idcnt = 0;
            }
            // ---- expansion rounds: the claims of a round are the next one's items ----
            unsigned fb = 0;  // F position of the current round's list
            unsigned above = NO_LVL;  // smallest old degree - (L + 2) of a decrement that left its vertex above L
            for (;;) {
                const unsigned total_items = cnt[r % 3];
                if (total_items == 0) break;
                if (tid == 0) {
                    cnt[(r + 2) % 3] = 0;   // last read when round r - 1 began
                    head[(r + 1) % 3] = 0;  // last used in round r - 2
                }
                const unsigned fb_next = fb + total_items;
                const unsigned long long *slot = ring + (r & 1) * q_cap;
                // Walks a warp's entries, U windows of 32 at a time: entry e of the
                // sequence is at rs + e of its owner, the last item with start <= e.
                // ONE: all of one item, rs the same on every lane.
                auto walk = [&](auto windows, auto one, Off rs, unsigned start, unsigned total) {
                    constexpr int U = decltype(windows)::value;
                    constexpr bool ONE = decltype(one)::value;
                    unsigned before = 0;  // items after the first that start before the window
                    for (unsigned base = 0; base < total; base += 32 * U) {
                        uint32_t u[U];
#pragma unroll
                        for (int k = 0; k < U; k++) {
                            const unsigned e = base + k * 32 + lane;
                            Off at = rs + (Off)e;
                            if constexpr (!ONE) {
                                const unsigned starts = __reduce_or_sync(KC_FULL_MASK, bit_or_zero(start - (base + k * 32)));
                                const unsigned owner = before + __popc(starts & le);
                                before += __popc(starts);
                                at = __shfl_sync(KC_FULL_MASK, rs, owner) + (Off)e;
                            }
                            u[k] = e < total ? __ldcs(&colv[at]) - v0 : NO_LVL;
                        }
                        // Decrement the unclaimed neighbours.  The decrement that
                        // moves a neighbour from L + 1 to L claims it, at core L,
                        // and queues its row; `above` tracks the smallest residual
                        // degree left above L (smaller old degrees wrap around).
                        unsigned claims = 0, old[U];
#pragma unroll
                        for (int k = 0; k < U; k++)
                            if (u[k] != NO_LVL && is_claimed<SMEM>(bits, flags, u[k])) u[k] = NO_LVL;
#pragma unroll
                        for (int k = 0; k < U; k++) {
                            old[k] = 0;
                            if (u[k] != NO_LVL) {
                                if (sizeof(DegT) == 2) {
                                    const unsigned sh = (u[k] & 1) * 16;
                                    old[k] = (atomicSub(reinterpret_cast<unsigned int *>(deg) + (u[k] >> 1), 1u << sh) >> sh) & 0xffffu;
                                } else {
                                    old[k] = atomicSub(reinterpret_cast<unsigned int *>(deg) + u[k], 1u);
                                }
                            }
                        }
#pragma unroll
                        for (int k = 0; k < U; k++) {
                            above = min(above, old[k] - (L + 2));
                            if (old[k] == L + 1) {
                                claims |= 1u << k;
                                if (SMEM) atomicOr(&bits[u[k] >> 5], 1u << (u[k] & 31));
                                else flags[u[k]] = 1;
                                if (sizeof(DegT) == 2 && !WIDE)
                                    atomicOr(reinterpret_cast<unsigned int *>(deg) + (u[k] >> 1), MARK << ((u[k] & 1) * 16));
                                else if (!WIDE)
                                    atomicOr(reinterpret_cast<unsigned int *>(deg) + u[k], MARK);
                                A.core[v0 + u[k]] = L;
                            }
                        }
                        while (__any_sync(KC_FULL_MASK, claims != 0)) {
                            uint32_t v = 0;
#pragma unroll
                            for (int k = U - 1; k >= 0; k--)
                                if ((claims >> k) & 1u) v = u[k];
                            enqueue(claims != 0, v, r + 1, fb_next);
                            claims &= claims - 1;
                        }
                    }
                };
                const unsigned per = min(32u, (total_items + nwarps - 1) / nwarps);
                if (per == 1) {
                    if ((tid >> 5) < total_items) {
                        const unsigned i = tid >> 5;
                        const unsigned long long it = i < q_cap ? slot[i] : __ldcg(&F[fb + i]);
                        const unsigned len = (unsigned)(it & 0xffffffull);
                        if (len <= 32) walk(std::integral_constant<int, 1>{}, std::true_type{}, (Off)(it >> 24), 0u, len);
                        else walk(std::integral_constant<int, 4>{}, std::true_type{}, (Off)(it >> 24), 0u, len);
                    }
                } else {
                    for (;;) {
                        unsigned i0 = 0;
                        if (lane == 0) i0 = atomicAdd(&head[r % 3], per);
                        i0 = __shfl_sync(KC_FULL_MASK, i0, 0);
                        if (i0 >= total_items) break;
                        Off rs = 0;
                        uint32_t len = 0;
                        const unsigned i = i0 + lane;
                        if (lane < per && i < total_items) {
                            const unsigned long long it = i < q_cap ? slot[i] : __ldcg(&F[fb + i]);
                            rs = (Off)(it >> 24);
                            len = (uint32_t)(it & 0xffffffull);
                        }
                        unsigned total;
                        const unsigned off = warp_excl_scan(len, lane, total);
                        rs -= (Off)off;  // entry e of the sequence is at rs + e of its owner
                        const unsigned start = len && lane ? off : 0x80000000u;  // items have at least one entry
                        walk(std::integral_constant<int, BATCH_U>{}, std::false_type{}, rs, start, total);
                    }
                }
                __syncthreads();
                fb = fb_next;
                r++;
            }
            // (old degrees of vertices claimed meanwhile have the top bit set, or are at most L)
            if (L + 2 < MARK && above < MARK - (L + 2)) my_min = min(my_min, above + L + 1);
            my_min = __reduce_min_sync(KC_FULL_MASK, my_min);
            if (lane == 0 && my_min != NO_LVL) atomicMin(&minlev[lev & 1], my_min);
            __syncthreads();
            L = minlev[lev & 1];
        }
        if (A.gtrace && tid == 0) A.gtrace[3ull * gi + 1] = global_ns();
    }
}

// The plan's view of a packed graph, three passes.  They share the work by
// entries and vertices, not by graphs: a warp per graph took 6.7 ms on one
// graph of 4.2 M entries, the passes below 0.03 ms.
constexpr uint32_t PLAN_TILE = 4096;

// Entry offset of each graph's first row (ebase[G] = entries in all), and the
// start of its part of the row-chunk queue: graph i's queue holds at most
// n_i + nnz_i / BATCH_MIN_CHUNK items.
__global__ void batch_bases(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ vbase, uint32_t G,
                            unsigned long long *ebase, unsigned long long *fbase, uint32_t *maxdeg) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i <= G; i += gridDim.x * blockDim.x) {
        const unsigned long long e = (unsigned long long)rowptr[vbase[i]];
        ebase[i] = e;
        if (i < G) {
            fbase[i] = (unsigned long long)vbase[i] + e / BATCH_MIN_CHUNK + i;
            maxdeg[i] = 0;
        }
    }
}

// The last i < G with base[i] <= x (base ascending, base[0] <= x): the graph of
// vertex or entry x, the last of those that start there.
template <typename T>
__device__ __forceinline__ uint32_t graph_of(const T *__restrict__ base, uint32_t G, uint64_t x) {
    uint32_t lo = 0, hi = G;
    while (hi - lo > 1) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if ((uint64_t)base[mid] <= x) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Largest degree of every graph: a tile of vertices per CTA, one atomic per
// warp and graph.
__global__ void batch_max_degrees(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ vbase, uint32_t G,
                                  uint32_t *maxdeg) {
    const uint64_t n = vbase[G];
    const unsigned lane = threadIdx.x & 31;
    for (uint64_t t0 = (uint64_t)blockIdx.x * PLAN_TILE; t0 < n; t0 += (uint64_t)gridDim.x * PLAN_TILE) {
        const uint64_t t1 = t0 + PLAN_TILE < n ? t0 + PLAN_TILE : n;
        for (uint64_t w = t0 + (threadIdx.x & ~31u); w < t1; w += blockDim.x) {
            const uint64_t v = w + lane;
            const uint32_t d = v < t1 ? (uint32_t)(rowptr[v + 1] - rowptr[v]) : 0u;
            const uint32_t i = graph_of(vbase, G, v < t1 ? v : w);
            const unsigned peers = __match_any_sync(KC_FULL_MASK, i);
            const uint32_t mx = __reduce_max_sync(peers, d);
            if ((int)lane == __ffs(peers) - 1) atomicMax(&maxdeg[i], mx);
        }
    }
}

// Rows of graph i may only reference vertices of graph i: a tile of entries
// per CTA, graph by graph within the tile.
__global__ void batch_check(const uint32_t *__restrict__ col, const uint32_t *__restrict__ vbase,
                            const unsigned long long *__restrict__ ebase, uint32_t G, unsigned long long *bad) {
    const uint64_t nnz = ebase[G];
    unsigned long long b = 0;
    for (uint64_t t0 = (uint64_t)blockIdx.x * PLAN_TILE; t0 < nnz; t0 += (uint64_t)gridDim.x * PLAN_TILE) {
        const uint64_t t1 = t0 + PLAN_TILE < nnz ? t0 + PLAN_TILE : nnz;
        for (uint32_t i = graph_of(ebase, G, t0); i < G && ebase[i] < t1; i++) {
            const uint64_t lo = ebase[i] > t0 ? ebase[i] : t0, hi = ebase[i + 1] < t1 ? ebase[i + 1] : t1;
            const uint32_t v0 = vbase[i], n = vbase[i + 1] - v0;
            for (uint64_t e = lo + threadIdx.x; e < hi; e += blockDim.x) b += col[e] - v0 >= n;
        }
    }
    b = __reduce_add_sync(KC_FULL_MASK, (unsigned)b);
    if ((threadIdx.x & 31) == 0 && b) atomicAdd(bad, b);
}

struct BatchConfig {
    uint32_t small_n = 12288;   // graphs up to this many vertices: small-CTA class
    int small_threads = 256;
    int large_threads = 1024;
    uint32_t chunk = 256;
    int large_shared = 1;  // 0: graphs above small_n keep their degrees in global memory (more CTAs per SM)
};

// Graphs of one size class run with the same kernel and launch shape.
enum : int { BATCH_U16 = 0, BATCH_U32 = 1, BATCH_GLOBAL = 2, BATCH_WIDE = 3 };
constexpr int BATCH_CLASSES = 7;
struct BatchClass {
    int kind = BATCH_U16;  // degree type and place
    int index = 0;         // work counter of the class
    std::vector<uint32_t> order;
    uint32_t smem_n = 0;
    unsigned q_cap = 0, id_cap = 32;
    uint32_t *d_order = nullptr;
    int threads = 256;
    int grid = 0;
    size_t smem_bytes = 0;
};

// Shared memory of the degrees and claim bits of n vertices (n a multiple of
// 32), and of the queues.
static size_t batch_graph_bytes(uint32_t n, size_t degsz) { return n * degsz + ((n / 8 + 15) & ~size_t(15)); }
static size_t batch_queue_bytes(unsigned q_cap, unsigned id_cap) { return 16ull * q_cap + 4ull * id_cap; }

}  // namespace kc

struct kc_batch {
    kc_graph *g = nullptr;
    uint32_t G = 0;
    std::vector<uint32_t> vbase, maxdeg;
    std::vector<uint64_t> nnz;
    uint32_t *d_vbase = nullptr;
    unsigned long long *d_fbase = nullptr;
    unsigned long long *d_F = nullptr;
    uint64_t F_cap = 0;
    unsigned int *d_next = nullptr;  // one counter per class
    uint32_t *d_gdeg = nullptr;
    uint8_t *d_gclaimed = nullptr;
    kc::BatchConfig cfg;
    std::vector<kc::BatchClass> classes;
    bool planned = false;
    bool use_graph = true;
    bool trace = false;
    unsigned long long *d_gtrace = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaStream_t exec_stream = nullptr;
    cudaStream_t side[kc::BATCH_CLASSES - 1] = {};
    cudaEvent_t fork = nullptr, join[kc::BATCH_CLASSES - 1] = {};
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    double last_ms = 0;
    ~kc_batch();
};

namespace kc {

static void free_classes(kc_batch *b) {
    for (auto &c : b->classes) dfree(c.d_order);
    b->classes.clear();
    if (b->exec) {
        cudaGraphExecDestroy(b->exec);
        b->exec = nullptr;
    }
    b->planned = false;
}

// Raises the dynamic shared-memory limit of batch_peel<DegT, SMEM, WIDE> on the
// current device to the opt-in maximum, once per device.  The limit is never
// lowered afterwards, so a launch planned for one size stays valid whatever
// other launches of the same kernel (a later plan, the allocation-free entry
// point, another host thread) need.
template <typename DegT, bool SMEM, bool WIDE = false>
static int batch_smem_limit() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    KC_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(KC_ERR_INVALID, "device %d out of range", dev);
    std::lock_guard<std::mutex> lk(mu);
    if (done[dev]) return KC_OK;
    auto fn = batch_peel<DegT, SMEM, WIDE>;
    int optin = 0;
    KC_CUDA(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    cudaFuncAttributes fa;
    KC_CUDA(cudaFuncGetAttributes(&fa, fn));
    KC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)fa.sharedSizeBytes));
    done[dev] = true;
    return KC_OK;
}

template <typename DegT, bool SMEM, bool WIDE = false>
static int class_grid(int threads, size_t smem, int sms, int *grid) {
    auto fn = batch_peel<DegT, SMEM, WIDE>;
    // whatever the size: 48 KB without the opt-in count the static variables too
    KC_TRY((batch_smem_limit<DegT, SMEM, WIDE>()));
    int occ = 0;
    KC_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, threads, smem));
    if (occ < 1) return fail(KC_ERR_UNSUPPORTED, "batch kernel (%d threads, %zu B shared) cannot be resident", threads, smem);
    *grid = occ * sms;
    return KC_OK;
}

// Size classes: graphs of at most small_n vertices; then, while the degrees
// fit 15 bits, graphs of which four, two or one fit the shared memory of an SM
// (large_threads / 4, / 2 and / 1 threads each: at 64 registers a thread an SM
// holds 1,024 threads, and the barriers of several CTAs overlap where one CTA
// of all the threads would wait); 32-bit degrees; 16-bit ones without the mark
// for what is too large for those (more than about 53,000 vertices) and has a hub
// of 32,768 to 65,534 entries; global memory.  304 graphs of 100,000 vertices,
// average degree 1 / 4 / 16, with a hub of 40,000 entries: 1.90 / 3.57 / 5.78 ms in
// global memory, 1.40 / 2.32 / 3.13 with wide degrees.
static int plan(kc_batch *b) {
    free_classes(b);
    int dev = b->g->device, smem_max = 0, smem_sm = 0;
    cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    const size_t budget = (size_t)smem_max - 1024;  // static shared variables and alignment
    const size_t qmin = batch_queue_bytes(0, 32);
    auto fits = [&](size_t bytes, size_t degsz) {
        uint32_t n = 0;
        while (batch_graph_bytes(n + 1024, degsz) + qmin <= bytes) n += 1024;
        return n;
    };
    const uint32_t large_u16 = fits(budget, 2), large_u32 = fits(budget, 4);
    const uint32_t small_n = std::min(b->cfg.small_n, large_u16);
    // per CTA of q on an SM: its share less the 1 KB that the SM reserves for
    // each CTA, the static variables and 8 bytes of queues per thread
    auto share = [&](int q) { return (size_t)smem_sm / q - 1280 - batch_queue_bytes(b->cfg.large_threads / q / 2, b->cfg.large_threads / q); };
    const uint32_t mid_n[2] = {fits(share(4), 2), fits(share(2), 2)};
    BatchClass cls[BATCH_CLASSES];
    for (int k = 0; k < BATCH_CLASSES; k++) cls[k].index = k;
    for (uint32_t i = 0; i < b->G; i++) {
        const uint32_t n = b->vbase[i + 1] - b->vbase[i];
        const bool fits16 = b->maxdeg[i] < 32768u;  // the top bit is the scan's mark
        const bool fits_wide = b->maxdeg[i] < 65535u;
        int k;
        if (b->nnz[i] >= (1ull << 31)) k = 6;  // 32-bit entry offsets in the shared-memory kernels
        else if (fits16 && n <= small_n) k = 0;
        else if (!b->cfg.large_shared) k = 6;
        else if (fits16 && n <= mid_n[0]) k = 1;
        else if (fits16 && n <= mid_n[1]) k = 2;
        else if (fits16 && n <= large_u16) k = 3;
        else if (n <= large_u32) k = 4;
        else if (fits_wide && n <= large_u16) k = 5;
        else k = 6;
        cls[k].order.push_back(i);
    }
    for (int k = 0; k < BATCH_CLASSES; k++) {
        BatchClass &c = cls[k];
        if (c.order.empty()) continue;
        c.kind = k <= 3 ? BATCH_U16 : k == 4 ? BATCH_U32 : k == 5 ? BATCH_WIDE : BATCH_GLOBAL;
        std::stable_sort(c.order.begin(), c.order.end(),
                         [&](uint32_t x, uint32_t y) { return b->nnz[x] > b->nnz[y]; });
        // shrink the shared arrays to the largest graph of the class
        uint32_t nmax = 0;
        for (uint32_t i : c.order) nmax = std::max(nmax, b->vbase[i + 1] - b->vbase[i]);
        c.smem_n = c.kind == BATCH_GLOBAL ? 0u : std::max<uint32_t>(32, (nmax + 31) & ~31u);
        c.threads = k == 0 ? b->cfg.small_threads : b->cfg.large_threads;
        if (k == 1 || k == 2) c.threads = std::max(64, c.threads / (k == 1 ? 4 : 2) & ~31);
        const size_t own = batch_graph_bytes(c.smem_n, c.kind == BATCH_U16 || c.kind == BATCH_WIDE ? 2 : 4);
        c.id_cap = (unsigned)c.threads;
        c.q_cap = (unsigned)c.threads / 2;
        while (own + batch_queue_bytes(c.q_cap, c.id_cap) > budget && c.q_cap) c.q_cap /= 2;
        if (own + batch_queue_bytes(c.q_cap, c.id_cap) > budget) c.id_cap = 32;
        c.smem_bytes = own + batch_queue_bytes(c.q_cap, c.id_cap);
        int grid = 0;
        int rc;
        if (c.kind == BATCH_U16) rc = class_grid<uint16_t, true>(c.threads, c.smem_bytes, b->g->sm_count, &grid);
        else if (c.kind == BATCH_U32) rc = class_grid<uint32_t, true>(c.threads, c.smem_bytes, b->g->sm_count, &grid);
        else if (c.kind == BATCH_WIDE) rc = class_grid<uint16_t, true, true>(c.threads, c.smem_bytes, b->g->sm_count, &grid);
        else rc = class_grid<uint32_t, false>(c.threads, c.smem_bytes, b->g->sm_count, &grid);
        if (rc) return rc;
        c.grid = (int)std::min<size_t>((size_t)grid, c.order.size());
        KC_TRY(dalloc(&c.d_order, c.order.size(), "batch class order"));
        if (c.kind == BATCH_GLOBAL && !b->d_gdeg) {
            // every graph's part starts at a multiple of 8 vertices
            KC_TRY(dalloc(&b->d_gdeg, (uint64_t)b->g->n + 8ull * b->G + 8, "batch global degrees"));
            KC_TRY(dalloc(&b->d_gclaimed, (uint64_t)b->g->n + 8ull * b->G + 8, "batch global flags"));
        }
        b->classes.push_back(std::move(c));
    }
    for (BatchClass &c : b->classes)
        KC_CUDA(cudaMemcpyAsync(c.d_order, c.order.data(), c.order.size() * 4, cudaMemcpyHostToDevice, b->g->stream));
    // The launches may be on any stream, and a plain cudaMemcpy of a few bytes
    // returns before they are on the device: behind other threads' uploads they
    // arrive after a kernel on a non-blocking stream has started.
    KC_CUDA(cudaStreamSynchronize(b->g->stream));
    b->planned = true;
    return KC_OK;
}

static int launch_all(kc_batch *b, cudaStream_t s) {
    Graph *g = b->g;
    const int nc = (int)b->classes.size();
    KC_CUDA(cudaMemsetAsync(b->d_next, 0, BATCH_CLASSES * 4, s));
    KC_CUDA(cudaEventRecord(b->fork, s));
    for (int k = 0; k < nc; k++) {
        // the class of largest graphs first: its CTAs take the SMs before the
        // many small-graph CTAs fill them
        BatchClass &c = b->classes[nc - 1 - k];
        cudaStream_t cs = k == 0 ? s : b->side[k - 1];
        if (k > 0) KC_CUDA(cudaStreamWaitEvent(cs, b->fork, 0));
        BatchArgs A;
        A.rowptr = g->rowptr;
        A.col = g->col;
        A.core = g->core;
        A.vbase = b->d_vbase;
        A.order = c.d_order;
        A.count = (uint32_t)c.order.size();
        A.F = b->d_F;
        A.fbase = b->d_fbase;
        A.next = b->d_next + c.index;
        A.gdeg = b->d_gdeg;
        A.gclaimed = b->d_gclaimed;
        A.chunk = b->cfg.chunk;
        A.smem_n = c.smem_n;
        A.gtrace = b->trace ? b->d_gtrace : nullptr;
        A.q_cap = c.q_cap;
        A.id_cap = c.id_cap;
        if (c.kind == BATCH_U16) batch_peel<uint16_t, true><<<c.grid, c.threads, c.smem_bytes, cs>>>(A);
        else if (c.kind == BATCH_U32) batch_peel<uint32_t, true><<<c.grid, c.threads, c.smem_bytes, cs>>>(A);
        else if (c.kind == BATCH_WIDE) batch_peel<uint16_t, true, true><<<c.grid, c.threads, c.smem_bytes, cs>>>(A);
        else batch_peel<uint32_t, false><<<c.grid, c.threads, c.smem_bytes, cs>>>(A);
        KC_CUDA(cudaGetLastError());
        if (k > 0) {
            KC_CUDA(cudaEventRecord(b->join[k - 1], cs));
            KC_CUDA(cudaStreamWaitEvent(s, b->join[k - 1], 0));
        }
    }
    return KC_OK;
}

static int run_batch(kc_batch *b, cudaStream_t s) {
    if (!b->planned) KC_TRY(plan(b));
    if (b->use_graph) {
        if (!b->exec || b->exec_stream != s) {
            if (b->exec) {
                cudaGraphExecDestroy(b->exec);
                b->exec = nullptr;
            }
            cudaGraph_t graph = nullptr;
            KC_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
            int rc = launch_all(b, s);
            cudaError_t e = cudaStreamEndCapture(s, &graph);
            if (rc) {
                if (graph) cudaGraphDestroy(graph);
                return rc;
            }
            if (e != cudaSuccess) return fail(KC_ERR_CUDA, "batch capture: %s", cudaGetErrorString(e));
            e = cudaGraphInstantiate(&b->exec, graph, 0);
            cudaGraphDestroy(graph);
            if (e != cudaSuccess) return fail(KC_ERR_CUDA, "batch graph instantiate: %s", cudaGetErrorString(e));
            b->exec_stream = s;
        }
        KC_CUDA(cudaGraphLaunch(b->exec, s));
        return KC_OK;
    }
    return launch_all(b, s);
}

}  // namespace kc

kc_batch::~kc_batch() {
    int cur = 0;
    cudaGetDevice(&cur);
    if (g) cudaSetDevice(g->device);
    kc::free_classes(this);
    kc::dfree(d_vbase);
    kc::dfree(d_fbase);
    kc::dfree(d_F);
    kc::dfree(d_next);
    kc::dfree(d_gdeg);
    kc::dfree(d_gclaimed);
    kc::dfree(d_gtrace);
    for (int i = 0; i < kc::BATCH_CLASSES - 1; i++) {
        if (side[i]) {
            cudaStreamSynchronize(side[i]);
            kc::release_stream(g ? g->device : 0, side[i]);
        }
        kc::release_event(join[i]);
    }
    kc::release_event(fork);
    kc::release_event(ev0);
    kc::release_event(ev1);
    cudaSetDevice(cur);
}

using namespace kc;

extern "C" {

int kc_batch_create(kc_graph *g, const uint32_t *vbase, uint32_t num_graphs, kc_batch **out) {
    clear_error();
    if (!g || !vbase || !out || num_graphs == 0) return fail(KC_ERR_INVALID, "null argument or empty batch");
    *out = nullptr;
    if (vbase[0] != 0 || vbase[num_graphs] != g->n) return fail(KC_ERR_INVALID, "vbase must start at 0 and end at n");
    for (uint32_t i = 0; i < num_graphs; i++)
        if (vbase[i + 1] < vbase[i]) return fail(KC_ERR_INVALID, "vbase must be non-decreasing");
    KC_CUDA(cudaSetDevice(g->device));
    kc_batch *b = new (std::nothrow) kc_batch();
    if (!b) return fail(KC_ERR_NOMEM, "batch handle");
    b->g = g;
    b->G = num_graphs;
    b->vbase.assign(vbase, vbase + num_graphs + 1);
    int rc = dalloc(&b->d_vbase, num_graphs + 1, "batch vbase");
    if (!rc) rc = dalloc(&b->d_fbase, num_graphs, "batch queue offsets");
    if (!rc) rc = dalloc(&b->d_next, BATCH_CLASSES, "batch counters");
    // entry bases, bad-entry count and largest degrees, read back in one copy
    const uint64_t words = (uint64_t)num_graphs + 2;
    const uint64_t bytes = 8 * words + 4ull * num_graphs;
    unsigned long long *d_plan = nullptr;
    if (!rc) rc = dalloc(&d_plan, words + (num_graphs + 1) / 2, "batch plan");
    if (!rc && !g->core) rc = dalloc(&g->core, (uint64_t)g->n + 1, "core");
    if (rc) {
        dfree(d_plan);
        delete b;
        return rc;
    }
    unsigned long long *d_bad = d_plan + num_graphs + 1;
    uint32_t *d_maxdeg = reinterpret_cast<uint32_t *>(d_plan + words);
    cudaStream_t s = g->stream;
    auto tiles = [&](uint64_t items) {
        return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((items + PLAN_TILE - 1) / PLAN_TILE, (uint64_t)g->sm_count * 16));
    };
    cudaMemcpyAsync(b->d_vbase, vbase, (num_graphs + 1) * 4ull, cudaMemcpyHostToDevice, s);
    cudaMemsetAsync(d_bad, 0, 8, s);
    batch_bases<<<tiles((uint64_t)num_graphs * 16), 256, 0, s>>>(g->rowptr, b->d_vbase, num_graphs, d_plan, b->d_fbase, d_maxdeg);
    batch_max_degrees<<<tiles(g->n), 256, 0, s>>>(g->rowptr, b->d_vbase, num_graphs, d_maxdeg);
    if (g->nnz) batch_check<<<tiles(g->nnz), 256, 0, s>>>(g->col, b->d_vbase, d_plan, num_graphs, d_bad);
    std::vector<unsigned char> host(bytes);
    cudaMemcpyAsync(host.data(), d_plan, bytes, cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    dfree(d_plan);
    if (e != cudaSuccess) {
        delete b;
        return fail(KC_ERR_CUDA, "batch setup: %s", cudaGetErrorString(e));
    }
    std::vector<unsigned long long> ebase(words);
    memcpy(ebase.data(), host.data(), 8 * words);
    b->maxdeg.resize(num_graphs);
    memcpy(b->maxdeg.data(), host.data() + 8 * words, 4ull * num_graphs);
    if (const unsigned long long bad = ebase[num_graphs + 1]) {
        delete b;
        return fail(KC_ERR_INVALID, "%llu entries reference a vertex outside their graph", bad);
    }
    b->nnz.resize(num_graphs);
    for (uint32_t i = 0; i < num_graphs; i++) b->nnz[i] = ebase[i + 1] - ebase[i];
    b->F_cap = (uint64_t)g->n + g->nnz / BATCH_MIN_CHUNK + num_graphs + 1;
    rc = dalloc(&b->d_F, b->F_cap, "batch row-chunk queue");
    if (!rc) {
        for (int i = 0; i < BATCH_CLASSES - 1 && !rc; i++) {
            if (acquire_stream(g->device, &b->side[i]) != cudaSuccess ||
                acquire_event(&b->join[i]) != cudaSuccess)
                rc = fail(KC_ERR_CUDA, "batch streams");
        }
        if (!rc && (acquire_event(&b->fork) != cudaSuccess || acquire_event(&b->ev0) != cudaSuccess ||
                    acquire_event(&b->ev1) != cudaSuccess))
            rc = fail(KC_ERR_CUDA, "batch events");
    }
    if (rc) {
        delete b;
        return rc;
    }
    *out = b;
    return KC_OK;
}

int kc_batch_set_param(kc_batch *b, const char *name, int64_t value) {
    clear_error();
    if (!b || !name) return fail(KC_ERR_INVALID, "null argument");
    std::string k(name);
    if (k == "batch.small_n") {
        if (value < 32 || value > (1 << 20)) return fail(KC_ERR_INVALID, "batch.small_n: [32, 2^20]");
        b->cfg.small_n = (uint32_t)value;
    } else if (k == "batch.small_threads" || k == "batch.large_threads") {
        if (value < 64 || value > 1024 || (value & 31)) return fail(KC_ERR_INVALID, "%s: multiple of 32 in [64, 1024]", name);
        (k == "batch.small_threads" ? b->cfg.small_threads : b->cfg.large_threads) = (int)value;
    } else if (k == "batch.chunk") {
        if (value < BATCH_MIN_CHUNK || value > (1 << 16) || (value & (value - 1)))
            return fail(KC_ERR_INVALID, "batch.chunk: power of two in [%u, 2^16]", BATCH_MIN_CHUNK);
        b->cfg.chunk = (uint32_t)value;
    } else if (k == "batch.large_shared") {
        b->cfg.large_shared = value ? 1 : 0;
    } else if (k == "batch.cuda_graph") {
        b->use_graph = value != 0;
        return KC_OK;
    } else if (k == "trace") {
        b->trace = value != 0;
        if (b->trace && !b->d_gtrace) KC_TRY(dalloc(&b->d_gtrace, 3ull * b->G, "batch trace"));
        if (b->exec) {
            cudaGraphExecDestroy(b->exec);
            b->exec = nullptr;
        }
        return KC_OK;
    } else {
        return fail(KC_ERR_INVALID, "unknown parameter %s", name);
    }
    KC_CUDA(cudaSetDevice(b->g->device));
    free_classes(b);
    return KC_OK;
}

int kc_batch_get_param(const kc_batch *b, const char *name, int64_t *value) {
    clear_error();
    if (!b || !name || !value) return fail(KC_ERR_INVALID, "null argument");
    std::string k(name);
    if (k == "batch.small_n") *value = b->cfg.small_n;
    else if (k == "batch.small_threads") *value = b->cfg.small_threads;
    else if (k == "batch.large_threads") *value = b->cfg.large_threads;
    else if (k == "batch.chunk") *value = b->cfg.chunk;
    else if (k == "batch.large_shared") *value = b->cfg.large_shared;
    else if (k == "batch.cuda_graph") *value = b->use_graph ? 1 : 0;
    else return fail(KC_ERR_INVALID, "unknown parameter %s", name);
    return KC_OK;
}

int kc_batch_decompose(kc_batch *b, uint32_t *core_out, int out_on_device, kc_stats *stats, void *stream) {
    clear_error();
    NvtxRange nvtx_("kc_batch_decompose");
    if (!b) return fail(KC_ERR_INVALID, "null batch");
    Graph *g = b->g;
    KC_CUDA(cudaSetDevice(g->device));
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : g->stream;
    KC_CUDA(cudaEventRecord(b->ev0, s));
    if (int rc = run_batch(b, s)) {
        cudaStreamSynchronize(s);  // nothing launched may outlive a failed call
        return rc;
    }
    KC_CUDA(cudaEventRecord(b->ev1, s));
    if (core_out && g->n)
        KC_CUDA(cudaMemcpyAsync(core_out, g->core, (uint64_t)g->n * 4,
                                out_on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, s));
    KC_CUDA(cudaStreamSynchronize(s));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, b->ev0, b->ev1);
    b->last_ms = ms;
    g->core_valid = true;
    if (stats) {
        memset(stats, 0, sizeof(*stats));
        stats->method = KC_PEELONE_DYN;
        stats->n = g->n;
        stats->nnz = g->nnz;
        stats->ms = ms;
        stats->build_ms = g->build_ms;
    }
    return KC_OK;
}

int kc_batch_autotune(kc_batch *b, double *best_ms) {
    clear_error();
    NvtxRange nvtx_("kc_batch_autotune");
    if (!b) return fail(KC_ERR_INVALID, "null batch");
    KC_CUDA(cudaSetDevice(b->g->device));
    const BatchConfig keep = b->cfg;
    BatchConfig best = keep;
    double best_t = 1e30;
    const uint32_t small_ns[] = {2048, 6144, 12288, 24576};
    const int small_threads[] = {128, 256, 512};
    const uint32_t chunks[] = {128, 256, 1024};
    for (uint32_t sn : small_ns)
        for (int st : small_threads)
            for (uint32_t ch : chunks) {
                b->cfg = keep;
                b->cfg.small_n = sn;
                b->cfg.small_threads = st;
                b->cfg.chunk = ch;
                free_classes(b);
                double t = 1e30;
                for (int rep = 0; rep < 2; rep++) {
                    int rc = kc_batch_decompose(b, nullptr, 0, nullptr, nullptr);
                    if (rc) {
                        b->cfg = keep;
                        free_classes(b);
                        return rc;
                    }
                    t = std::min(t, b->last_ms);
                }
                if (t < best_t) {
                    best_t = t;
                    best = b->cfg;
                }
            }
    b->cfg = best;
    free_classes(b);
    if (best_ms) *best_ms = best_t;
    return KC_OK;
}

int kc_batch_trace(const kc_batch *b, uint64_t *out, uint32_t cap) {
    clear_error();
    if (!b || !out) return fail(KC_ERR_INVALID, "null argument");
    if (!b->d_gtrace) return fail(KC_ERR_STATE, "batch trace not enabled");
    KC_CUDA(cudaSetDevice(b->g->device));
    KC_CUDA(cudaMemcpy(out, b->d_gtrace, 8ull * std::min<uint64_t>(cap, 3ull * b->G), cudaMemcpyDeviceToHost));
    return KC_OK;
}

int kc_batch_free(kc_batch *b) {
    clear_error();
    delete b;
    return KC_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Allocation-free decomposition of one small graph.
//
// For callers that cannot allocate device memory on this path: code running
// under a framework that owns all device memory through its own pool (so a
// cudaMalloc by this library would break its budget), latency-critical loops
// where cudaMalloc/cudaFree would synchronize the device, and code paths that
// must not create allocations at all.  The caller passes the graph and the
// output in device memory; the only scratch the batched kernel needs -- its
// row-chunk queue and a few control words -- lives in the fixed file-scope
// array below, which every GPU that loads this library holds until the
// process exits.  All calls share that array: calls whose work overlaps on
// the GPU (different streams, or different host threads) race on it and must
// be serialised by the caller.
namespace kc {

constexpr uint32_t NOALLOC_MAX_N = 50000;            // vertices
constexpr uint64_t NOALLOC_MAX_NNZ = 1ull << 22;     // directed CSR entries
constexpr uint64_t NOALLOC_CTRL_WORDS = 32;          // control block (256 bytes)
constexpr uint64_t NOALLOC_QUEUE = NOALLOC_MAX_N + NOALLOC_MAX_NNZ / BATCH_MIN_CHUNK + 2;
constexpr uint64_t NOALLOC_WORDS = NOALLOC_CTRL_WORDS + NOALLOC_QUEUE;  // 8-byte words, ~663 KB

static __device__ __align__(256) unsigned long long g_noalloc_scratch[NOALLOC_WORDS];

// Writes the one-graph work list into the control block: vbase = {0, n},
// order = {0}, fbase = {0}, work counter = 0, bad-entry count = 0.
__global__ void noalloc_prep(unsigned long long *scratch, uint32_t n) {
    uint32_t *w = reinterpret_cast<uint32_t *>(scratch);
    w[0] = 0;  // vbase[0]
    w[1] = n;  // vbase[1]
    w[2] = 0;  // order[0]
    w[4] = 0;  // next (work counter)
    scratch[3] = 0ull;  // fbase[0]
    w[8] = 0;  // entries that fail noalloc_check
}

// Counts, into control word 8, the row offsets that decrease (or a negative
// rowptr[0]) and the column ids >= n among col[0, nnz): the kernel indexes its
// shared-memory arrays by column id, so a caller's bad id must be turned into
// an error before it runs.
__global__ void noalloc_check(const int64_t *__restrict__ rowptr, const uint32_t *__restrict__ col, uint32_t n,
                              uint64_t nnz, unsigned long long *scratch) {
    unsigned bad = 0;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (uint64_t v = t0; v < n; v += stride) bad += (rowptr[v + 1] < rowptr[v]) ? 1u : 0u;
    if (t0 == 0 && rowptr[0] < 0) bad++;
    for (uint64_t e = t0; e < nnz; e += stride) bad += (col[e] >= n) ? 1u : 0u;
    bad = __reduce_add_sync(KC_FULL_MASK, bad);
    if ((threadIdx.x & 31) == 0 && bad) atomicAdd(reinterpret_cast<uint32_t *>(scratch) + 8, bad);
}

static std::mutex g_noalloc_mu;
static void *g_noalloc_ptr[64];

// Device address of the scratch array, looked up once per device with that
// device current (a host-side use of the symbol's name is not a device
// address).
static int noalloc_setup(int dev, unsigned long long **out) {
    if (dev < 0 || dev >= 64) return fail(KC_ERR_INVALID, "device %d out of range", dev);
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess || !p)
            return fail(KC_ERR_CUDA, "cudaGetSymbolAddress(no-alloc scratch): %s", cudaGetErrorString(e));
        KC_TRY((batch_smem_limit<uint32_t, true>()));
        g_noalloc_ptr[dev] = p;
    }
    *out = static_cast<unsigned long long *>(g_noalloc_ptr[dev]);
    return KC_OK;
}

}  // namespace kc

extern "C" int kc_decompose_noalloc(const int64_t *d_rowptr, const uint32_t *d_col, uint32_t n, uint32_t *d_core,
                                    void *stream) {
    using namespace kc;
    clear_error();
    if (!d_rowptr || !d_core) return fail(KC_ERR_INVALID, "null argument");
    if (n > NOALLOC_MAX_N)
        return fail(KC_ERR_CAPACITY, "kc_decompose_noalloc: %u vertices exceed the limit of %u", n, NOALLOC_MAX_N);
    int dev = 0;
    KC_CUDA(cudaGetDevice(&dev));
    unsigned long long *scratch = nullptr;
    KC_TRY(noalloc_setup(dev, &scratch));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int64_t nnz = 0;
    KC_CUDA(cudaMemcpyAsync(&nnz, d_rowptr + n, sizeof(nnz), cudaMemcpyDeviceToHost, s));
    KC_CUDA(cudaStreamSynchronize(s));
    if (nnz < 0 || (uint64_t)nnz > NOALLOC_MAX_NNZ)
        return fail(KC_ERR_CAPACITY, "kc_decompose_noalloc: %lld entries exceed the limit of %llu", (long long)nnz,
                    (unsigned long long)NOALLOC_MAX_NNZ);
    if (n == 0) return KC_OK;
    if (nnz > 0 && !d_col) return fail(KC_ERR_INVALID, "null column array with %lld entries", (long long)nnz);
    noalloc_prep<<<1, 1, 0, s>>>(scratch, n);
    {
        const uint64_t work = std::max<uint64_t>((uint64_t)nnz, n);
        const unsigned blocks = (unsigned)std::min<uint64_t>((work + 255) / 256, 1024);
        noalloc_check<<<blocks, 256, 0, s>>>(d_rowptr, d_col, n, (uint64_t)nnz, scratch);
        uint32_t bad = 0;
        KC_CUDA(cudaGetLastError());
        KC_CUDA(cudaMemcpyAsync(&bad, reinterpret_cast<uint32_t *>(scratch) + 8, sizeof(bad), cudaMemcpyDeviceToHost,
                                s));
        KC_CUDA(cudaStreamSynchronize(s));
        if (bad)
            return fail(KC_ERR_INVALID,
                        "kc_decompose_noalloc: %u row offsets or column ids invalid (ids must be < n = %u, "
                        "offsets non-decreasing from 0)", bad, n);
    }
    uint32_t *ctrl = reinterpret_cast<uint32_t *>(scratch);
    BatchArgs A;
    A.rowptr = d_rowptr;
    A.col = d_col;
    A.core = d_core;
    A.vbase = ctrl;
    A.order = ctrl + 2;
    A.count = 1;
    A.F = scratch + NOALLOC_CTRL_WORDS;
    A.fbase = scratch + 3;
    A.next = ctrl + 4;
    A.gdeg = nullptr;
    A.gclaimed = nullptr;
    A.chunk = 256;
    A.smem_n = (n + 31) & ~31u;
    A.gtrace = nullptr;
    A.q_cap = A.id_cap = 1024;  // 20 KB beside the 206 KB of 50,000 vertices
    const size_t smem = batch_graph_bytes(A.smem_n, sizeof(uint32_t)) + batch_queue_bytes(A.q_cap, A.id_cap);
    // the kernel's shared-memory limit was raised to the device maximum once,
    // in noalloc_setup, and is never lowered
    batch_peel<uint32_t, true><<<1, 1024, smem, s>>>(A);
    KC_CUDA(cudaGetLastError());
    KC_CUDA(cudaStreamSynchronize(s));
    return KC_OK;
}
