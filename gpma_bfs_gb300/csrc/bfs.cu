// bfs.cu - GPU-only BFS over the gapped PMA.
//
// Replaces gpma_bfs (gpma_bfs.cuh:511-533) and its gather/contract kernels
// (:150-395), whose level loop crossed host<->device every level
// (:479,495). Semantics are the reference's: the edges of node v are the
// slots [row_offset[v], row_offset[v+1]) whose low 32 bits are not
// 0xFFFFFFFF (row guards, empty slots) and whose value is non-zero
// (tombstones, bulk-rebuild gaps); levels[src] = 1 and a node first reached
// from level L gets L+1.
//
// Single source: one persistent cooperative kernel runs every level,
// separated by bounded grid barriers (a second one goes on after LONG_LEVELS
// levels). Node sets are bitmaps (no queue, no queue
// atomics): seen (every node reached, the only one that searching threads
// write), done (those that have their level) and front (the level's frontier).
// Per level,
//   the scan takes each warp's words of seen: what is not in done is the
//     frontier; its nodes get their level (a warp's stores are one line) and
//     the rows of a word's up to 32 nodes, taken as one concatenated slot
//     range, are queued in pieces of ITEM_SLOTS slots (LARGE_ITEM_SLOTS in
//     large arrays);
//   the walk, after a barrier, spreads the pieces over every warp (warp-level
//     load balancing, LANE_SLOTS slots per lane per step, all loads issued
//     before any claim). A target is claimed with one atomicOr on seen (a plain
//     load filters targets already there).
// The scan after a level that claims nothing finds no frontier and ends the
// search.
//
// Direction switch (off by default): with dense_div, a level whose frontier
// rows span >= size / dense_div slots sweeps the whole slot array once,
// coalesced, instead of the walk (a PMA of out-edges has no in-edges to pull
// from; the sweep reads each key's source row from its high word and tests it
// against the frontier bitmap). Both give the same levels.
//
#include "gpma_internal.cuh"

#include <algorithm>
#include <mutex>

namespace gpma {
namespace {

// bfs_ctl layout (u32 words). Zero before a launch; a launch that ends well
// leaves it zero again when it reports to the host itself (BfsArgs::host).
enum : uint32_t {
    CTL_CNT = 0,      // 3 rotating counters: frontier nodes per level
    CTL_ITEMS = 3,    // 3 rotating counters: items queued per level
    CTL_ERR = 6,
    CTL_LEVELS = 7,
    CTL_REACHED = 8,
    CTL_OVERFLOW = 9, // times a CTA or warp found the item list full and kept its items
    CTL_SLOTS = 12,   // 3 rotating counters: slots of the frontier's rows (dense_div only)
    CTL_DONE = 15,    // CTAs that have added their reached nodes
    CTL_WORDS = 16,   // what the host reads
    CTL_BAR = BAR_ALIGN_WORDS,  // GridBarrier
    CTL_ALL = CTL_BAR + BAR_WORDS,
    // profiling record after those: u64 start stamp of each level
    // (and of the final check), then u32 per level: frontier size | dense << 31
    CTL_PROFILE_LEVELS = 64,
    CTL_PROFILE_WORDS = 3 * CTL_PROFILE_LEVELS,
};
// CTL_ERR of the host's copy before the kernel has reported.
constexpr uint32_t HOST_PENDING = 0xFFFFFFFFu;

// A warp walks LANE_SLOTS slots per lane per step (build option), all loads of
// a step issued before any claim.
#ifndef GPMA_BFS_LANE_SLOTS
#define GPMA_BFS_LANE_SLOTS 4
#endif
constexpr uint32_t LANE_SLOTS = GPMA_BFS_LANE_SLOTS;
static_assert(LANE_SLOTS >= 1 && LANE_SLOTS <= 8, "BFS lane slots out of range");
constexpr uint32_t STEP_SLOTS = 32 * LANE_SLOTS;
// Slots of one work item: a step of a warp. A word's rows hold 20 slots per
// frontier node on average, up to hundreds of thousands with a hub; walked by
// the warp that owns the word (its long rows apart), warps spent 40 % of their
// time waiting at the level's barrier. Social graph, 2^25 slots: 350 us with items
// of one step, about 445 with four (a warp reads its next item's rows one item ahead).
// Arrays of LARGE_SLOTS slots and more have work for every warp at four steps an
// item, and each item costs the offsets of its word's 32 rows again (R-MAT, items of
// 1 / 2 / 4 / 8 steps: scale 21, 2^27 slots, 511 / 481 / 481 / 500 us; scale 24, 2^30
// slots, 3651 / 3316 / 3180 / 3091). Below, one step: scale 20, 2^26 slots, 308 and
// 308 with four, 2^25 slots 228 and 243. A build of its own, so that the smaller one
// keeps its single step.
constexpr uint32_t ITEM_SLOTS = STEP_SLOTS;
constexpr uint32_t LARGE_ITEM_SLOTS = 4 * STEP_SLOTS;
constexpr uint32_t LARGE_SLOTS = 1u << 27;
// Items of one level at most: the last piece of every word and whole pieces.
inline uint64_t bfs_item_need(uint32_t n, uint32_t size) {
    return n / 32 + 1 + size / (size >= LARGE_SLOTS ? LARGE_ITEM_SLOTS : ITEM_SLOTS);
}
// Items that a CTA collects in shared memory and adds to the grid's list under
// one atomic; a warp that finds no room adds its own. (An atomic per frontier
// word, all on one counter, serialises at 4.4 ns apiece.)
constexpr uint32_t CTA_ITEMS = 1024;

// bfs_long_kernel takes over at this level (counted from 0), which bfs_kernel has
// scanned and not walked; a level of it is short when the
// one before had at most SHORT_NODES nodes per CTA, and a CTA then walks its first
// SHORT_ITEMS items before the barrier.
constexpr uint32_t LONG_LEVELS = 64;
constexpr uint32_t SHORT_NODES = 4;
constexpr uint32_t SHORT_ITEMS = 2 * (BLOCK / 32);
constexpr int LONG_CTAS_PER_SM = 3;

struct BfsArgs {
    const uint64_t *keys;
    const uint8_t *vals;
    const uint32_t *ro;
    uint32_t n;
    uint32_t size;
    uint32_t src;
    uint32_t *levels;
    // bitmaps of n/32+2 words each; over: non-zero for words whose items no list took
    uint32_t *seen, *done, *front, *over;
    uint32_t *claimed[2];  // bfs_long_kernel: bitmaps of what short levels claim
    uint2 *items;      // {word, piece}
    uint32_t item_cap;
    uint32_t *ctl;
    uint32_t *host;      // page-locked words that receive the control words at the end, or null
    uint32_t dense_div;  // a level whose frontier rows span >= size / dense_div slots sweeps every slot (0: never)
    unsigned long long *stamps;  // per-level profile (CTL_PROFILE_LEVELS stamps + info words) or null
    const unsigned char *gate;   // status slot of the update before this search, or null: with host work or an
                                 // error reported there the search does not run (nothing is written)
    // test hooks: extra arrivals the first grid barrier waits for, and its limit
    uint32_t stall;
    uint64_t stall_limit_ns;
};

// N edge slots of one lane (SIZE_NONE: absent): every key, value and seen
// word is loaded before any claim, so each lane keeps several requests in
// flight. A target that was not seen when its word was read is claimed without
// waiting for a result (an old word costs an atomic that changes nothing).
template <uint32_t N>
__device__ __forceinline__ void visit_slots(const BfsArgs &A, const uint32_t (&sl)[N], uint32_t *claims) {
    uint32_t w[N], seen[N];
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) {
        uint64_t k = KEY_NONE;
        uint8_t v = 0;
        if (sl[j] != SIZE_NONE) {
            k = A.keys[sl[j]];
            v = A.vals[sl[j]];
        }
        w[j] = (uint32_t)k;
        seen[j] = (w[j] != 0xFFFFFFFFu && v != 0 && w[j] < A.n) ? 0u : 0xFFFFFFFFu;
    }
#pragma unroll
    for (uint32_t j = 0; j < N; ++j)
        if (!seen[j])
            seen[j] = A.seen[w[j] >> 5];
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) {
        const uint32_t bit = 1u << (w[j] & 31);
        if (!(seen[j] & bit))
            atomicOr(&claims[w[j] >> 5], bit);
    }
}

// Dense levels: 8 consecutive slots of the linear sweep. The key's high word
// is its source row, so the frontier test needs no row_offset lookup; guards,
// empty slots, tombstones and bulk-rebuild gaps fail the same tests as in the
// row walk (low word 0xFFFFFFFF or value 0; KEY_NONE's source is out of
// range). The frontier words of all 8, then their seen words, are loaded
// before any claim, so each thread keeps 8 requests in flight per stage.
__device__ __forceinline__ void dense_visit8(const BfsArgs &A, const uint64_t (&k)[8], uint2 v) {
    uint32_t dst[8], word[8];
    bool c[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint32_t src = (uint32_t)(k[j] >> 32);
        const uint32_t val = ((j < 4 ? v.x : v.y) >> (8 * (j & 3))) & 0xFFu;
        dst[j] = (uint32_t)k[j];
        c[j] = dst[j] != 0xFFFFFFFFu && val != 0 && src < A.n && dst[j] < A.n;
        word[j] = c[j] ? A.front[src >> 5] >> (src & 31) : 0u;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        c[j] = c[j] && (word[j] & 1u);
        word[j] = c[j] ? A.seen[dst[j] >> 5] : 0xFFFFFFFFu;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint32_t bit = 1u << (dst[j] & 31);
        if (c[j] && !(word[j] & bit))
            atomicOr(&A.seen[dst[j] >> 5], bit);
    }
}

// Slot of concatenated-range position p (< total) of a warp's rows: lane r holds
// its exclusive prefix excl and how far its row's start lies from it; finds the last
// r with excl[r] <= p. All lanes must call it together.
__device__ __forceinline__ uint32_t lb_slot(uint32_t p, uint32_t total, uint32_t start, uint32_t excl) {
    uint32_t r = 0;
#pragma unroll
    for (uint32_t step = 16; step >= 1; step >>= 1) {
        const uint32_t cand = r + step;
        const uint32_t ex_c = __shfl_sync(0xFFFFFFFFu, excl, cand & 31);
        if (cand < 32 && ex_c <= p)
            r = cand;
    }
    const uint32_t from = __shfl_sync(0xFFFFFFFFu, start, r);
    return p < total ? p + from : SIZE_NONE;
}

// One frontier word as a warp walks it: lane l's row of node 32 * word + l.
struct WordRows {
    uint32_t f = 0, b = 0, e = 0;  // the word's frontier bits; this lane's row, unclipped
    __device__ __forceinline__ void load(const BfsArgs &A, uint32_t word, uint32_t lane) {
        const uint32_t u = (word << 5) + lane;
        f = A.front[word];
        b = u < A.n ? A.ro[u] : 0u;
        e = u < A.n ? A.ro[u + 1] : 0u;
    }
};

// This lane's row length if its node is in `bits`.
__device__ __forceinline__ uint32_t row_slots(const BfsArgs &A, uint32_t bits, uint32_t lane, uint32_t b, uint32_t e) {
    if (!((bits >> lane) & 1u))
        return 0;
    if (!in_bounds(A.ctl + CTL_ERR, b <= e && e <= A.size, BS_ROW))
        return 0;  // an inconsistent row_offset: the row is skipped
    const uint32_t end = min(e, A.size);
    return end > b ? end - b : 0u;
}

// Walks slots [p0, p1) of a word's concatenated rows (p1: or their end).
__device__ __forceinline__ void walk_word(const BfsArgs &A, const WordRows &W, uint32_t p0, uint32_t p1,
                                          uint32_t lane, uint32_t *claims) {
    const uint32_t len = row_slots(A, W.f, lane, W.b, W.e);
    const uint32_t incl = warp_incl_scan(len);
    const uint32_t excl = incl - len;
    const uint32_t total = min(p1, __shfl_sync(0xFFFFFFFFu, incl, 31));
    for (; p0 < total; p0 += STEP_SLOTS) {  // once for an item of ITEM_SLOTS
        uint32_t sl[LANE_SLOTS];
#pragma unroll
        for (uint32_t j = 0; j < LANE_SLOTS; ++j)
            sl[j] = lb_slot(p0 + 32 * j + lane, total, W.b - excl, excl);
        visit_slots<LANE_SLOTS>(A, sl, claims);
    }
}

// The end of a search: the CTA's reached nodes (reached, in thread 0) are added, and
// the last CTA to come here hands the control words to the host.
__device__ __forceinline__ void report(const BfsArgs &A, uint32_t levels, uint32_t reached) {
    if (threadIdx.x != 0)
        return;
    if (reached)
        atomicAdd(A.ctl + CTL_REACHED, reached);
    if (blockIdx.x == 0)
        A.ctl[CTL_LEVELS] = levels;
    __threadfence();
    if (!A.host || atomicAdd(A.ctl + CTL_DONE, 1u) != gridDim.x - 1)
        return;
    __threadfence();
    for (uint32_t c = 0; c < CTL_WORDS; ++c) {
        A.host[c] = ld_volatile(A.ctl + c);
        A.ctl[c] = 0;
    }
    reinterpret_cast<GridBarrier *>(A.ctl + CTL_BAR)->count = 0;
}

// Social graph (1.6M nodes, 15.3M edges, 33.5M slots), a search of 18 levels: 350 us
// (374 with claims of three L2 operations, two bitmaps and the level). The walks of
// the middle levels (a key, a value and a seen word per slot; the largest moves about
// 230 MB) are 190 us of it, the rest the scans and two grid barriers per level. More
// slots per lane, fewer registers for more warps, slots read an item ahead and runs
// of 2 or 4 slots per lane all measured within 4 % of this or slower. The compiler's
// schedule of the walk hangs on little: with the limit of levels in the loop's head
// the same search takes 361 us, and one of 2^28 slots 909 in place of 823.
template <uint32_t ITEM>
__global__ void __launch_bounds__(BLOCK, 5) bfs_kernel(BfsArgs A) {
    __shared__ uint2 s_items[CTA_ITEMS];
    __shared__ uint32_t s_nit, s_end, s_at;  // items claimed and filled; place in the grid's list
    if (A.gate) {
        const DeviceStatus *h = reinterpret_cast<const DeviceStatus *>(A.gate);
        const GraphStatus *gs = reinterpret_cast<const GraphStatus *>(A.gate + STAT_GS_OFFSET);
        if (h->err | h->invalid_keys | h->significant | gs->remaining)
            return;
    }
    GridBarrier *bar = reinterpret_cast<GridBarrier *>(A.ctl + CTL_BAR);
    uint32_t *err = A.ctl + CTL_ERR;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t gwarp = blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * (BLOCK / 32);
    const uint32_t gtid = blockIdx.x * BLOCK + threadIdx.x, nthreads = gridDim.x * BLOCK;
    const uint32_t words = (A.n + 31) >> 5;
    for (uint32_t v = gtid; v < A.n; v += nthreads)
        A.levels[v] = 0;
    for (uint32_t w = gtid; w < words; w += nthreads) {
        A.seen[w] = w == A.src >> 5 ? 1u << (A.src & 31) : 0u;
        A.done[w] = 0;
        A.over[w] = 0;
    }
    if (!grid_barrier(bar, err, A.stall, A.stall_limit_ns))
        return;
    uint32_t reached = 0;
    uint32_t i = 0;
    for (;; ++i) {
        const bool stamper = A.stamps && gtid == 0 && i < CTL_PROFILE_LEVELS;
        if (stamper)
            A.stamps[i] = globaltimer_ns();
        if (threadIdx.x == 0) {
            s_nit = 0;
            s_end = CTA_ITEMS;
        }
        __syncthreads();
        // Scan: warp gwarp owns words gwarp, gwarp + nwarps, ... (hub rows
        // spread over the grid); it reads 32 of them at once, one per lane, and
        // a word's row offsets while the word before is queued.
        uint32_t *item_cnt = A.ctl + CTL_ITEMS + i % 3;
        uint32_t count = 0, slots = 0;
        for (uint32_t it = 0; gwarp + it * nwarps < words; it += 32) {
            const uint32_t w0 = gwarp + it * nwarps, wl = w0 + lane * nwarps;
            uint32_t mine = 0;
            if (wl < words) {
                const uint32_t s = A.seen[wl];
                mine = s & ~A.done[wl];
                A.front[wl] = mine;
                if (mine)
                    A.done[wl] = s;
            }
            count += __popc(mine);
            uint32_t pending = __ballot_sync(0xFFFFFFFFu, mine != 0u);
            uint32_t nb = 0, ne = 0;
            auto offsets = [&]() {
                const uint32_t u = ((w0 + (__ffs(pending) - 1) * nwarps) << 5) + lane;
                nb = u < A.n ? A.ro[u] : 0u;
                ne = u < A.n ? A.ro[u + 1] : 0u;
            };
            if (pending)
                offsets();
            while (pending) {
                const uint32_t at = __ffs(pending) - 1;
                pending &= pending - 1;
                const uint32_t word = w0 + at * nwarps;
                const uint32_t bits = __shfl_sync(0xFFFFFFFFu, mine, at);
                const uint32_t b = nb, e = ne;
                if (pending)
                    offsets();
                if ((bits >> lane) & 1u)
                    A.levels[(word << 5) + lane] = i + 1;
                const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, row_slots(A, bits, lane, b, e));
                slots += lane == 0 ? total : 0u;
                const uint32_t pieces = (total + ITEM - 1) / ITEM;
                uint32_t base = 0;
                if (lane == 0)
                    base = atomicAdd(&s_nit, pieces);
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                uint2 *list = s_items;
                if (base + pieces > CTA_ITEMS) {
                    // no room: to the grid's list, or, that being full too, left
                    // to this warp's walk
                    if (lane == 0) {
                        atomicMin(&s_end, base);  // every later warp finds no room either
                        base = atomicAdd(item_cnt, pieces);
                    }
                    base = __shfl_sync(0xFFFFFFFFu, base, 0);
                    list = A.items;
                    if (base + pieces > A.item_cap) {
                        for (uint32_t c = base + lane; c < min(base + pieces, A.item_cap); c += 32)
                            A.items[c] = make_uint2(0, SIZE_NONE);
                        if (lane == 0) {
                            A.over[word] = 1;
                            atomicAdd(A.ctl + CTL_OVERFLOW, 1u);
                        }
                        continue;
                    }
                }
                for (uint32_t c = lane; c < pieces; c += 32)
                    list[base + c] = make_uint2(word, c);
            }
        }
        reached += count;
        // the CTA's counts, and its items into the grid's list (or kept)
        {
            __shared__ uint32_t s_cnt[BLOCK / 32], s_slots[BLOCK / 32];
            count = __reduce_add_sync(0xFFFFFFFFu, count);
            slots = __reduce_add_sync(0xFFFFFFFFu, slots);
            if (lane == 0) {
                s_cnt[threadIdx.x >> 5] = count;
                s_slots[threadIdx.x >> 5] = slots;
            }
            __syncthreads();
            if (threadIdx.x == 0) {
                for (int w = 1; w < BLOCK / 32; ++w) {
                    count += s_cnt[w];
                    slots += s_slots[w];
                }
                if (count)
                    atomicAdd(A.ctl + CTL_CNT + i % 3, count);
                if (A.dense_div && slots)
                    atomicAdd(A.ctl + CTL_SLOTS + i % 3, slots);
                s_end = min(s_nit, s_end);
                s_at = s_end ? atomicAdd(item_cnt, s_end) : 0u;
            }
            __syncthreads();
        }
        uint32_t kept = s_end;  // items the CTA walks itself
        if (s_at + s_end <= A.item_cap) {
            kept = 0;
            for (uint32_t c = threadIdx.x; c < s_end; c += BLOCK)
                A.items[s_at + c] = s_items[c];
        } else {
            for (uint32_t c = s_at + threadIdx.x; c < min(s_at + s_end, A.item_cap); c += BLOCK)
                A.items[c] = make_uint2(0, SIZE_NONE);
            if (threadIdx.x == 0)
                atomicAdd(A.ctl + CTL_OVERFLOW, 1u);
        }
        if (!grid_barrier(bar, err))
            return;
        const uint32_t frontier = cta_broadcast_read(A.ctl + CTL_CNT + i % 3);
        if (frontier == 0 || i == LONG_LEVELS)  // done, or bfs_long_kernel's, whose nodes are in front
            break;
        if (gtid == 0) {
            A.ctl[CTL_CNT + (i + 1) % 3] = 0;
            A.ctl[CTL_SLOTS + (i + 1) % 3] = 0;
            A.ctl[CTL_ITEMS + (i + 1) % 3] = 0;
        }
        const bool dense =
            A.dense_div && (uint64_t)cta_broadcast_read(A.ctl + CTL_SLOTS + i % 3) * A.dense_div >= A.size;
        if (stamper)
            reinterpret_cast<uint32_t *>(A.stamps + CTL_PROFILE_LEVELS)[i] = frontier | (dense ? 1u << 31 : 0u);
        if (dense) {
            // every slot in one coalesced sweep, 8 slots per thread per step
            const ulonglong2 *kv = reinterpret_cast<const ulonglong2 *>(A.keys);
            const uint2 *vv = reinterpret_cast<const uint2 *>(A.vals);
            for (uint32_t o = gtid; o < (A.size >> 3); o += nthreads) {
                const ulonglong2 k0 = kv[4 * o], k1 = kv[4 * o + 1], k2 = kv[4 * o + 2], k3 = kv[4 * o + 3];
                const uint64_t k[8] = {k0.x, k0.y, k1.x, k1.y, k2.x, k2.y, k3.x, k3.y};
                dense_visit8(A, k, vv[o]);
            }
            // an array of 4 slots (the smallest size): one thread takes it, padded with empty slots
            if (A.size < 8 && gtid == 0) {
                const uint64_t k[8] = {A.keys[0], A.keys[1], A.keys[2], A.keys[3], KEY_NONE, KEY_NONE, KEY_NONE, KEY_NONE};
                const uint2 v = make_uint2(A.vals[0] | (A.vals[1] << 8) | (A.vals[2] << 16) | ((uint32_t)A.vals[3] << 24), 0u);
                dense_visit8(A, k, v);
            }
        } else {
            // Walk: an item is read two rounds ahead and its word's rows one
            // round ahead. A neutral item starts past any row (piece SIZE_NONE).
            const uint32_t nit = min(cta_broadcast_read(item_cnt), A.item_cap);
            auto item = [&](uint64_t c) { return c < nit ? A.items[c] : make_uint2(0, SIZE_NONE); };
            uint2 cur = item(gwarp), nxt = item((uint64_t)gwarp + nwarps);
            WordRows W;
            W.load(A, cur.x, lane);
            for (uint64_t c = gwarp; c < nit; c += nwarps) {
                const uint2 after = item(c + 2ull * nwarps);
                WordRows N;
                N.load(A, nxt.x, lane);
                if (cur.y != SIZE_NONE)
                    walk_word(A, W, cur.y * ITEM, (cur.y + 1) * ITEM, lane, A.seen);
                W = N;
                cur = nxt;
                nxt = after;
            }
            // what found no room in the list
            for (uint32_t c = threadIdx.x >> 5; c < kept; c += BLOCK / 32) {
                const uint2 own = s_items[c];
                W.load(A, own.x, lane);
                walk_word(A, W, own.y * ITEM, (own.y + 1) * ITEM, lane, A.seen);
            }
            if (cta_broadcast_read(A.ctl + CTL_OVERFLOW)) {
                for (uint32_t w = gwarp; w < words; w += nwarps) {
                    if (!A.over[w])
                        continue;
                    W.load(A, w, lane);
                    walk_word(A, W, 0, SIZE_NONE, lane, A.seen);
                    __syncwarp();
                    if (lane == 0)
                        A.over[w] = 0;
                }
            }
        }
        if (!grid_barrier(bar, err))
            return;
    }
    // reached nodes: every frontier's; the last CTA to add its own reports
    reached = __reduce_add_sync(0xFFFFFFFFu, reached);
    __syncthreads();
    if (threadIdx.x == 0)
        s_at = 0;
    __syncthreads();
    if (lane == 0 && reached)
        atomicAdd(&s_at, reached);
    __syncthreads();
    report(A, i, s_at);
}

// A search from the walk of level LONG_LEVELS on, over the maps that bfs_kernel left
// (that level's frontier is in front, and has its levels and counts): levels of
// few nodes end with one grid barrier instead of two (a 300 x 300 grid, 599 levels:
// 8.4 us per level with two, 5.5 with one). A short level claims nodes in a bitmap of
// the level's parity, which the next level's scan adds to seen, so that a CTA can
// walk its items while others still scan; items beyond SHORT_ITEMS go to the grid's
// list for a walk behind the barrier, and where no CTA has any the level is done.
// A kernel of its own, since bfs_kernel is up to 15 % slower on the social graph with
// any of this inside. (No dense levels here: they would be the same.) Three CTAs per
// SM: 72 registers without spills, and a cheaper barrier.
template <uint32_t ITEM>
__global__ void __launch_bounds__(BLOCK, LONG_CTAS_PER_SM) bfs_long_kernel(BfsArgs A) {
    __shared__ uint2 s_items[CTA_ITEMS];
    __shared__ uint32_t s_nit, s_end, s_at;  // as in bfs_kernel
    __shared__ uint32_t s_cnt[BLOCK / 32];
    GridBarrier *bar = reinterpret_cast<GridBarrier *>(A.ctl + CTL_BAR);
    uint32_t *err = A.ctl + CTL_ERR;
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t gwarp = blockIdx.x * (BLOCK / 32) + warp;
    const uint32_t nwarps = gridDim.x * (BLOCK / 32);
    const uint32_t gtid = blockIdx.x * BLOCK + threadIdx.x, nthreads = gridDim.x * BLOCK;
    const uint32_t words = (A.n + 31) >> 5;
    for (uint32_t w = gtid; w < words; w += nthreads) {
        A.claimed[0][w] = 0;
        A.claimed[1][w] = 0;
    }
    if (!grid_barrier_long(bar, err))
        return;
    uint32_t reached = 0, frontier = SIZE_NONE;  // nodes of all levels, of the last one
    bool brief = false;                          // the last level was a short one
    uint32_t i = LONG_LEVELS;
    for (;; ++i) {
        if (threadIdx.x == 0) {
            s_nit = 0;
            s_end = CTA_ITEMS;
        }
        __syncthreads();
        // scan, as in bfs_kernel
        uint32_t *item_cnt = A.ctl + CTL_ITEMS + i % 3;
        uint32_t count = 0;
        for (uint32_t it = 0; gwarp + it * nwarps < words; it += 32) {
            const uint32_t w0 = gwarp + it * nwarps, wl = w0 + lane * nwarps;
            uint32_t mine = 0;
            if (wl < words && i == LONG_LEVELS) {
                mine = A.front[wl];  // scanned and counted by bfs_kernel
            } else if (wl < words) {
                uint32_t s = A.seen[wl];
                if (brief) {
                    // what the short level before claimed; only this lane has the word
                    uint32_t *p = A.claimed[(i + 1) & 1] + wl;
                    const uint32_t c = *p;
                    if (c) {
                        *p = 0;
                        s |= c;
                        A.seen[wl] = s;
                    }
                }
                mine = s & ~A.done[wl];
                A.front[wl] = mine;
                if (mine)
                    A.done[wl] = s;
            }
            count += __popc(mine);
            uint32_t pending = __ballot_sync(0xFFFFFFFFu, mine != 0u);
            uint32_t nb = 0, ne = 0;
            auto offsets = [&]() {
                const uint32_t u = ((w0 + (__ffs(pending) - 1) * nwarps) << 5) + lane;
                nb = u < A.n ? A.ro[u] : 0u;
                ne = u < A.n ? A.ro[u + 1] : 0u;
            };
            if (pending)
                offsets();
            while (pending) {
                const uint32_t at = __ffs(pending) - 1;
                pending &= pending - 1;
                const uint32_t word = w0 + at * nwarps;
                const uint32_t bits = __shfl_sync(0xFFFFFFFFu, mine, at);
                const uint32_t b = nb, e = ne;
                if (pending)
                    offsets();
                if ((bits >> lane) & 1u)
                    A.levels[(word << 5) + lane] = i + 1;
                const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, row_slots(A, bits, lane, b, e));
                const uint32_t pieces = (total + ITEM - 1) / ITEM;
                uint32_t base = 0;
                if (lane == 0)
                    base = atomicAdd(&s_nit, pieces);
                base = __shfl_sync(0xFFFFFFFFu, base, 0);
                uint2 *list = s_items;
                if (base + pieces > CTA_ITEMS) {
                    // no room: to the grid's list, or, that being full too, left
                    // to this warp's walk
                    if (lane == 0) {
                        atomicMin(&s_end, base);  // every later warp finds no room either
                        base = atomicAdd(item_cnt, pieces);
                    }
                    base = __shfl_sync(0xFFFFFFFFu, base, 0);
                    list = A.items;
                    if (base + pieces > A.item_cap) {
                        for (uint32_t c = base + lane; c < min(base + pieces, A.item_cap); c += 32)
                            A.items[c] = make_uint2(0, SIZE_NONE);
                        if (lane == 0) {
                            A.over[word] = 1;
                            atomicAdd(A.ctl + CTL_OVERFLOW, 1u);
                        }
                        continue;
                    }
                }
                for (uint32_t c = lane; c < pieces; c += 32)
                    list[base + c] = make_uint2(word, c);
            }
        }
        brief = frontier <= SHORT_NODES * gridDim.x;
        uint32_t *claims = brief ? A.claimed[i & 1] : A.seen;
        count = __reduce_add_sync(0xFFFFFFFFu, count);
        if (lane == 0)
            s_cnt[warp] = count;
        __syncthreads();
        const uint32_t filled = min(s_nit, s_end), own = brief ? min(filled, SHORT_ITEMS) : 0u;
        uint32_t kept = filled - own;  // for the grid's list, or, where that is full, for this CTA
        if (threadIdx.x == 0) {
            for (int w = 1; w < BLOCK / 32; ++w)
                count += s_cnt[w];
            if (count)
                atomicAdd(A.ctl + CTL_CNT + i % 3, count);
            s_at = kept ? atomicAdd(item_cnt, kept) : 0u;
        }
        __syncthreads();
        if (s_at + kept <= A.item_cap) {
            for (uint32_t c = threadIdx.x; c < kept; c += BLOCK)
                A.items[s_at + c] = s_items[own + c];
            kept = 0;
        } else {
            for (uint32_t c = s_at + threadIdx.x; c < min(s_at + kept, A.item_cap); c += BLOCK)
                A.items[c] = make_uint2(0, SIZE_NONE);
            if (threadIdx.x == 0)
                atomicAdd(A.ctl + CTL_OVERFLOW, 1u);
        }
        // items c0, c0 + step, ... below c1
        auto walk = [&](const uint2 *items, uint32_t c0, uint32_t step, uint32_t c1) {
            for (uint32_t c = c0; c < c1; c += step) {
                const uint2 it = items[c];
                if (it.y == SIZE_NONE)
                    continue;  // neutral
                WordRows W;
                W.load(A, it.x, lane);
                walk_word(A, W, it.y * ITEM, (it.y + 1) * ITEM, lane, claims);
            }
        };
        walk(s_items, warp, BLOCK / 32, own);
        if (!grid_barrier_long(bar, err))
            return;
        frontier = cta_broadcast_read(A.ctl + CTL_CNT + i % 3);
        if (frontier == 0)
            break;
        reached += i == LONG_LEVELS ? 0u : frontier;
        if (gtid == 0) {
            // read last before this barrier, added to after the next one
            A.ctl[CTL_CNT + (i + 2) % 3] = 0;
            A.ctl[CTL_ITEMS + (i + 2) % 3] = 0;
        }
        const uint32_t nit = min(cta_broadcast_read(item_cnt), A.item_cap);
        const bool overflow = cta_broadcast_read(A.ctl + CTL_OVERFLOW) != 0;
        if (brief && nit == 0 && !overflow)
            continue;
        walk(A.items, gwarp, nwarps, nit);
        walk(s_items, own + warp, BLOCK / 32, own + kept);
        if (overflow) {
            for (uint32_t w = gwarp; w < words; w += nwarps) {
                if (!A.over[w])
                    continue;
                WordRows W;
                W.load(A, w, lane);
                walk_word(A, W, 0, SIZE_NONE, lane, claims);
                __syncwarp();
                if (lane == 0)
                    A.over[w] = 0;
            }
        }
        if (!grid_barrier_long(bar, err))
            return;
    }
    report(A, i, blockIdx.x == 0 ? reached : 0u);
}

const void *bfs_kernel_ptr(uint32_t size, bool long_search = false) {
    if (long_search)
        return size >= LARGE_SLOTS ? (const void *)bfs_long_kernel<LARGE_ITEM_SLOTS>
                                   : (const void *)bfs_long_kernel<ITEM_SLOTS>;
    return size >= LARGE_SLOTS ? (const void *)bfs_kernel<LARGE_ITEM_SLOTS> : (const void *)bfs_kernel<ITEM_SLOTS>;
}

// Resident CTAs per SM of either build (of those for long searches,
// LONG_CTAS_PER_SM by their launch bounds).
cudaError_t bfs_fit(int *per_sm) {
    int large = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, bfs_kernel_ptr(0), BLOCK, 0);
    if (e == cudaSuccess)
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&large, bfs_kernel_ptr(LARGE_SLOTS), BLOCK, 0);
    *per_sm = std::min(*per_sm, large);
    return e;
}

gpma_status ensure_bfs(gpma_graph *g) {
    if (g->bfs_cap >= g->row_num && g->bfs_map)
        return GPMA_OK;
    free_bfs(g);
    uint32_t n = std::max<uint32_t>(g->row_num, 1);
    GPMA_TRY(dev_alloc(&g->bfs_map, BFS_MAPS * (n / 32 + 2)));
    GPMA_TRY(dev_alloc(&g->bfs_ctl, CTL_ALL + CTL_PROFILE_WORDS));
    g->bfs_dirty = true;
    if (!g->h_bfs_ctl) {
        cudaError_t e = cudaMallocHost((void **)&g->h_bfs_ctl, sizeof(uint32_t) * (CTL_WORDS + CTL_PROFILE_WORDS));
        if (e != cudaSuccess)
            return cuda_fail(e, "cudaMallocHost(bfs ctl)");
    }
    g->bfs_cap = n;
    if (g->bfs_grid == 0) {
        int per_sm = 0;
        GPMA_CUDA(bfs_fit(&per_sm));
        if (per_sm < 1) {
            set_error("BFS kernel cannot be resident (occupancy 0)");
            return GPMA_ERR_CUDA;
        }
        g->bfs_grid = std::min(per_sm, MAX_BLOCKS_PER_SM);  // resident CTAs per SM
    }
    return GPMA_OK;
}

// CTAs for an array of `size` slots, at most `most`: one per BFS_CTA_SLOTS
// slots, since the barriers of a small search cost more the more CTAs meet.
constexpr uint32_t BFS_CTA_SLOTS = 1024;
int bfs_ctas(uint32_t size, int most) {
    return (int)std::max<uint32_t>(1, std::min<uint32_t>((uint32_t)most, size / BFS_CTA_SLOTS));
}

void fill_maps(BfsArgs &A, uint32_t *maps, size_t words) {
    A.seen = maps;
    A.done = maps + words;
    A.front = maps + 2 * words;
    A.over = maps + 3 * words;
}

// Whether a launch ended at LONG_LEVELS with a frontier left to walk.
bool long_search(const uint32_t *h_ctl) {
    return h_ctl[CTL_LEVELS] == LONG_LEVELS && h_ctl[CTL_CNT + LONG_LEVELS % 3] != 0;
}

// The launch that goes on with a search after LONG_LEVELS levels, from its
// arguments and two more maps; the control words are zero.
cudaError_t launch_long(BfsArgs A, uint32_t *maps, size_t words, int sms, int per_sm, cudaStream_t s) {
    A.claimed[0] = maps;
    A.claimed[1] = maps + words;
    A.gate = nullptr;
    A.stamps = nullptr;
    A.stall = 0;
    A.stall_limit_ns = WAIT_LIMIT_NS;
    void *params[] = {&A};
    return cudaLaunchCooperativeKernel(bfs_kernel_ptr(A.size, true),
                                       dim3(bfs_ctas(A.size, sms * std::min(per_sm, LONG_CTAS_PER_SM))), dim3(BLOCK),
                                       params, 0, s);
}

}  // namespace

void free_bfs(gpma_graph *g) {
    dev_free(g->bfs_levels);
    g->bfs_levels_cap = 0;
    dev_free(g->bfs_map);
    dev_free(g->bfs_claimed);
    dev_free(g->bfs_items);
    g->bfs_item_cap = 0;
    dev_free(g->bfs_ctl);
    g->bfs_cap = 0;
}

gpma_status bfs_plan(gpma_graph *g, uint32_t src, uint32_t *levels, BfsPlan *P, const unsigned char *gate) {
    static_assert(sizeof(BfsArgs) <= KernelLaunch::ARG_BYTES, "BFS arguments exceed the launch record");
    GPMA_TRY(ensure_bfs(g));
    const uint64_t items = bfs_item_need(g->row_num, g->geo.size);
    if (items > g->bfs_item_cap) {
        dev_free(g->bfs_items);
        g->bfs_item_cap = 0;
        GPMA_TRY(dev_alloc(&g->bfs_items, items));
        g->bfs_item_cap = (uint32_t)items;
    }
    const uint32_t n = g->row_num;
    // levels go straight to the caller's array where that is this device's memory
    P->direct = levels && levels_in_place(levels, g->device);
    if (!P->direct && n > g->bfs_levels_cap) {
        dev_free(g->bfs_levels);
        g->bfs_levels_cap = 0;
        GPMA_TRY(dev_alloc(&g->bfs_levels, n));
        g->bfs_levels_cap = n;
    }
    BfsArgs A;
    memset(&A, 0, sizeof(A));  // padding too: launches are compared byte-wise
    A.keys = g->keys;
    A.vals = g->values;
    A.ro = g->row_offset;
    A.n = n;
    A.size = g->geo.size;
    A.src = src;
    A.levels = P->direct ? levels : g->bfs_levels;
    fill_maps(A, g->bfs_map, n / 32 + 2);
    A.items = g->bfs_items;
    A.item_cap = g->bfs_item_cap;
    A.ctl = g->bfs_ctl;
    A.host = g->h_bfs_ctl;
    A.dense_div = g_tuning.bfs_dense_div;
    A.gate = gate;
    A.stamps = g->profiling ? reinterpret_cast<unsigned long long *>(g->bfs_ctl + CTL_ALL) : nullptr;
    A.stall = g_test_hooks.bfs_stall;
    A.stall_limit_ns = g_test_hooks.bfs_stall ? g_test_hooks.wait_limit_ns : WAIT_LIMIT_NS;
    P->main.set(bfs_kernel_ptr(A.size),
                bfs_ctas(g->geo.size, g->sms * blocks_per_sm(g->bfs_grid, g_tuning.bfs_blocks_per_sm)), 0, &A,
                sizeof(A));
    return GPMA_OK;
}

gpma_status bfs_begin(gpma_graph *g, cudaStream_t s) {
    if (g->bfs_dirty)  // first launch, or one that gave up: clear what a finished launch leaves zero
        GPMA_CUDA(cudaMemsetAsync(g->bfs_ctl, 0, sizeof(uint32_t) * CTL_ALL, s));
    g->bfs_dirty = true;
    g->h_bfs_ctl[CTL_ERR] = HOST_PENDING;
    return GPMA_OK;
}

gpma_status bfs_finish(gpma_graph *g, const BfsPlan &P, cudaStream_t s, uint64_t *reached) {
    uint32_t before = 0;  // nodes reached by the first launch of a long search
    if (g->h_bfs_ctl[CTL_ERR] == 0 && long_search(g->h_bfs_ctl)) {
        before = g->h_bfs_ctl[CTL_REACHED];
        BfsArgs A;
        memcpy(&A, P.main.args, sizeof(A));
        const size_t words = g->bfs_cap / 32 + 2;
        if (!g->bfs_claimed)
            GPMA_TRY(dev_alloc(&g->bfs_claimed, 2 * words));
        g->h_bfs_ctl[CTL_ERR] = HOST_PENDING;
        GPMA_CUDA(launch_long(A, g->bfs_claimed, words, g->sms, blocks_per_sm(g->bfs_grid, g_tuning.bfs_blocks_per_sm), s));
        prof_mark(g, 1, s);
        GPMA_CUDA(cudaStreamSynchronize(s));
        g->prof.kernel_launches += 1;
    }
    if (g->h_bfs_ctl[CTL_ERR] == HOST_PENDING) {
        // the kernel stopped before its end: its error word is on the device
        GPMA_CUDA(cudaMemcpy(g->h_bfs_ctl, g->bfs_ctl, sizeof(uint32_t) * CTL_WORDS, cudaMemcpyDeviceToHost));
        return device_error("the BFS kernel", g->h_bfs_ctl[CTL_ERR]);
    }
    g->bfs_dirty = false;
    if (g->h_bfs_ctl[CTL_ERR])
        return device_error("the BFS kernel", g->h_bfs_ctl[CTL_ERR]);
    if (reached)
        *reached = (uint64_t)before + g->h_bfs_ctl[CTL_REACHED];
    return GPMA_OK;
}

// Levels land in `levels` (host or device; null: nowhere); *reached is the
// count of reached nodes.
gpma_status bfs_run(gpma_graph *g, uint32_t src, uint32_t *levels, cudaStream_t s, uint64_t *reached) {
    BfsPlan P;
    GPMA_TRY(bfs_plan(g, src, levels, &P));
    GPMA_TRY(bfs_begin(g, s));
    prof_mark(g, 0, s);
    GPMA_CUDA(P.main.launch_cooperative(s));
    prof_mark(g, 1, s);
    if (g->profiling)
        GPMA_CUDA(cudaMemcpyAsync(g->h_bfs_ctl + CTL_WORDS, g->bfs_ctl + CTL_ALL,
                                  sizeof(uint32_t) * CTL_PROFILE_WORDS, cudaMemcpyDeviceToHost, s));
    GPMA_CUDA(cudaStreamSynchronize(s));
    g->prof.kernel_launches += 1;
    g->prof.bfs_kernels++;
    GPMA_TRY(bfs_finish(g, P, s, reached));
    g->prof.bfs_ms += prof_elapsed(g, 0, 1);
    if (levels && !P.direct) {
        GPMA_TRY(copy_any(levels, g->bfs_levels, sizeof(uint32_t) * g->row_num, s));
        GPMA_CUDA(cudaStreamSynchronize(s));
    }
    return GPMA_OK;
}

// ---- BFS without device allocation ------------------------------------------
// Some callers cannot allocate device memory on the fly: code that runs under
// a host-side memory arena or a fixed device-memory budget, plug-ins whose
// host process owns every cudaMalloc, or hosts whose pool forbids growth once
// serving starts. For them gpma_bfs_noalloc keeps the BFS working set (six
// bitmaps, item list, control words) in one file-scope device array
// of a fixed size instead of buffers allocated per graph. Every GPU that loads
// this library holds the array (about 2.1 MB) until the process exits.
namespace {

constexpr uint32_t NOALLOC_MAX_ROWS = 1u << 21;  // 2,097,152 nodes
constexpr uint32_t NOALLOC_BITMAP_WORDS = NOALLOC_MAX_ROWS / 32 + 2;
constexpr uint32_t NOALLOC_ITEM_CAP = 1u << 16;  // further items stay with the CTA that found them
constexpr size_t NOALLOC_WORDS = CTL_ALL + (size_t)(BFS_MAPS + 2) * NOALLOC_BITMAP_WORDS + 2ull * NOALLOC_ITEM_CAP;
constexpr int NOALLOC_MAX_DEVICES = 64;

static __device__ __align__(256) uint32_t g_noalloc_scratch[NOALLOC_WORDS];

std::mutex g_noalloc_mu;
uint32_t *g_noalloc_ptr[NOALLOC_MAX_DEVICES] = {};
int g_noalloc_grid[NOALLOC_MAX_DEVICES] = {};

// Device address of the scratch array on the current device. The host-side
// symbol is only a stand-in, so the address is looked up once per device
// (with that device current) and cached.
gpma_status noalloc_scratch(uint32_t **out, int *grid, int sms) {
    int dev = 0;
    GPMA_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= NOALLOC_MAX_DEVICES) {
        set_error("gpma_bfs_noalloc: device %d outside the supported range 0..%d", dev, NOALLOC_MAX_DEVICES - 1);
        return GPMA_ERR_INVALID;
    }
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (e != cudaSuccess)
            return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
        int per_sm = 0;
        e = bfs_fit(&per_sm);
        // a kernel is loaded when it is first used, which takes device memory: not in the middle of a later search
        cudaFuncAttributes attr;
        for (uint32_t size : {0u, LARGE_SLOTS})
            if (e == cudaSuccess)
                e = cudaFuncGetAttributes(&attr, bfs_kernel_ptr(size, true));
        if (e != cudaSuccess)
            return cuda_fail(e, "cudaOccupancyMaxActiveBlocksPerMultiprocessor(bfs_kernel)");
        if (per_sm < 1) {
            set_error("gpma_bfs_noalloc: BFS kernel cannot be resident (occupancy 0)");
            return GPMA_ERR_CUDA;
        }
        g_noalloc_grid[dev] = std::min(per_sm, MAX_BLOCKS_PER_SM);
        g_noalloc_ptr[dev] = static_cast<uint32_t *>(p);
    }
    *out = g_noalloc_ptr[dev];
    *grid = sms * blocks_per_sm(g_noalloc_grid[dev], g_tuning.bfs_blocks_per_sm);
    return GPMA_OK;
}

}  // namespace

gpma_status bfs_noalloc_run(gpma_graph *g, uint32_t src, uint32_t *levels, uint64_t *reached, cudaStream_t s) {
    const uint32_t n = g->row_num;
    if (n > NOALLOC_MAX_ROWS) {
        set_error("gpma_bfs_noalloc: graph has %u nodes; the fixed scratch holds at most %u", n, NOALLOC_MAX_ROWS);
        return GPMA_ERR_CAPACITY;
    }
    uint32_t *scratch = nullptr;
    int grid = 0;
    GPMA_TRY(noalloc_scratch(&scratch, &grid, g->sms));
    uint32_t *ctl = scratch;
    uint32_t *maps = scratch + CTL_ALL;
    // the scratch keeps the previous call's control words: clear them
    GPMA_CUDA(cudaMemsetAsync(ctl, 0, sizeof(uint32_t) * CTL_ALL, s));
    BfsArgs A;
    memset(&A, 0, sizeof(A));
    A.keys = g->keys;
    A.vals = g->values;
    A.ro = g->row_offset;
    A.n = n;
    A.size = g->geo.size;
    A.levels = levels;
    A.src = src;
    fill_maps(A, maps, NOALLOC_BITMAP_WORDS);
    A.items = reinterpret_cast<uint2 *>(maps + (size_t)(BFS_MAPS + 2) * NOALLOC_BITMAP_WORDS);
    A.item_cap = g_test_hooks.noalloc_chunk_cap ? std::min(g_test_hooks.noalloc_chunk_cap, NOALLOC_ITEM_CAP)
                                                : NOALLOC_ITEM_CAP;
    A.ctl = ctl;
    A.dense_div = g_tuning.bfs_dense_div;
    A.stamps = nullptr;
    A.stall = g_test_hooks.bfs_stall;
    A.stall_limit_ns = g_test_hooks.bfs_stall ? g_test_hooks.wait_limit_ns : WAIT_LIMIT_NS;
    void *params[] = {&A};
    GPMA_CUDA(cudaLaunchCooperativeKernel(bfs_kernel_ptr(A.size), dim3(bfs_ctas(A.size, grid)), dim3(BLOCK), params, 0, s));
    uint32_t h_ctl[CTL_WORDS], before = 0;
    GPMA_CUDA(cudaMemcpyAsync(h_ctl, ctl, sizeof(h_ctl), cudaMemcpyDeviceToHost, s));
    GPMA_CUDA(cudaStreamSynchronize(s));
    if (!h_ctl[CTL_ERR] && long_search(h_ctl)) {
        before = h_ctl[CTL_REACHED];
        const uint32_t overflows = h_ctl[CTL_OVERFLOW];
        GPMA_CUDA(cudaMemsetAsync(ctl, 0, sizeof(uint32_t) * CTL_ALL, s));
        GPMA_CUDA(launch_long(A, maps + (size_t)BFS_MAPS * NOALLOC_BITMAP_WORDS, NOALLOC_BITMAP_WORDS, g->sms, grid / g->sms, s));
        GPMA_CUDA(cudaMemcpyAsync(h_ctl, ctl, sizeof(h_ctl), cudaMemcpyDeviceToHost, s));
        GPMA_CUDA(cudaStreamSynchronize(s));
        h_ctl[CTL_OVERFLOW] += overflows;
    }
    g_test_hooks.noalloc_overflows = h_ctl[CTL_OVERFLOW];
    if (h_ctl[CTL_ERR])
        return device_error("the BFS kernel", h_ctl[CTL_ERR]);
    if (reached)
        *reached = (uint64_t)before + h_ctl[CTL_REACHED];
    return GPMA_OK;
}

}  // namespace gpma

extern "C" gpma_status gpma_bfs_level_profile(const gpma_graph *g, double *ms, uint32_t *frontier, uint8_t *dense,
                                              uint32_t capacity, uint32_t *levels) {
    using namespace gpma;
    if (!g || !levels) {
        gpma::set_error("gpma_bfs_level_profile: null argument");
        return GPMA_ERR_INVALID;
    }
    *levels = 0;
    if (!g->profiling || !g->h_bfs_ctl)
        return GPMA_OK;
    const uint32_t L = std::min<uint32_t>(g->h_bfs_ctl[CTL_LEVELS], CTL_PROFILE_LEVELS - 1);
    const uint64_t *st = reinterpret_cast<const uint64_t *>(g->h_bfs_ctl + CTL_WORDS);
    const uint32_t *info = reinterpret_cast<const uint32_t *>(st + CTL_PROFILE_LEVELS);
    *levels = L;
    for (uint32_t i = 0; i < std::min(L, capacity); ++i) {
        if (ms)
            ms[i] = (double)(st[i + 1] - st[i]) * 1e-6;
        if (frontier)
            frontier[i] = info[i] & 0x7FFFFFFFu;
        if (dense)
            dense[i] = (uint8_t)(info[i] >> 31);
    }
    return GPMA_OK;
}
