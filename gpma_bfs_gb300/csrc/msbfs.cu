// msbfs.cu - multi-source BFS over one or many GPMA graphs in one launch.
//
// No reference counterpart (the reference BFS, gpma_bfs.cuh:446-533, takes one
// source of one graph); each of the up to 64 searches per graph has the
// reference's level semantics (levels[src] = 1, a node first reached from
// level L gets L+1, slots with column 0xFFFFFFFF or value 0 are not edges).
//
// The nodes of all graphs form one index space (graph g owns
// [voff[g], voff[g+1])). Each node carries three masks of 32 or 64 bits, one bit
// lane per source: visited (reached before this level), frontier and seen (visited
// and what this level has reached so far). One persistent cooperative kernel
// runs every level, separated by bounded grid barriers:
//   expand (phase 1): a warp takes 32 consecutive nodes; the rows of those in
//     the frontier are walked as one concatenated slot range (warp-level load
//     balancing, MS_LANE_SLOTS slots per lane per step) and every edge ORs the
//     source's frontier mask, minus the lanes already there, into
//     seen[target]; rows longer than 64 slots are queued as 128-slot chunks;
//   expand (phase 2): every warp takes chunks;
//   commit: seen minus visited becomes the new frontier, visited becomes seen,
//     and the level of each newly reached (node, lane) goes into bit planes.
// A final pass counts the reached nodes per lane and writes the levels.
// The traversed-edge count (edges scanned from reached nodes, per source) is
// summed on the fly for GTEPS.
#include "gpma_internal.cuh"

#include <algorithm>
#include <numeric>

namespace gpma {
namespace {

enum : uint32_t {
    MS_CHANGE = 0,  // 3 rotating counters: CTAs that reached a new (node, lane)
    MS_CHUNKS = 3,  // 3 rotating chunk counters
    MS_ERR = 6,
    MS_LEVELS = 7,
    MS_FSLOTS = 16, // 3 rotating u64 counters (words 16..21): slots of the rows in the next union frontier
    MS_CTL_WORDS = 24,          // what the host reads
    MS_BAR = BAR_ALIGN_WORDS,   // GridBarrier
    MS_ALL = MS_BAR + BAR_WORDS,
};

constexpr uint32_t MS_BIG_ROW = 64;
constexpr uint32_t MS_CHUNK_SLOTS = 128;  // one step of a warp
// Chunk list entries for `slots` slots over all graphs: rows over MS_BIG_ROW
// slots yield at most len/128 + 1 chunks each, at most slots/65 such rows, so
// a level queues fewer than slots/128 + slots/65 < slots/32 chunks.
inline uint64_t ms_chunk_need(uint64_t slots) { return slots / 32 + 1024; }
// Chunks a CTA collects in shared memory and adds to the grid's list under one
// atomic; a warp that finds no room adds its own. (An atomic per warp and 32
// nodes, all on one word, serialised at 4.4 ns apiece.)
constexpr uint32_t MS_CTA_CHUNKS = 512;

struct MsGraph {
    const uint64_t *keys;
    const uint8_t *vals;
    const uint32_t *ro;
    uint32_t *levels;  // [nsrc][n] or null
    uint32_t n, size, nsrc, pad;
};

struct MsArgs {
    const MsGraph *gr;
    uint32_t G;
    const uint32_t *voff;  // G + 1
    const uint32_t *src;   // G * 64
    const uint64_t *soff;  // slot offsets of the concatenated arrays, G + 1 (multiples of 4)
    // masks of every node, 32 or 64 bits each (MsMask of the kernel)
    void *visited, *frontier, *seen;
    void *planes;          // MS_PLANES bit planes of the level of every (node, lane), or null without levels
    uint4 *chunks;         // {slot begin, slot end, graph, node}
    uint32_t chunk_cap;
    uint32_t *ctl;
    unsigned long long *reached;  // G * 64
    unsigned long long *traversed;
    uint32_t dense_div;    // a level whose union frontier's rows span >= slots / dense_div slots sweeps every slot (0: never)
    const uint32_t *abort;  // non-zero: return at once (a recorded step after one needing host work)
};

// Levels below 2^MS_PLANES are kept as bit planes and written once, at the
// end, whole rows of 32 nodes at a time; written when they are found, 16 lanes
// of the social graph cost 18-54 us in each of the middle levels (partly filled
// sectors of 104 MB). The few (node, lane) pairs of a deeper search go straight
// to the level arrays.
constexpr uint32_t MS_PLANES = 6;

__device__ __forceinline__ uint32_t mask_count(uint32_t m) { return __popc(m); }
__device__ __forceinline__ uint32_t mask_count(uint64_t m) { return __popcll(m); }
__device__ __forceinline__ void mask_or(uint32_t *p, uint32_t m) { atomicOr(p, m); }
__device__ __forceinline__ void mask_or(uint64_t *p, uint64_t m) {
    atomicOr((unsigned long long *)p, (unsigned long long)m);
}

__device__ __forceinline__ uint32_t graph_of_node(const MsArgs &A, uint32_t u) {
    return A.G == 1 ? 0u : segment_of(A.voff, A.G, u);
}

// Slots a lane takes per step of a row walk or a chunk, all loaded before any
// of them is used.
constexpr uint32_t MS_LANE_SLOTS = 4;
// Nodes per thread per step of a commit: as many as leave the kernel at 64
// registers, four CTAs per SM (social graph, 16 sources: 30 us per middle level
// with 1, 12 with 4; 128 graphs, 64 sources: 39 with 1, 37 with 2, and with 4
// the whole kernel half as fast again, at 108 registers).
template <typename M>
constexpr uint32_t ms_commit_nodes() { return sizeof(M) == 8 ? 2 : 4; }

// N edge slots of one lane: slot sl[j] (SIZE_NONE: none) of a graph with nodes
// from vo on, scanned with frontier mask fm[j]. The targets' seen masks are all
// read before the first update; a mask read too early costs an atomic that
// changes nothing. Returns the lanes that traverse the edges.
template <typename M, uint32_t N>
__device__ __forceinline__ uint32_t ms_visit(M *seen, const MsGraph *const (&gr)[N], const uint32_t (&vo)[N],
                                             const uint32_t (&sl)[N], const M (&fm)[N]) {
    uint32_t w[N];
    M nb[N];
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) {
        uint64_t k = KEY_NONE;
        uint8_t v = 0;
        if (sl[j] != SIZE_NONE) {
            k = gr[j]->keys[sl[j]];
            v = gr[j]->vals[sl[j]];
        }
        // the reserved column is no node
        w[j] = sl[j] != SIZE_NONE && v != 0 && (uint32_t)k < gr[j]->n ? (uint32_t)k : 0xFFFFFFFFu;
    }
#pragma unroll
    for (uint32_t j = 0; j < N; ++j)
        nb[j] = w[j] != 0xFFFFFFFFu ? fm[j] & ~seen[vo[j] + w[j]] : M(0);
    uint32_t lanes = 0;
#pragma unroll
    for (uint32_t j = 0; j < N; ++j) {
        if (w[j] != 0xFFFFFFFFu)
            lanes += mask_count(fm[j]);
        if (nb[j])
            mask_or(&seen[vo[j] + w[j]], nb[j]);
    }
    return lanes;
}

// Dense levels: 4 consecutive slots of the sweep over every graph's array
// (node offset vo, n nodes). The key's high word is its source row. The
// frontier masks of all 4, then the seen masks of their targets, are loaded
// before any update. Returns the lanes that traverse the 4 slots.
template <typename M>
__device__ __forceinline__ uint32_t ms_dense_visit4(const M *frontier, M *seen, uint32_t n, const uint64_t (&k)[4],
                                                    uint32_t v4) {
    uint32_t dst[4];
    M fm[4], nb[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t src = (uint32_t)(k[j] >> 32);
        dst[j] = (uint32_t)k[j];
        const bool ok = dst[j] != 0xFFFFFFFFu && ((v4 >> (8 * j)) & 0xFFu) != 0 && src < n && dst[j] < n;
        fm[j] = ok ? frontier[src] : M(0);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
        nb[j] = fm[j] ? fm[j] & ~seen[dst[j]] : M(0);
    uint32_t lanes = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        lanes += mask_count(fm[j]);
        if (nb[j])
            mask_or(&seen[dst[j]], nb[j]);
    }
    return lanes;
}

// Graph of concatenated slot t: the last g with soff[g] <= t.
__device__ __forceinline__ uint32_t graph_of_slot(const MsArgs &A, uint64_t t) {
    uint32_t lo = 0, hi = A.G;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (A.soff[mid] <= t)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// With several graphs the sweep goes round the CTAs in tiles of MS_TILE steps
// of 4 slots per thread, so that a thread looks for the graph of its slots once
// per tile, not once per step (128 graphs: 118-185 us per dense level, 145-246 with
// a search per step). One graph needs no search and goes step by step, which
// spreads its busy rows more evenly (8 % less per level).
constexpr uint32_t MS_TILE = 8;

// One thread's 4 slots of step i of its CTA's sweep.
struct MsQuad {
    ulonglong2 k01, k23;
    uint32_t v4, vo, n;  // the 4 values; node offset and nodes of the graph
    uint32_t g = 0;
    uint64_t base = 0, end = 0;  // the graph's concatenated slots (end 0: none looked up)
    bool ok;
    __device__ __forceinline__ void load(const MsArgs &A, uint32_t i) {
        const uint32_t steps = A.G == 1 ? 1u : MS_TILE;
        const uint64_t tile = blockIdx.x + (uint64_t)(i / steps) * gridDim.x;
        const uint64_t t = (tile * (steps * BLOCK) + (i % steps) * BLOCK + threadIdx.x) << 2;
        ok = t < A.soff[A.G];
        if (!ok)
            return;
        if (t >= end) {
            g = A.G == 1 ? 0u : graph_of_slot(A, t);
            base = A.soff[g];
            end = A.soff[g + 1];
            vo = A.voff[g];
            n = A.gr[g].n;
        }
        const uint32_t s = (uint32_t)(t - base);
        const MsGraph &Gr = A.gr[g];
        k01 = *reinterpret_cast<const ulonglong2 *>(Gr.keys + s);
        k23 = *reinterpret_cast<const ulonglong2 *>(Gr.keys + s + 2);
        v4 = *reinterpret_cast<const uint32_t *>(Gr.vals + s);
    }
};

__device__ __forceinline__ unsigned long long *fslots(const MsArgs &A, uint32_t level) {
    return reinterpret_cast<unsigned long long *>(A.ctl + MS_FSLOTS) + level % 3;
}

// Bit matrix transpose over a warp: bit i of lane l's result is bit l of lane
// i's word.
__device__ __forceinline__ uint32_t warp_transpose(uint32_t x, uint32_t lane) {
    uint32_t m = 0x0000FFFFu;  // the bits whose index has bit `j` clear
#pragma unroll
    for (uint32_t j = 16; j >= 1; j >>= 1) {
        const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, x, j);
        x = (lane & j) ? (x & ~m) | ((y >> j) & m) : (x & m) | ((y & m) << j);
        m ^= m << (j >> 1);
    }
    return x;
}

// The end of level lv - 1 (lv = 1: the seeds): what seen holds beyond visited
// is the frontier of level lv and gets that level; visited becomes seen. The
// first commit and the first use of a plane write every entry, so only seen is
// cleared beforehand. Counts the next frontier's row slots and flags a change.
template <typename M>
__device__ __forceinline__ void ms_commit(const MsArgs &A, uint32_t lv, uint32_t N, uint32_t gwarp, uint32_t nwarps,
                                          uint32_t lane) {
    constexpr uint32_t MS_COMMIT = ms_commit_nodes<M>();
    M *visited = (M *)A.visited, *frontier = (M *)A.frontier, *planes = (M *)A.planes;
    const M *seen = (const M *)A.seen;
    uint32_t changed = 0;
    unsigned long long fnext = 0;
    const bool in_planes = lv < (1u << MS_PLANES), new_plane = in_planes && planes && (lv & (lv - 1)) == 0;
    const uint32_t top = 31 - __clz(lv);
    // every load of a kind is issued before its use: the passes over the masks
    // are short, so their chains of loads decide
    for (uint64_t w0 = (uint64_t)gwarp * 32 * MS_COMMIT; w0 < N; w0 += (uint64_t)nwarps * 32 * MS_COMMIT) {
        M now[MS_COMMIT], nx[MS_COMMIT];
#pragma unroll
        for (uint32_t u = 0; u < MS_COMMIT; ++u) {
            const uint64_t w = w0 + 32 * u + lane;
            now[u] = w < N ? seen[w] : M(0);
            nx[u] = w < N && lv > 1 ? visited[w] : M(0);
        }
        uint32_t g[MS_COMMIT], r0[MS_COMMIT], r1[MS_COMMIT];
#pragma unroll
        for (uint32_t u = 0; u < MS_COMMIT; ++u) {
            const uint32_t w = (uint32_t)(w0 + 32 * u + lane);
            nx[u] = now[u] & ~nx[u];
            g[u] = r0[u] = r1[u] = 0;
            if (nx[u]) {
                g[u] = graph_of_node(A, w);
                const uint32_t *ro = A.gr[g[u]].ro + (w - A.voff[g[u]]);
                r0[u] = ro[0];
                r1[u] = ro[1];
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < MS_COMMIT; ++u) {
            const uint64_t w = w0 + 32 * u + lane;
            if (w >= N)
                continue;
            frontier[w] = nx[u];
            if (nx[u] || lv == 1)
                visited[w] = now[u];
            if (new_plane)
                planes[(size_t)top * N + w] = nx[u];
        }
        if (in_planes && planes) {
            for (uint32_t b = 0; b < MS_PLANES; ++b) {
                if (!((lv >> b) & 1) || (new_plane && b == top))
                    continue;
                M old[MS_COMMIT];
#pragma unroll
                for (uint32_t u = 0; u < MS_COMMIT; ++u)
                    old[u] = nx[u] ? planes[(size_t)b * N + w0 + 32 * u + lane] : M(0);
#pragma unroll
                for (uint32_t u = 0; u < MS_COMMIT; ++u)
                    if (nx[u])
                        planes[(size_t)b * N + w0 + 32 * u + lane] = old[u] | nx[u];
            }
        }
#pragma unroll
        for (uint32_t u = 0; u < MS_COMMIT; ++u) {
            if (!nx[u])
                continue;
            changed = 1;
            const MsGraph &Gr = A.gr[g[u]];
            const uint32_t e = min(r1[u], Gr.size);
            fnext += e > r0[u] ? e - r0[u] : 0u;
            if (in_planes || !Gr.levels)
                continue;
            const uint32_t lw = (uint32_t)(w0 + 32 * u + lane) - A.voff[g[u]];
            for (M m = nx[u]; m; m &= m - 1) {
                const uint32_t bit = sizeof(M) == 8 ? __ffsll((long long)m) - 1 : __ffs((int)m) - 1;
                Gr.levels[(size_t)bit * Gr.n + lw] = lv;
            }
        }
    }
    // one atomic per CTA and word (a plain store of a flag here, to the line
    // that the barrier polls, made every commit 35 us longer)
    if (__syncthreads_or(changed) && threadIdx.x == 0)
        atomicAdd(A.ctl + MS_CHANGE + (lv - 1) % 3, 1u);
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1)
        fnext += __shfl_xor_sync(0xFFFFFFFFu, fnext, d);
    __shared__ unsigned long long s_fnext[BLOCK / 32];
    if (lane == 0)
        s_fnext[threadIdx.x >> 5] = fnext;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < BLOCK / 32; ++i)
            fnext += s_fnext[i];
        if (fnext)
            atomicAdd(fslots(A, lv), fnext);
    }
}

// M: uint32_t for up to 32 sources in every graph, uint64_t for up to 64.
template <typename M>
__global__ void __launch_bounds__(BLOCK) msbfs_kernel(MsArgs A) {
    if (A.abort && *(const volatile uint32_t *)A.abort)
        return;
    GridBarrier *bar = reinterpret_cast<GridBarrier *>(A.ctl + MS_BAR);
    uint32_t *err = A.ctl + MS_ERR;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t gwarp = blockIdx.x * (BLOCK / 32) + (threadIdx.x >> 5);
    const uint32_t nwarps = gridDim.x * (BLOCK / 32);
    const uint32_t gtid = blockIdx.x * BLOCK + threadIdx.x;
    const uint32_t nthreads = gridDim.x * BLOCK;
    const uint32_t N = A.voff[A.G];
    M *seen = (M *)A.seen;
    const M *frontier = (const M *)A.frontier;
    unsigned long long traversed = 0;
    for (uint32_t w = gtid; w < N; w += nthreads)
        seen[w] = 0;
    if (!grid_barrier_long(bar, err))
        return;
    for (uint32_t t = gtid; t < A.G * 64; t += nthreads) {
        const uint32_t g = t >> 6, j = t & 63;
        if (j < A.gr[g].nsrc)
            mask_or(&seen[A.voff[g] + A.src[t]], M(1) << j);
    }
    if (!grid_barrier_long(bar, err))
        return;
    ms_commit<M>(A, 1, N, gwarp, nwarps, lane);
    if (!grid_barrier_long(bar, err))
        return;
    uint32_t level = 1;
    for (;; ++level) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            A.ctl[MS_CHANGE + (level + 1) % 3] = 0;
            A.ctl[MS_CHUNKS + (level + 1) % 3] = 0;
            *fslots(A, level + 2) = 0;
        }
        uint32_t *chunk_cnt = A.ctl + MS_CHUNKS + level % 3;
        __shared__ unsigned long long s_fs;
        __shared__ uint4 s_chunks[MS_CTA_CHUNKS];
        __shared__ uint32_t s_nch, s_end;  // entries claimed, entries filled
        __syncthreads();
        if (threadIdx.x == 0) {
            s_nch = 0;
            s_end = MS_CTA_CHUNKS;
            s_fs = *reinterpret_cast<volatile unsigned long long *>(fslots(A, level));
        }
        __syncthreads();
        const bool dense = A.dense_div && s_fs * A.dense_div >= A.soff[A.G];
        if (dense) {
            // expand, dense: every slot of every graph, 4 per thread per step,
            // the next step's slots read while this one's masks are gathered
            MsQuad nq;
            nq.load(A, 0);
            for (uint32_t i = 1; nq.ok; ++i) {
                const uint64_t k[4] = {nq.k01.x, nq.k01.y, nq.k23.x, nq.k23.y};
                const uint32_t v4 = nq.v4, vo = nq.vo, n = nq.n;
                nq.load(A, i);
                traversed += ms_dense_visit4<M>(frontier + vo, seen + vo, n, k, v4);
            }
        }
        // expand, phase 1 (sparse levels); the next 32 masks are read ahead
        M nf = !dense && gwarp * 32 + lane < N ? frontier[gwarp * 32 + lane] : M(0);
        for (uint32_t base = gwarp * 32; !dense && base < N; base += nwarps * 32) {
            const uint32_t u = base + lane;
            const M f = nf;
            const uint64_t un = (uint64_t)u + nwarps * 32;
            nf = un < N ? frontier[un] : M(0);
            if (__ballot_sync(0xFFFFFFFFu, f != 0) == 0)
                continue;
            uint32_t g = 0, vo = 0, b = 0, e = 0, len = 0;
            if (f) {
                g = graph_of_node(A, u);
                vo = A.voff[g];
                const MsGraph &Gr = A.gr[g];
                const uint32_t lu = u - vo;
                const uint32_t r1 = Gr.ro[lu + 1];
                b = Gr.ro[lu];
                e = min(r1, Gr.size);
                if (!in_bounds(err, b <= r1 && r1 <= Gr.size, BS_ROW))
                    b = e;  // an inconsistent row_offset: the row is skipped
                len = e > b ? e - b : 0;
            }
            const uint32_t nch = len > MS_BIG_ROW ? (len + MS_CHUNK_SLOTS - 1) / MS_CHUNK_SLOTS : 0;
            const uint32_t ch_incl = warp_incl_scan(nch);
            const uint32_t ch_total = __shfl_sync(0xFFFFFFFFu, ch_incl, 31);
            if (ch_total) {
                // into the CTA's list, or, once that is full, the grid's
                uint32_t cb = 0;
                if (lane == 0)
                    cb = atomicAdd(&s_nch, ch_total);
                cb = __shfl_sync(0xFFFFFFFFu, cb, 0);
                uint4 *list = s_chunks;
                uint32_t cap = MS_CTA_CHUNKS;
                if (cb + ch_total > cap) {
                    if (lane == 0) {
                        atomicMin(&s_end, cb);  // every later warp finds no room either
                        cb = atomicAdd(chunk_cnt, ch_total);
                    }
                    cb = __shfl_sync(0xFFFFFFFFu, cb, 0);
                    list = A.chunks;
                    cap = A.chunk_cap;
                }
                if (cb + ch_total <= cap) {
                    const uint32_t pos = cb + ch_incl - nch;
                    for (uint32_t c = 0; c < nch; ++c)
                        list[pos + c] = make_uint4(b + c * MS_CHUNK_SLOTS, min(e, b + (c + 1) * MS_CHUNK_SLOTS), g, u);
                    if (nch)
                        len = 0;
                } else {
                    for (uint32_t c = cb + lane; c < min(cb + ch_total, cap); c += 32)
                        list[c] = make_uint4(0, 0, 0, 0);
                }
            }
            const uint32_t incl = warp_incl_scan(len);
            const uint32_t excl = incl - len;
            const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
            for (uint32_t p0 = 0; p0 < total; p0 += 32 * MS_LANE_SLOTS) {
                uint32_t sl[MS_LANE_SLOTS], rvo[MS_LANE_SLOTS];
                const MsGraph *gr[MS_LANE_SLOTS];
                M fm[MS_LANE_SLOTS];
#pragma unroll
                for (uint32_t j = 0; j < MS_LANE_SLOTS; ++j) {
                    const uint32_t p = p0 + 32 * j + lane;
                    uint32_t r = 0;
#pragma unroll
                    for (uint32_t step = 16; step >= 1; step >>= 1) {
                        const uint32_t cand = r + step;
                        const uint32_t ex_c = __shfl_sync(0xFFFFFFFFu, excl, cand & 31);
                        if (cand < 32 && ex_c <= p)
                            r = cand;
                    }
                    const uint32_t rb = __shfl_sync(0xFFFFFFFFu, b, r);
                    const uint32_t rex = __shfl_sync(0xFFFFFFFFu, excl, r);
                    gr[j] = A.gr + __shfl_sync(0xFFFFFFFFu, g, r);
                    rvo[j] = __shfl_sync(0xFFFFFFFFu, vo, r);
                    fm[j] = __shfl_sync(0xFFFFFFFFu, f, r);
                    sl[j] = p < total ? rb + (p - rex) : SIZE_NONE;
                }
                traversed += ms_visit<M, MS_LANE_SLOTS>(seen, gr, rvo, sl, fm);
            }
        }
        if (!dense) {
            // the CTA's chunks join the grid's list under one atomic
            __syncthreads();
            const uint32_t mine = min(s_nch, s_end);
            __syncthreads();
            if (threadIdx.x == 0 && mine)
                s_nch = atomicAdd(chunk_cnt, mine);
            __syncthreads();
            for (uint32_t c = threadIdx.x; c < mine; c += BLOCK)
                if (in_bounds(err, s_nch + c < A.chunk_cap, BS_ROW))  // the list holds every level's chunks
                    A.chunks[s_nch + c] = s_chunks[c];
            if (!grid_barrier_long(bar, err))
                return;
        }
        // expand, phase 2: long-row chunks
        const uint32_t nch_all = dense ? 0u : min(cta_broadcast_read(chunk_cnt), A.chunk_cap);
        for (uint32_t c = gwarp; c < nch_all; c += nwarps) {
            const uint4 ch = A.chunks[c];
            if (ch.x >= ch.y)
                continue;
            const M f = frontier[ch.w];
            const uint32_t vo = A.voff[ch.z];
            uint32_t sl[MS_LANE_SLOTS], cvo[MS_LANE_SLOTS];
            const MsGraph *gr[MS_LANE_SLOTS];
            M fm[MS_LANE_SLOTS];
#pragma unroll
            for (uint32_t j = 0; j < MS_LANE_SLOTS; ++j) {
                const uint32_t sj = ch.x + 32 * j + lane;  // a chunk is one step
                sl[j] = sj < ch.y ? sj : SIZE_NONE;
                cvo[j] = vo;
                gr[j] = A.gr + ch.z;
                fm[j] = f;
            }
            traversed += ms_visit<M, MS_LANE_SLOTS>(seen, gr, cvo, sl, fm);
        }
        if (!grid_barrier_long(bar, err))
            return;
        ms_commit<M>(A, level + 1, N, gwarp, nwarps, lane);
        if (!grid_barrier_long(bar, err))
            return;
        if (cta_broadcast_read(A.ctl + MS_CHANGE + level % 3) == 0)
            break;
    }
    // reached (graph, lane) counts, and the levels from their planes (0 where a
    // lane never came): each CTA walks a contiguous node range graph by graph,
    // a warp 32 nodes at a time. Transposed over the warp, lane l's word holds
    // mask lane l of the 32 nodes, so one population count serves 32 of them
    // (a vote per mask lane took 109 us on 3M nodes and 64 lanes).
    __shared__ unsigned int cnt[64];
    const uint32_t per = (N + gridDim.x - 1) / gridDim.x;
    const uint32_t lo = min(N, blockIdx.x * per), hi = min(N, lo + per);
    const M *visited = (const M *)A.visited, *planes = (const M *)A.planes;
    // planes in use: every level is at most level + 1 (the last commit found nothing)
    const uint32_t np = min(MS_PLANES, 32u - __clz(level + 1));
    uint32_t pos = lo;
    while (__syncthreads_or(pos < hi)) {
        const uint32_t g = graph_of_node(A, pos);
        const uint32_t end = min(hi, A.voff[g + 1]);
        const uint32_t nsrc = A.gr[g].nsrc, n = A.gr[g].n;
        uint32_t *levels = A.gr[g].levels;
        const uint32_t v0 = A.voff[g];
        if (threadIdx.x < 64)
            cnt[threadIdx.x] = 0;
        __syncthreads();
        uint32_t c0 = 0, c1 = 0;
        for (uint32_t w0 = pos + (threadIdx.x & ~31u); w0 < end; w0 += BLOCK) {
            const uint32_t w = w0 + lane;
            const M m = w < end ? visited[w] : M(0);
            c0 += __popc(warp_transpose((uint32_t)m, lane));
            if (sizeof(M) == 8)
                c1 += __popc(warp_transpose((uint32_t)((uint64_t)m >> 32), lane));
            if (!levels || w >= end)
                continue;
            M pl[MS_PLANES];
#pragma unroll
            for (uint32_t b = 0; b < MS_PLANES; ++b)
                pl[b] = b < np ? planes[(size_t)b * N + w] : M(0);
            for (uint32_t j = 0; j < nsrc; ++j) {
                uint32_t lv = 0;
#pragma unroll
                for (uint32_t b = 0; b < MS_PLANES; ++b)
                    lv |= (uint32_t)((pl[b] >> j) & 1) << b;
                if (lv != 0 || !((m >> j) & 1))  // else a deep level, already written
                    levels[(size_t)j * n + (w - v0)] = lv;
            }
        }
        if (c0)
            atomicAdd(&cnt[lane], c0);
        if (c1)
            atomicAdd(&cnt[lane + 32], c1);
        __syncthreads();
        if (threadIdx.x < 64 && cnt[threadIdx.x])
            atomicAdd(&A.reached[(size_t)g * 64 + threadIdx.x], (unsigned long long)cnt[threadIdx.x]);
        pos = end;
    }
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1)
        traversed += __shfl_xor_sync(0xFFFFFFFFu, traversed, d);
    if (lane == 0 && traversed)
        atomicAdd(A.traversed, traversed);
    if (blockIdx.x == 0 && threadIdx.x == 0)
        A.ctl[MS_LEVELS] = level;
}

const void *ms_kernel_ptr(bool wide) {
    return wide ? (const void *)msbfs_kernel<uint64_t> : (const void *)msbfs_kernel<uint32_t>;
}

int g_ms_fit[64][2] = {};  // resident CTAs per SM of the two mask widths, per device

int ms_grid_size(int sms, bool wide) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64)
        dev = 0;
    int &fit = g_ms_fit[dev][wide];
    if (fit == 0) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, ms_kernel_ptr(wide), BLOCK, 0) != cudaSuccess)
            return 0;
        fit = std::min(per_sm, MAX_BLOCKS_PER_SM);
    }
    return sms * blocks_per_sm(fit, g_tuning.ms_blocks_per_sm);
}

}  // namespace

void free_batch_bfs(gpma_batch *b) {
    for (int i = 0; i < 3; ++i)
        dev_free(b->ms_mask[i]);
    dev_free(b->ms_planes);
    b->ms_planes_cap = 0;
    dev_free(b->ms_tab);
    if (b->h_ms_tab)
        cudaFreeHost(b->h_ms_tab);
    b->h_ms_tab = nullptr;
    dev_free(b->ms_ctl);
    dev_free(b->ms_reached);
    if (b->h_ms_reached)
        cudaFreeHost(b->h_ms_reached);
    b->h_ms_reached = nullptr;
    dev_free(b->ms_chunks);
    b->ms_chunk_cap = 0;
    if (b->h_ms_ctl)
        cudaFreeHost(b->h_ms_ctl);
    b->h_ms_ctl = nullptr;
    b->ms_cap = 0;
    b->ms_gcap = 0;
}

namespace {

// Byte layout of the per-call graph table (device copy and pinned mirror):
// node offsets (k + 1 u32), slot offsets (k + 1 u64), sources (64 k u32),
// graph descriptors (k MsGraph), each part 16-byte aligned.
struct MsTabLayout {
    size_t voff, soff, src, gdesc, bytes;
    explicit MsTabLayout(uint32_t k) {
        auto up = [](size_t x) { return (x + 15) & ~size_t(15); };
        voff = 0;
        soff = up(voff + 4ull * (k + 1));
        src = up(soff + 8ull * (k + 1));
        gdesc = up(src + 4ull * 64 * k);
        bytes = up(gdesc + sizeof(MsGraph) * k);
    }
};

}  // namespace

gpma_status batch_bfs_plan(gpma_batch *b, gpma_graph *const *graphs, const uint32_t *const *srcs,
                           const uint32_t *nsrc, uint32_t k, uint32_t *const *stage, BatchBfsPlan *P,
                           const uint32_t *abort) {
    static_assert(sizeof(MsArgs) <= KernelLaunch::ARG_BYTES, "multi-source BFS arguments exceed the launch record");
    // masks of 32 bits where no graph has more than 32 sources: half the mask
    // bytes of every commit, gather and plane
    bool wide = false;
    for (uint32_t i = 0; i < k; ++i)
        wide = wide || nsrc[i] > 32;
    const int grid = ms_grid_size(b->sms, wide);
    if (grid == 0) {
        set_error("multi-source BFS kernel cannot be resident");
        return GPMA_ERR_CUDA;
    }
    uint64_t N = 0, slots = 0;
    for (uint32_t i = 0; i < k; ++i) {
        N += graphs[i]->row_num;
        slots += graphs[i]->geo.size;  // sizes are powers of two >= 4
    }
    if (N > b->ms_cap || !b->ms_mask[0]) {
        for (int i = 0; i < 3; ++i)
            dev_free(b->ms_mask[i]);
        b->ms_cap = 0;
        for (int i = 0; i < 3; ++i)
            GPMA_TRY(dev_alloc(&b->ms_mask[i], std::max<uint64_t>(N, 1)));
        b->ms_cap = std::max<uint64_t>(N, 1);
    }
    bool any_levels = false;
    for (uint32_t i = 0; stage && i < k; ++i)
        any_levels = any_levels || stage[i];
    const uint64_t plane_bytes = any_levels ? (wide ? 8 : 4) * MS_PLANES * N : 0;
    if (plane_bytes > b->ms_planes_cap) {
        dev_free(b->ms_planes);
        b->ms_planes_cap = 0;
        GPMA_TRY(dev_alloc(&b->ms_planes, plane_bytes));
        b->ms_planes_cap = plane_bytes;
    }
    const MsTabLayout lay(k);
    if (k > b->ms_gcap || !b->ms_tab) {
        dev_free(b->ms_tab);
        dev_free(b->ms_reached);
        if (b->h_ms_tab)
            cudaFreeHost(b->h_ms_tab);
        if (b->h_ms_reached)
            cudaFreeHost(b->h_ms_reached);
        b->h_ms_tab = nullptr;
        b->h_ms_reached = nullptr;
        b->ms_gcap = 0;
        GPMA_TRY(dev_alloc(&b->ms_tab, lay.bytes));
        GPMA_TRY(dev_alloc(&b->ms_reached, 64ull * k + 1));
        GPMA_CUDA(cudaMallocHost((void **)&b->h_ms_tab, lay.bytes));
        GPMA_CUDA(cudaMallocHost((void **)&b->h_ms_reached, sizeof(unsigned long long) * (64ull * k + 1)));
        b->ms_gcap = k;
    }
    if (ms_chunk_need(slots) > b->ms_chunk_cap) {
        dev_free(b->ms_chunks);
        b->ms_chunk_cap = 0;
        GPMA_TRY(dev_alloc(&b->ms_chunks, 2 * ms_chunk_need(slots)));  // uint4 = 2 x uint2
        b->ms_chunk_cap = ms_chunk_need(slots);
    }
    if (!b->ms_ctl) {
        GPMA_TRY(dev_alloc(&b->ms_ctl, MS_ALL));
        GPMA_CUDA(cudaMallocHost((void **)&b->h_ms_ctl, sizeof(uint32_t) * MS_CTL_WORDS));
    }
    // the table, in the pinned mirror (the previous call's upload has finished)
    uint32_t *voff = reinterpret_cast<uint32_t *>(b->h_ms_tab + lay.voff);
    uint64_t *soff = reinterpret_cast<uint64_t *>(b->h_ms_tab + lay.soff);
    uint32_t *src = reinterpret_cast<uint32_t *>(b->h_ms_tab + lay.src);
    MsGraph *gr = reinterpret_cast<MsGraph *>(b->h_ms_tab + lay.gdesc);
    voff[0] = 0;
    soff[0] = 0;
    memset(src, 0, 4ull * 64 * k);
    for (uint32_t i = 0; i < k; ++i) {
        const gpma_graph *g = graphs[i];
        voff[i + 1] = voff[i] + g->row_num;
        soff[i + 1] = soff[i] + g->geo.size;
        gr[i].keys = g->keys;
        gr[i].vals = g->values;
        gr[i].ro = g->row_offset;
        gr[i].n = g->row_num;
        gr[i].size = g->geo.size;
        gr[i].nsrc = nsrc[i];
        gr[i].pad = 0;
        gr[i].levels = stage ? stage[i] : nullptr;
        for (uint32_t j = 0; j < nsrc[i]; ++j)
            src[64ull * i + j] = srcs[i][j];
    }
    P->tab_bytes = lay.bytes;
    void *ptr[BatchBfsPlan::CLEARS] = {b->ms_ctl, b->ms_reached};  // the kernel clears the masks
    const size_t bytes[BatchBfsPlan::CLEARS] = {sizeof(uint32_t) * MS_ALL,
                                                sizeof(unsigned long long) * (64ull * k + 1)};
    for (int i = 0; i < BatchBfsPlan::CLEARS; ++i) {
        P->clear_ptr[i] = ptr[i];
        P->clear_bytes[i] = bytes[i];
    }
    MsArgs A;
    memset(&A, 0, sizeof(A));  // padding too: launches are compared byte-wise
    A.gr = reinterpret_cast<const MsGraph *>(b->ms_tab + lay.gdesc);
    A.G = k;
    A.voff = reinterpret_cast<const uint32_t *>(b->ms_tab + lay.voff);
    A.src = reinterpret_cast<const uint32_t *>(b->ms_tab + lay.src);
    A.soff = reinterpret_cast<const uint64_t *>(b->ms_tab + lay.soff);
    A.dense_div = g_tuning.ms_dense_div;
    A.visited = b->ms_mask[0];
    A.frontier = b->ms_mask[1];
    A.seen = b->ms_mask[2];
    A.planes = any_levels ? b->ms_planes : nullptr;
    A.chunks = reinterpret_cast<uint4 *>(b->ms_chunks);
    A.chunk_cap = (uint32_t)std::min<uint64_t>(b->ms_chunk_cap, 0xFFFFFFFFull);
    A.ctl = b->ms_ctl;
    A.reached = reinterpret_cast<unsigned long long *>(b->ms_reached);
    A.traversed = reinterpret_cast<unsigned long long *>(b->ms_reached) + 64ull * k;
    A.abort = abort;
    P->main.set(ms_kernel_ptr(wide), grid, 0, &A, sizeof(A));
    P->ctl_bytes = sizeof(uint32_t) * MS_CTL_WORDS;
    P->reached_bytes = sizeof(unsigned long long) * (64ull * k + 1);
    return GPMA_OK;
}

gpma_status batch_bfs_enqueue_readback(gpma_batch *b, const BatchBfsPlan &P, cudaStream_t s) {
    GPMA_CUDA(cudaMemcpyAsync(b->h_ms_ctl, b->ms_ctl, P.ctl_bytes, cudaMemcpyDeviceToHost, s));
    GPMA_CUDA(cudaMemcpyAsync(b->h_ms_reached, b->ms_reached, P.reached_bytes, cudaMemcpyDeviceToHost, s));
    return GPMA_OK;
}

gpma_status batch_bfs_finish(gpma_batch *b, const uint32_t *nsrc, uint32_t k, uint64_t *reached) {
    b->prof.kernel_launches += 1;
    b->prof.bfs_kernels++;
    if (b->h_ms_ctl[MS_ERR])
        return device_error("the multi-source BFS kernel", b->h_ms_ctl[MS_ERR]);
    const unsigned long long *r = b->h_ms_reached;
    if (reached) {
        uint64_t o = 0;
        for (uint32_t i = 0; i < k; ++i)
            for (uint32_t j = 0; j < nsrc[i]; ++j)
                reached[o++] = r[64ull * i + j];
    }
    b->last_traversed = r[64ull * k];
    b->prof.bfs_edges += r[64ull * k];
    return GPMA_OK;
}

// Multi-source BFS of graphs[0..k) with nsrc[i] sources each. Levels (when
// levels != NULL) go to the caller's pointers, through device staging where
// those are host memory; reached receives sum(nsrc) counts.
gpma_status batch_bfs_run(gpma_batch *b, gpma_graph *const *graphs, const uint32_t *const *srcs, const uint32_t *nsrc,
                          uint32_t k, uint32_t *const *levels, uint64_t *reached, cudaStream_t s) {
    // where the kernel writes each graph's levels: the caller's array on this
    // device, or staging memory copied out afterwards (every entry is written,
    // so neither needs clearing)
    std::vector<uint32_t *> stage(k, nullptr), staged(k, nullptr);
    auto cleanup = [&]() {
        for (auto *p : staged)
            if (p)
                cudaFree(p);
    };
    auto run = [&]() -> gpma_status {
        if (levels) {
            for (uint32_t i = 0; i < k; ++i) {
                if (!levels[i])
                    continue;
                if (levels_in_place(levels[i], b->device)) {
                    stage[i] = levels[i];
                    continue;
                }
                GPMA_TRY(dev_alloc(&staged[i], (uint64_t)nsrc[i] * graphs[i]->row_num));
                stage[i] = staged[i];
            }
        }
        BatchBfsPlan P;
        GPMA_TRY(batch_bfs_plan(b, graphs, srcs, nsrc, k, levels ? stage.data() : nullptr, &P));
        GPMA_CUDA(cudaMemcpyAsync(b->ms_tab, b->h_ms_tab, P.tab_bytes, cudaMemcpyHostToDevice, s));
        for (int i = 0; i < BatchBfsPlan::CLEARS; ++i)
            GPMA_CUDA(cudaMemsetAsync(P.clear_ptr[i], 0, P.clear_bytes[i], s));
        prof_mark(b->profiling, b->ev, 0, s);
        GPMA_CUDA(P.main.launch_cooperative(s));
        prof_mark(b->profiling, b->ev, 1, s);
        GPMA_TRY(batch_bfs_enqueue_readback(b, P, s));
        GPMA_CUDA(cudaStreamSynchronize(s));
        b->prof.bfs_ms += prof_elapsed(b->profiling, b->ev, 0, 1);
        GPMA_TRY(batch_bfs_finish(b, nsrc, k, reached));
        bool copied = false;
        for (uint32_t i = 0; i < k; ++i)
            if (staged[i]) {
                GPMA_TRY(copy_any(levels[i], staged[i], sizeof(uint32_t) * nsrc[i] * (uint64_t)graphs[i]->row_num, s));
                copied = true;
            }
        if (copied)
            GPMA_CUDA(cudaStreamSynchronize(s));
        return GPMA_OK;
    };
    const gpma_status st = run();
    cleanup();
    return st;
}

}  // namespace gpma
