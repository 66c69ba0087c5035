// analytics.cu - PageRank and weakly connected components over the gapped PMA.
//
// No reference counterpart: the reference's only analytic is the BFS
// (gpma_bfs.cuh); GPMA+'s setting also covers connected components and
// PageRank. Both run as persistent cooperative kernels that read the edges in
// coalesced sweeps over every slot of the array (16-byte key loads, 8 slots
// per thread): a slot is an edge u -> v when its value is non-zero and its
// column is not 0xFFFFFFFF (the BFS's rule), with u = key >> 32 and
// v = low word, both < row_num. No in-edge index is kept between calls.
//
// PageRank (y = d * A^T (x / deg) + teleport): per iteration
//   contrib[u] = rank[u] / outdeg[u] (dangling nodes pool their rank),
//   acc[v]     = sum of contrib[u] over the edges u -> v (gathered from the
//                in-edges laid out once per call, or, for few iterations,
//                by float atomics),
//   rank'[v]   = (1 - d) / n + d * (acc[v] + dangling / n);
// it stops after `iterations` or when sum |rank' - rank| < tol.
// Weakly connected components: parents start as the node ids; an edge links
// its endpoints' trees by hooking the larger root under the smaller (a
// compare-and-swap retried from the parents it found), so one sweep over the
// edges finishes the components. Before it, passes over the first few slots of
// every row link some edges and flatten the trees; the sweep then finds most
// endpoints with equal parents and only reads (linking and sampling as in
// Afforest: Sutton, Ben-Nun and Barak, 2018). Parents only decrease and stay
// inside their component, so each node ends labelled with the smallest node id
// of its component, whatever the order of the atomics.
#include "gpma_internal.cuh"

namespace gpma {
namespace {

enum : uint32_t {
    AN_ERR = 0,
    AN_ITERS = 1,
    AN_ROOTS = 2,    // components counted
    AN_CHUNKS = 3,   // PageRank by gathering: chunks of long in-edge rows
    AN_MULTI = 4,    // ... and rows of more than one chunk
    AN_DBL = 8,      // doubles from word 8: dangling[3], delta[3]
    AN_WORDS = 8 + 12,        // what the host reads
    AN_BAR = BAR_ALIGN_WORDS, // GridBarrier
    AN_ALL = AN_BAR + BAR_WORDS,
};

constexpr int AN_MAX_FIT = 8;  // CTAs per SM

struct AnArgs {
    const uint64_t *keys;
    const uint8_t *vals;
    const uint32_t *ro;  // row offsets (components)
    uint32_t n, size;
    uint32_t *deg;     // out-degree (PageRank)
    float *rank, *acc, *contrib;
    uint32_t *parent;  // components
    // PageRank by gathering: contributions of the next iteration (acc holds
    // none of its own), ends of the in-edge rows, sources of the in-edges, long
    // rows' chunks {node, first, end, multi index}, rows of several chunks
    // {node, sum} and one word per CTA
    uint32_t *end, *csc;
    uint4 *chunks;
    uint2 *multi;
    uint32_t *cta;
    uint32_t *ctl;
    float damping;
    double tol;
    uint32_t max_iter;
};

// The 8 slots at o*8 as (u, v) edges; edge[j] false where the slot is not an edge.
__device__ __forceinline__ void load8(const AnArgs &A, uint32_t o, uint32_t (&u)[8], uint32_t (&v)[8],
                                      bool (&edge)[8]) {
    const ulonglong2 *kv = reinterpret_cast<const ulonglong2 *>(A.keys);
    const ulonglong2 k0 = kv[4 * o], k1 = kv[4 * o + 1], k2 = kv[4 * o + 2], k3 = kv[4 * o + 3];
    const uint2 vv = reinterpret_cast<const uint2 *>(A.vals)[o];
    const uint64_t k[8] = {k0.x, k0.y, k1.x, k1.y, k2.x, k2.y, k3.x, k3.y};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        u[j] = (uint32_t)(k[j] >> 32);
        v[j] = (uint32_t)k[j];
        const uint32_t val = ((j < 4 ? vv.x : vv.y) >> (8 * (j & 3))) & 0xFFu;
        edge[j] = v[j] != 0xFFFFFFFFu && val != 0 && u[j] < A.n && v[j] < A.n;
    }
}

// Arrays of 4 slots (the smallest size) as one padded group of 8.
__device__ __forceinline__ void load_small(const AnArgs &A, uint32_t (&u)[8], uint32_t (&v)[8], bool (&edge)[8]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint64_t k = j < 4 ? A.keys[j] : KEY_NONE;
        const uint32_t val = j < 4 ? A.vals[j] : 0u;
        u[j] = (uint32_t)(k >> 32);
        v[j] = (uint32_t)k;
        edge[j] = v[j] != 0xFFFFFFFFu && val != 0 && u[j] < A.n && v[j] < A.n;
    }
}

__device__ __forceinline__ double *an_dbl(const AnArgs &A, int which, uint32_t it) {
    return reinterpret_cast<double *>(A.ctl + AN_DBL) + which * 3 + it % 3;
}

__device__ __forceinline__ double block_sum_f64(double x, double *tmp) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1)
        x += __shfl_xor_sync(0xFFFFFFFFu, x, d);
    __syncthreads();
    if ((threadIdx.x & 31) == 0)
        tmp[threadIdx.x >> 5] = x;
    __syncthreads();
    double t = 0;
    if (threadIdx.x == 0)
        for (int w = 0; w < BLOCK / 32; ++w)
            t += tmp[w];
    return t;  // valid in thread 0
}

// PageRank calls of up to SHORT_CALL iterations (three barriers each) take fewer than
// 2^32 tickets and so the plain barrier, in builds of their own (20 iterations on
// the social graph, by gathering: 1,995 us, 2,040 with the other).
constexpr uint32_t SHORT_CALL = 1u << 18;
template <bool LONG>
__device__ __forceinline__ bool an_barrier(GridBarrier *bar, uint32_t *err) {
    return LONG ? grid_barrier_long(bar, err) : grid_barrier(bar, err);
}

// Ranks, degrees and sums of a call's start, and the out-degrees: slots are sorted
// by source, so a thread's 8 slots form a few runs of one source, with one atomic
// each. False when a barrier gave up.
template <bool LONG>
__device__ __forceinline__ bool pr_begin(const AnArgs &A, GridBarrier *bar, uint32_t gtid, uint32_t nthreads) {
    uint32_t *err = A.ctl + AN_ERR;
    for (uint32_t v = gtid; v < A.n; v += nthreads) {
        A.deg[v] = 0;
        A.rank[v] = 1.0f / (float)A.n;
        A.acc[v] = 0.0f;
    }
    if (!an_barrier<LONG>(bar, err))
        return false;
    for (uint32_t o = gtid; o < A.size >> 3 || (A.size < 8 && o == 0); o += nthreads) {
        uint32_t u[8], v[8];
        bool e[8];
        if (A.size < 8)
            load_small(A, u, v, e);
        else
            load8(A, o, u, v, e);
        uint32_t run_u = 0xFFFFFFFFu, run = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (!e[j])
                continue;
            if (u[j] != run_u) {
                if (run)
                    atomicAdd(&A.deg[run_u], run);
                run_u = u[j];
                run = 0;
            }
            ++run;
        }
        if (run)
            atomicAdd(&A.deg[run_u], run);
        if (A.size < 8)
            break;
    }
    return an_barrier<LONG>(bar, err);
}

// Iteration `it` by adding every edge's contribution; the change of the ranks, the
// same in every thread of the grid, or a negative number when a barrier gave up.
template <bool LONG>
__device__ __forceinline__ double pr_push(const AnArgs &A, GridBarrier *bar, uint32_t it, uint32_t gtid,
                                          uint32_t nthreads, double *tmp, double &s_val) {
    uint32_t *err = A.ctl + AN_ERR;
    const float teleport = (1.0f - A.damping) / (float)A.n;
    if (gtid == 0) {
        *an_dbl(A, 0, it + 1) = 0.0;  // next iteration's sums start at zero
        *an_dbl(A, 1, it + 1) = 0.0;
    }
    double dang = 0;
    for (uint32_t v = gtid; v < A.n; v += nthreads) {
        const uint32_t d = A.deg[v];
        const float r = A.rank[v];
        A.contrib[v] = d ? r / (float)d : 0.0f;
        if (!d)
            dang += r;
    }
    dang = block_sum_f64(dang, tmp);
    if (threadIdx.x == 0 && dang != 0.0)
        atomicAdd(an_dbl(A, 0, it), dang);
    if (!an_barrier<LONG>(bar, err))
        return -1.0;
    for (uint32_t o = gtid; o < A.size >> 3 || (A.size < 8 && o == 0); o += nthreads) {
        uint32_t u[8], v[8];
        bool e[8];
        if (A.size < 8)
            load_small(A, u, v, e);
        else
            load8(A, o, u, v, e);
        float c[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            c[j] = e[j] ? A.contrib[u[j]] : 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (e[j] && c[j] != 0.0f)
                atomicAdd(&A.acc[v[j]], c[j]);
        if (A.size < 8)
            break;
    }
    if (!an_barrier<LONG>(bar, err))
        return -1.0;
    if (threadIdx.x == 0)
        s_val = *reinterpret_cast<volatile double *>(an_dbl(A, 0, it));
    __syncthreads();
    const float base = teleport + A.damping * (float)(s_val / (double)A.n);
    double delta = 0;
    for (uint32_t v = gtid; v < A.n; v += nthreads) {
        const float nr = base + A.damping * A.acc[v];
        delta += fabs((double)nr - (double)A.rank[v]);
        A.rank[v] = nr;
        A.acc[v] = 0.0f;
    }
    delta = block_sum_f64(delta, tmp);
    if (threadIdx.x == 0)
        atomicAdd(an_dbl(A, 1, it), delta);
    if (!an_barrier<LONG>(bar, err))
        return -1.0;
    if (threadIdx.x == 0)
        s_val = *reinterpret_cast<volatile double *>(an_dbl(A, 1, it));
    __syncthreads();
    delta = s_val;
    __syncthreads();  // s_val is written again
    return delta;
}

template <bool LONG>
__global__ void __launch_bounds__(BLOCK) pagerank_kernel(AnArgs A) {
    GridBarrier *bar = reinterpret_cast<GridBarrier *>(A.ctl + AN_BAR);
    __shared__ double tmp[BLOCK / 32];
    __shared__ double s_val;
    const uint32_t gtid = blockIdx.x * BLOCK + threadIdx.x, nthreads = gridDim.x * BLOCK;
    if (!pr_begin<LONG>(A, bar, gtid, nthreads))
        return;
    uint32_t it = 0;
    for (; it < A.max_iter; ++it) {
        const double delta = pr_push<LONG>(A, bar, it, gtid, nthreads, tmp, s_val);
        if (delta < 0.0)
            return;
        if (delta < A.tol) {
            ++it;
            break;
        }
    }
    if (gtid == 0)
        A.ctl[AN_ITERS] = it;
}

// ---- PageRank by gathering ---------------------------------------------------
// In-edge rows of at most PR_SHORT edges are summed by a thread each, PR_STEP
// edges at a time; longer ones are cut into chunks of PR_CHUNK edges, a warp
// per chunk. Per iteration on the social graph (15.3M edges, 1.6M nodes):
// 74 us; 80, 124 and 214 us with 2, 4 and 8 lanes per row (each row has its
// bounds, degree and result to handle, whatever the lanes), 106 and 84 us with
// chunks from 16 and 128 edges on, 79 us with steps of 4.
constexpr uint32_t PR_STEP = 8;
constexpr uint32_t PR_SHORT = 64;
constexpr uint32_t PR_CHUNK = 4096;
// PageRank calls of at least PR_GATHER_ITERATIONS iterations lay out the
// in-edges first (one count and one scatter sweep with an atomic per edge):
// social graph, 3 / 4 / 5 iterations, adding per edge 734 / 930 / 1130 us,
// gathering 738 / 812 / 883 us; R-MAT scale 14 123 / 150 / 178 against 118 /
// 126 / 136 us.
constexpr uint32_t PR_GATHER_ITERATIONS = 4;
// How far the ranks' change falls from the first iteration to the second, about
// (R-MAT graphs 0.35, the social graph 0.47, uniformly random ones 0.2).
constexpr double PR_FALL = 0.4;

// New rank, next contribution and this thread's share of the sums of node v.
struct PrNode {
    float base, damping;
    float *next;
    bool want_delta;
    double dang, delta;
    __device__ __forceinline__ void finish(const AnArgs &A, uint32_t v, uint32_t d, float acc) {
        const float nr = base + damping * acc;
        if (want_delta)
            delta += fabs((double)nr - (double)A.rank[v]);
        A.rank[v] = nr;
        next[v] = d ? nr / (float)d : 0.0f;
        if (!d)
            dang += nr;
    }
};

// PageRank with the in-edges of the array's current edges laid out once per
// call (counts, a grid-wide scan, one scatter of source ids), so that an
// iteration gathers contributions and writes each rank once (one float atomic
// per edge takes 198 us per iteration). Bound by the 4-byte gathers of the
// contributions (L2). 20 iterations on the social graph: 1.99 ms per call, 0.44 of
// it the layout; 4.37 by atomics.
// TOL (a tolerance is given): the iterations are not known beforehand. The call begins
// with iterations by atomics, and lays out the in-edges after the first one from which
// PR_GATHER_ITERATIONS more are to be expected: R-MAT 18, tolerance 0.5 (2 iterations)
// 402 us with the layout at once, 315 so, 313 by atomics alone; 1e-2 (6 iterations)
// 597, 708 and 822.
template <bool LONG, bool TOL>
__global__ void __launch_bounds__(BLOCK) pagerank_gather_kernel(AnArgs A) {
    GridBarrier *bar = reinterpret_cast<GridBarrier *>(A.ctl + AN_BAR);
    uint32_t *err = A.ctl + AN_ERR;
    __shared__ double tmp[BLOCK / 32];
    __shared__ uint32_t utmp[BLOCK / 32 + 1];
    __shared__ double s_val;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t gtid = blockIdx.x * BLOCK + threadIdx.x, nthreads = gridDim.x * BLOCK;
    const uint32_t gwarp = gtid >> 5, nwarps = nthreads >> 5;
    const uint32_t groups = A.size >> 3;
    const float teleport = (1.0f - A.damping) / (float)A.n;
    uint32_t first = 0;  // iterations done before the layout
    if constexpr (TOL) {
        for (uint32_t v = gtid; v < A.n; v += nthreads)
            A.end[v] = 0;
        if (!pr_begin<LONG>(A, bar, gtid, nthreads))
            return;
        for (double last = 0.0;;) {
            const double delta = pr_push<LONG>(A, bar, first, gtid, nthreads, tmp, s_val);
            if (delta < 0.0)
                return;
            ++first;
            if (delta < A.tol || first == A.max_iter) {
                if (gtid == 0)
                    A.ctl[AN_ITERS] = first;
                return;
            }
            // iterations to come, if the change goes on falling as it did
            const double fall = first == 1 ? PR_FALL : delta / last;
            uint32_t more = 0;
            for (double x = delta; x >= A.tol && more < PR_GATHER_ITERATIONS; x *= fall)
                ++more;
            if (more == PR_GATHER_ITERATIONS && A.max_iter - first >= PR_GATHER_ITERATIONS)
                break;
            last = delta;
        }
        if (gtid == 0)
            *an_dbl(A, 0, first + 1) = 0.0;
        for (uint32_t o = gtid; o < groups; o += nthreads) {
            uint32_t u[8], v[8];
            bool e[8];
            load8(A, o, u, v, e);
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (e[j])
                    atomicAdd(&A.end[v[j]], 1u);
        }
    } else {
        for (uint32_t v = gtid; v < A.n; v += nthreads) {
            A.deg[v] = 0;
            A.end[v] = 0;
        }
        if (!an_barrier<LONG>(bar, err))
            return;
        // out-degrees (one atomic per run of a source) and in-degrees
        for (uint32_t o = gtid; o < groups; o += nthreads) {
            uint32_t u[8], v[8];
            bool e[8];
            load8(A, o, u, v, e);
            uint32_t run_u = 0xFFFFFFFFu, run = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (!e[j])
                    continue;
                if (u[j] != run_u) {
                    if (run)
                        atomicAdd(&A.deg[run_u], run);
                    run_u = u[j];
                    run = 0;
                }
                ++run;
                atomicAdd(&A.end[v[j]], 1u);
            }
            if (run)
                atomicAdd(&A.deg[run_u], run);
        }
    }
    if (!an_barrier<LONG>(bar, err))
        return;
    // each CTA's nodes: in-edge total, initial ranks' contributions
    const uint32_t per = (A.n + gridDim.x - 1) / gridDim.x;
    const uint32_t lo = min(A.n, blockIdx.x * per), hi = min(A.n, lo + per);
    const float r0 = 1.0f / (float)A.n;
    {
        uint32_t in = 0;
        double dang = 0;
        for (uint32_t v = lo + threadIdx.x; v < hi; v += BLOCK) {
            const uint32_t d = A.deg[v];
            in += A.end[v];
            const float r = TOL ? A.rank[v] : r0;
            if (!TOL)
                A.rank[v] = r0;
            A.contrib[v] = d ? r / (float)d : 0.0f;
            if (!d)
                dang += r;
        }
        in = block_sum(in, utmp);
        dang = block_sum_f64(dang, tmp);
        if (threadIdx.x == 0) {
            A.cta[blockIdx.x] = in;
            if (dang != 0.0)
                atomicAdd(an_dbl(A, 0, first), dang);
        }
    }
    if (!an_barrier<LONG>(bar, err))
        return;
    {
        // first in-edge of every row (the cursor of the scatter, which leaves
        // it at the row's end), and the chunks of long rows
        uint32_t run = 0;
        for (uint32_t c = threadIdx.x; c < blockIdx.x; c += BLOCK)
            run += __ldcg(A.cta + c);
        run = block_sum(run, utmp);
        for (uint32_t v0 = lo; v0 < hi; v0 += BLOCK) {
            const uint32_t v = v0 + threadIdx.x;
            const uint32_t len = v < hi ? A.end[v] : 0u;
            uint32_t tot;
            const uint32_t b = run + block_excl_scan(len, &tot, utmp);
            if (v < hi)
                A.end[v] = b;
            if (len > PR_SHORT) {
                const uint32_t nch = (len + PR_CHUNK - 1) / PR_CHUNK;
                uint32_t m = SIZE_NONE;
                if (nch > 1) {
                    m = atomicAdd(A.ctl + AN_MULTI, 1u);
                    A.multi[m] = make_uint2(v, 0u);
                }
                const uint32_t at = atomicAdd(A.ctl + AN_CHUNKS, nch);
                for (uint32_t c = 0; c < nch; ++c)
                    A.chunks[at + c] = make_uint4(v, b + c * PR_CHUNK, b + min(len, (c + 1) * PR_CHUNK), m);
            }
            run += tot;
        }
    }
    if (!an_barrier<LONG>(bar, err))
        return;
    for (uint32_t o = gtid; o < groups; o += nthreads) {
        uint32_t u[8], v[8], at[8];
        bool e[8];
        load8(A, o, u, v, e);
#pragma unroll
        for (int j = 0; j < 8; ++j)
            at[j] = e[j] ? atomicAdd(&A.end[v[j]], 1u) : 0u;
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (e[j])
                A.csc[at[j]] = u[j];
    }
    if (!an_barrier<LONG>(bar, err))
        return;
    const uint32_t nch = cta_broadcast_read(A.ctl + AN_CHUNKS), nmulti = cta_broadcast_read(A.ctl + AN_MULTI);
    uint32_t it = first;
    for (; it < A.max_iter; ++it) {
        if (gtid == 0) {
            *an_dbl(A, 0, it + 2) = 0.0;  // the sums of the iteration after next / of the next start at zero
            *an_dbl(A, 1, it + 1) = 0.0;
        }
        if (threadIdx.x == 0)
            s_val = *reinterpret_cast<volatile double *>(an_dbl(A, 0, it));
        __syncthreads();
        const float *cur = (it - first) & 1 ? A.acc : A.contrib;
        PrNode P;
        P.base = teleport + A.damping * (float)(s_val / (double)A.n);
        P.damping = A.damping;
        P.next = (it - first) & 1 ? A.contrib : A.acc;
        P.want_delta = TOL;
        P.dang = P.delta = 0.0;
        for (uint32_t c = gwarp; c < nch; c += nwarps) {
            const uint4 ch = A.chunks[c];
            float sum = 0.0f;
            for (uint32_t p = ch.y + lane; p < ch.z; p += 8 * 32) {
                uint32_t id[8];
                float x[8];
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    id[j] = p + 32 * j < ch.z ? A.csc[p + 32 * j] : SIZE_NONE;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    x[j] = id[j] != SIZE_NONE ? cur[id[j]] : 0.0f;
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    sum += x[j];
            }
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1)
                sum += __shfl_xor_sync(0xFFFFFFFFu, sum, d);
            if (lane == 0) {
                if (ch.w == SIZE_NONE)
                    P.finish(A, ch.x, A.deg[ch.x], sum);
                else
                    atomicAdd(reinterpret_cast<float *>(&A.multi[ch.w].y), sum);
            }
        }
        // short rows as a pipeline: a row's bounds are read two rows ahead and
        // its first sources one row ahead, so a row waits for its
        // contributions only
        auto bounds = [&](uint32_t r, uint32_t &b, uint32_t &e) {
            b = r > 0 && r < A.n ? A.end[r - 1] : 0u;
            e = r < A.n ? A.end[r] : 0u;
        };
        auto sources = [&](uint32_t p, uint32_t e, uint32_t (&id)[PR_STEP]) {
#pragma unroll
            for (uint32_t j = 0; j < PR_STEP; ++j)
                id[j] = p + j < e ? A.csc[p + j] : SIZE_NONE;
        };
        uint32_t b, e, nb, ne, id[PR_STEP];
        bounds(gtid, b, e);
        bounds(gtid + nthreads, nb, ne);
        sources(b, e, id);
        for (uint32_t v = gtid; v < A.n; v += nthreads) {
            const bool mine = e - b <= PR_SHORT;
            const uint32_t deg = mine ? A.deg[v] : 0u;
            float x[PR_STEP];
#pragma unroll
            for (uint32_t j = 0; j < PR_STEP; ++j)
                x[j] = id[j] != SIZE_NONE ? cur[id[j]] : 0.0f;
            uint32_t nid[PR_STEP], b2, e2;
            sources(nb, ne, nid);
            bounds(v + 2 * nthreads, b2, e2);
            float sum = 0.0f;
#pragma unroll
            for (uint32_t j = 0; j < PR_STEP; ++j)
                sum += x[j];
            if (mine) {
                for (uint32_t p = b + PR_STEP; p < e; p += PR_STEP) {
                    sources(p, e, id);
#pragma unroll
                    for (uint32_t j = 0; j < PR_STEP; ++j)
                        x[j] = id[j] != SIZE_NONE ? cur[id[j]] : 0.0f;
#pragma unroll
                    for (uint32_t j = 0; j < PR_STEP; ++j)
                        sum += x[j];
                }
                P.finish(A, v, deg, sum);
            }
            b = nb;
            e = ne;
            nb = b2;
            ne = e2;
#pragma unroll
            for (uint32_t j = 0; j < PR_STEP; ++j)
                id[j] = nid[j];
        }
        if (nmulti) {
            // rows of several chunks, once every chunk has been added
            if (!an_barrier<LONG>(bar, err))
                return;
            for (uint32_t m = gtid; m < nmulti; m += nthreads) {
                const uint2 r = A.multi[m];
                P.finish(A, r.x, A.deg[r.x], __uint_as_float(r.y));
                A.multi[m].y = 0u;
            }
        }
        const double dang = block_sum_f64(P.dang, tmp);
        if (threadIdx.x == 0 && dang != 0.0)
            atomicAdd(an_dbl(A, 0, it + 1), dang);
        if (P.want_delta) {
            const double delta = block_sum_f64(P.delta, tmp);
            if (threadIdx.x == 0)
                atomicAdd(an_dbl(A, 1, it), delta);
        }
        if (!an_barrier<LONG>(bar, err))
            return;
        if (P.want_delta) {
            if (threadIdx.x == 0)
                s_val = *reinterpret_cast<volatile double *>(an_dbl(A, 1, it));
            __syncthreads();
            const bool done = s_val < A.tol;
            __syncthreads();  // s_val is written again
            if (done) {
                ++it;
                break;
            }
        }
    }
    if (gtid == 0)
        A.ctl[AN_ITERS] = it;
}

// Joins the trees of nodes p1 and p2 (any nodes of them): the larger of the
// two is hooked under the smaller if it is a root, else its parent goes on
// instead. Parents are read through L1: every walk ends at the same few nodes
// near the root, and reading those from L2 (240 us against 81 for the second
// sampled pass), or trying a swap on each node of a walk (7.8 ms for the whole
// call), serialises there. An old parent is still a node of the tree, and the
// swap's result is never old. The larger node decreases in every step, so the
// loop ends.
__device__ __forceinline__ void cc_link(uint32_t *parent, uint32_t p1, uint32_t p2) {
    while (p1 != p2) {
        const uint32_t hi = max(p1, p2), lo = min(p1, p2);
        uint32_t up = parent[hi];
        if (up == hi) {
            up = atomicCAS(&parent[hi], hi, lo);
            if (up == hi)
                return;
        }
        p1 = up;
        p2 = parent[lo];
    }
}

// Every node of the grid's stride to the root of its (decreasing) chain;
// returns the roots among them.
__device__ __forceinline__ uint32_t cc_flatten(uint32_t *parent, uint32_t n, uint32_t gtid, uint32_t nthreads) {
    uint32_t roots = 0;
    for (uint32_t v = gtid; v < n; v += nthreads) {
        const uint32_t first = parent[v];
        uint32_t p = first;
        for (uint32_t q = parent[p]; q != p; q = parent[p])
            p = q;
        if (p != first)
            parent[v] = p;
        roots += p == v;
    }
    return roots;
}

// Slots at the start of every row that the sampled passes look at: the guard
// of the row before and, at the array's density, the row's first edges.
constexpr uint32_t CC_SAMPLE = 4;

// Links edge number `which` among the first CC_SAMPLE slots of rows 0, step,
// 2 * step, ...
__device__ __forceinline__ void cc_sample(const AnArgs &A, uint32_t which, uint32_t step, uint32_t gtid,
                                          uint32_t nthreads) {
    for (uint64_t t = (uint64_t)gtid * step; t < A.n; t += (uint64_t)nthreads * step) {
        const uint32_t u = (uint32_t)t;
        const uint32_t r1 = A.ro[u + 1], b = A.ro[u];
        uint32_t e = min(r1, A.size);
        if (!in_bounds(A.ctl + AN_ERR, b <= r1 && r1 <= A.size, BS_ROW))
            e = b;  // an inconsistent row_offset: the row is skipped
        uint64_t k[CC_SAMPLE];
        uint32_t val[CC_SAMPLE];
#pragma unroll
        for (uint32_t j = 0; j < CC_SAMPLE; ++j) {
            k[j] = b + j < e ? A.keys[b + j] : KEY_NONE;
            val[j] = b + j < e ? A.vals[b + j] : 0u;
        }
        uint32_t v = u, seen = 0;
#pragma unroll
        for (uint32_t j = 0; j < CC_SAMPLE; ++j) {
            const uint32_t w = (uint32_t)k[j];
            const bool edge = val[j] != 0 && w < A.n;  // guards and empty slots: w is 0xFFFFFFFF
            if (edge && seen == which)
                v = w;
            seen += edge;
        }
        if (v != u)
            cc_link(A.parent, A.parent[u], A.parent[v]);
    }
}

// Bound by the 4-byte parent gathers of the edges' targets (L2) beside one
// read of the array. Linking to completion takes one sweep, and few of its edges
// link anything after the sampled passes, whose trees are flattened after each
// so that the next pass finds roots with one read: 0.22 ms on 15.3M edges, 1.6M
// nodes (33.5M slots). Hooking parents found once per round takes three sweeps with
// an atomicMin per edge in the first: 2.11 ms.
__global__ void __launch_bounds__(BLOCK) components_kernel(AnArgs A) {
    GridBarrier *bar = reinterpret_cast<GridBarrier *>(A.ctl + AN_BAR);
    uint32_t *err = A.ctl + AN_ERR;
    __shared__ uint32_t tmp[BLOCK / 32 + 1];
    const uint32_t gtid = blockIdx.x * BLOCK + threadIdx.x, nthreads = gridDim.x * BLOCK;
    const uint32_t groups = A.size >> 3;
    for (uint32_t v = gtid; v < A.n; v += nthreads)
        A.parent[v] = v;
    if (!grid_barrier(bar, err))
        return;
    // the first edge of every row, then the second of every 8th row (the large
    // component forms, with an eighth of the walks that would meet in it; 81 us
    // without this pass, 64 with it), then of all rows
    for (uint32_t pass = 0; pass < 3; ++pass) {
        cc_sample(A, pass > 0, pass == 1 ? 8 : 1, gtid, nthreads);
        if (!grid_barrier(bar, err))
            return;
        cc_flatten(A.parent, A.n, gtid, nthreads);
        if (!grid_barrier(bar, err))
            return;
    }
    for (uint32_t o = gtid; o < groups || (A.size < 8 && o == 0); o += nthreads) {
        uint32_t u[8], v[8];
        bool e[8];
        if (A.size < 8)
            load_small(A, u, v, e);
        else
            load8(A, o, u, v, e);
        // parents read once (an older parent is still a node of the tree)
        uint32_t pu[8], pv[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            pu[j] = e[j] ? A.parent[u[j]] : 0u;
            pv[j] = e[j] ? A.parent[v[j]] : 0u;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (pu[j] != pv[j])
                cc_link(A.parent, pu[j], pv[j]);
    }
    if (!grid_barrier(bar, err))
        return;
    const uint32_t roots = block_sum(cc_flatten(A.parent, A.n, gtid, nthreads), tmp);
    if (threadIdx.x == 0 && roots)
        atomicAdd(A.ctl + AN_ROOTS, roots);
    if (gtid == 0)
        A.ctl[AN_ITERS] = 1;
}

// Rows of the fit table: the kernels of this file.
enum AnKernel {
    AN_PAGERANK,
    AN_PAGERANK_GATHER,
    AN_PAGERANK_LONG,
    AN_PAGERANK_GATHER_LONG,
    AN_PAGERANK_TOL,
    AN_COMPONENTS,
    AN_KERNELS
};
int an_fit[64][AN_KERNELS] = {};  // resident CTAs per SM, per device

gpma_status launch(AnKernel which, AnArgs &A, int sms, cudaStream_t s, uint32_t *h_ctl) {
    const void *const kernels[AN_KERNELS] = {
        (const void *)pagerank_kernel<false>,      (const void *)pagerank_gather_kernel<false, false>,
        (const void *)pagerank_kernel<true>,       (const void *)pagerank_gather_kernel<true, false>,
        (const void *)pagerank_gather_kernel<true, true>, (const void *)components_kernel};
    if (A.max_iter > SHORT_CALL && which <= AN_PAGERANK_GATHER)
        which = which == AN_PAGERANK ? AN_PAGERANK_LONG : AN_PAGERANK_GATHER_LONG;
    const void *kernel = kernels[which];
    int dev = 0;
    GPMA_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64)
        dev = 0;
    int &fit = an_fit[dev][which];
    if (fit == 0) {
        int f = 0;
        GPMA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&f, kernel, BLOCK, 0));
        if (f < 1) {
            set_error("analytics kernels cannot be resident");
            return GPMA_ERR_CUDA;
        }
        fit = std::min(f, AN_MAX_FIT);
    }
    void *params[] = {&A};
    GPMA_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(sms * fit), dim3(BLOCK), params, 0, s));
    GPMA_CUDA(cudaMemcpyAsync(h_ctl, A.ctl, sizeof(uint32_t) * AN_WORDS, cudaMemcpyDeviceToHost, s));
    GPMA_CUDA(cudaStreamSynchronize(s));
    if (h_ctl[AN_ERR])
        return device_error("an analytics kernel", h_ctl[AN_ERR]);
    return GPMA_OK;
}

// The graph's analytics buffer: 5 arrays of row_num words, one word per CTA,
// then the control words.
size_t an_cta_words(const gpma_graph *g) { return (size_t)g->sms * AN_MAX_FIT; }
gpma_status an_buffers(gpma_graph *g, uint32_t **base, uint32_t **ctl) {
    const uint32_t n = g->row_num;
    if (!g->an_buf || g->an_cap < n) {
        dev_free(g->an_buf);
        g->an_cap = 0;
        GPMA_TRY(dev_alloc(&g->an_buf, 5ull * n + an_cta_words(g) + AN_ALL + BAR_ALIGN_WORDS));
        g->an_cap = n;
    }
    *base = g->an_buf;
    // on a line of their own, as the barrier among them wants
    *ctl = g->an_buf + ((5ull * n + an_cta_words(g) + BAR_ALIGN_WORDS - 1) & ~uint64_t(BAR_ALIGN_WORDS - 1));
    return GPMA_OK;
}

// The gathering's sweeps take whole groups of 8 slots. It pays in the smallest arrays
// too (256 slots, 4 / 20 iterations: 90 / 250 us, by atomics 114 / 413).
constexpr uint32_t PR_GATHER_MIN_SLOTS = 8;

}  // namespace
}  // namespace gpma

using namespace gpma;

extern "C" {

gpma_status gpma_pagerank(gpma_graph *g, float damping, uint32_t iterations, double tol, float *ranks,
                          uint32_t *iterations_run, void *stream) {
    CallRange range("gpma_pagerank");
    if (!g || !ranks || !(damping >= 0.0f && damping <= 1.0f) || g->row_num == 0) {
        set_error("gpma_pagerank: bad arguments (damping in [0, 1], a graph with nodes, an output array)");
        return GPMA_ERR_INVALID;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t n = g->row_num;
    uint32_t h_ctl[AN_WORDS];
    gpma_status st = [&]() -> gpma_status {
        uint32_t *base = nullptr, *ctl = nullptr;
        GPMA_TRY(an_buffers(g, &base, &ctl));
        GPMA_CUDA(cudaMemsetAsync(ctl, 0, sizeof(uint32_t) * AN_ALL, s));
        AnArgs A{};
        A.keys = g->keys;
        A.vals = g->values;
        A.n = n;
        A.size = g->geo.size;
        A.deg = base;
        float *rank = A.rank = reinterpret_cast<float *>(base + n);
        A.acc = reinterpret_cast<float *>(base + 2ull * n);
        A.contrib = reinterpret_cast<float *>(base + 3ull * n);
        A.end = base + 4ull * n;
        A.cta = base + 5ull * n;
        A.ctl = ctl;
        A.damping = damping;
        A.tol = tol;
        A.max_iter = iterations;
        const bool gather = iterations >= PR_GATHER_ITERATIONS && g->geo.size >= PR_GATHER_MIN_SLOTS;
        if (gather) {
            // the in-edges in the graph's window scratch (8 bytes per slot,
            // idle between updates): the sources in its first half, then, a
            // row of more than PR_SHORT edges having one chunk per PR_CHUNK
            // of them at most, up to size / PR_SHORT chunks (16 bytes) and
            // size / PR_CHUNK rows of several (8 bytes)
            static_assert(16 <= 2 * PR_SHORT && 8 <= 2 * PR_CHUNK, "chunk lists exceed the scratch");
            GPMA_TRY(ensure_scratch(g, g->geo.size));
            A.csc = reinterpret_cast<uint32_t *>(g->skeys);
            A.chunks = reinterpret_cast<uint4 *>(A.csc + g->geo.size);
            A.multi = reinterpret_cast<uint2 *>(A.csc + g->geo.size + g->geo.size / 2);
        }
        prof_mark(g, 0, s);
        GPMA_TRY(launch(!gather ? AN_PAGERANK : tol > 0.0 ? AN_PAGERANK_TOL : AN_PAGERANK_GATHER, A, g->sms, s, h_ctl));
        prof_mark(g, 1, s);
        GPMA_TRY(copy_any(ranks, rank, sizeof(float) * n, s));
        GPMA_CUDA(cudaStreamSynchronize(s));
        g->prof.kernel_launches += 1;
        if (iterations_run)
            *iterations_run = h_ctl[AN_ITERS];
        return GPMA_OK;
    }();
    return st;
}

gpma_status gpma_components(gpma_graph *g, uint32_t *labels, uint64_t *components, uint32_t *rounds, void *stream) {
    CallRange range("gpma_components");
    if (!g || !labels) {
        set_error("gpma_components: null argument");
        return GPMA_ERR_INVALID;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t n = g->row_num;
    if (n == 0) {
        if (components)
            *components = 0;
        return GPMA_OK;
    }
    uint32_t h_ctl[AN_WORDS];
    gpma_status st = [&]() -> gpma_status {
        uint32_t *base = nullptr, *ctl = nullptr;
        GPMA_TRY(an_buffers(g, &base, &ctl));
        uint32_t *parent = base;
        GPMA_CUDA(cudaMemsetAsync(ctl, 0, sizeof(uint32_t) * AN_ALL, s));
        AnArgs A{};
        A.keys = g->keys;
        A.vals = g->values;
        A.ro = g->row_offset;
        A.n = n;
        A.size = g->geo.size;
        A.parent = parent;
        A.ctl = ctl;
        GPMA_TRY(launch(AN_COMPONENTS, A, g->sms, s, h_ctl));
        GPMA_TRY(copy_any(labels, parent, sizeof(uint32_t) * n, s));
        GPMA_CUDA(cudaStreamSynchronize(s));
        if (components)
            *components = h_ctl[AN_ROOTS];
        if (rounds)
            *rounds = h_ctl[AN_ITERS];
        g->prof.kernel_launches += 1;
        return GPMA_OK;
    }();
    return st;
}

}  // extern "C"
