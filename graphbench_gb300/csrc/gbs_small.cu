// gbs_small.cu -- shortest paths of small graphs on one CTA (sm_103a).
//
// What bounds a small graph is the chain of dependent phases, not its edges:
// in the persistent kernel a phase of a few hundred entries is a chain of
// about eight L2 round trips (list, distance, row, edges, target distance,
// three atomics), 4-10 us, and an R-MAT of 1,024 vertices takes 50 of them.
// Here the distances, the frontier and the queued sets of the whole graph sit
// in the shared memory of one CTA, so a sweep is one global round trip (the
// edges, which L1 or L2 holds) and a few shared-memory ones.
//
//   dist[n]   uint32 distance bits (float32 bits order like the values);
//             0xFFFFFFFF unreached
//   near      one bit per vertex: below `hi` and improved since it was relaxed
//   far       one bit per vertex: improved to `hi` or beyond (a vertex that
//             drops below `hi` later keeps its bit; the next advance clears it)
//   queue[n]  this sweep's vertices (the near bits, compacted)
//   pieces    long rows of this sweep in pieces of kPiece edges, so a hub's row
//             is shared by all warps
//   pred[n]   written after the search: the smallest u with dist[u] + w(u, v)
//             == dist[v], over every edge of every reached vertex
//
// A sweep relaxes every near vertex; when none is left `hi` moves past the
// smallest far distance by `width`.  Any width gives the same least fixpoint.
// 32-bit shared-memory atomicMin is one instruction, a 64-bit one (distance
// and predecessor together, as the persistent kernel keeps them) a
// compare-and-swap loop, so predecessors take a pass over the edges at the end.
#include <algorithm>
#include <cstring>

#include "gbs_small.cuh"

namespace gbs {
namespace {

constexpr uint32_t kFar = 0xFFFFFFFFu;      // unreached
constexpr unsigned kAll = 0xffffffffu;
// Edges of one piece of a long row: shorter pieces spread a hub better over the
// warps, longer ones cost fewer row reads.  R-MAT of 8,192 vertices, kernel us:
// 256 217, 128 203, 64 235.
constexpr uint32_t kPiece = 128;
constexpr size_t kSmallBytes = 200u << 10;  // most dynamic shared memory a launch asks for
// Threads of a CTA, one CTA per SM.  Two of 512 hold more instances at once
// but each takes 1.5x as long and the largest sets a plan's time: pack of 256
// graphs of 1,024..8,192 vertices 288 us with 1024 threads, 335 with 768, 464
// with 512.
constexpr int kSmallTPB = 1024;
// The graphs solved here.  Beyond kSmallM edges (kSmallBatchM in a plan, whose
// other SMs work on other instances) one SM's instruction rate outweighs the
// phases it saves.  Persistent kernel -> one CTA, us: one source of an R-MAT of
// 1,024 vertices 262 -> 74 a call, 4,096 (97 K edges) 330 -> 151, 8,192 (204 K)
// 360 -> 229, 16,384 (427 K) 394 -> 414; 64 sources of the last 642 -> 450,
// pack of 256 730 -> 288; 64 x 100 grid 584 -> 237, 110 x 140 877 -> 404.
constexpr uint32_t kSmallN = 16384;
constexpr uint64_t kSmallM = 262144;
constexpr uint64_t kSmallBatchM = 524288;
// A graph whose default width is kWideRatio mean weights or more (unit weights,
// few distinct ones, skewed ones) takes a handful of buckets, which the grid
// shares well: beyond kSmallWideM edges it is left to the persistent kernel
// where one CTA is slower.  Persistent kernel before buckets merged -> one CTA,
// us a call: unit weights, 131,072 edges 88..149 -> 84..119, 196,608 76..101 ->
// 83..118, 262,144 77..166 -> 99..168; lognormal (sigma 3), 131,072 250..480 ->
// 190..350, 262,144 247, 261, 458 -> 359, 371, 501.  Weights 1 to 255 at 0.02 to
// 0.25 widths a mean weight: 262,144 edges 298..864 -> 110..241.
constexpr uint64_t kSmallWideM = 131072;
constexpr double kWideRatio = 0.28;
// In a plan that holds up to a number of instances, whose CTAs fill the other
// SMs from there on: kWideStep, one step more beyond kSmallM edges and one more
// on graphs that are not skewed (largest weight at most kSkew mean weights).
// Beyond kSmallM edges it holds for every skewed graph.  Persistent kernel before
// buckets merged -> one CTA, us a plan of 1, 16, 64: unit weights, 4,096 vertices
// and 262,144 edges 77, 93, 171 -> 128, 128, 130, 520,000 75, 104, 222 -> 236,
// 247, 247 (152 of them 370 -> 252); lognormal (sigma 2), 262,144 211, 315, 673 ->
// 305, 329, 343 (sigma 3, 16,384 vertices, 32 of them: 823 -> 605); exponential,
// 520,000 402, 494, 846 -> 590, 608, 649.
constexpr uint32_t kWideStep = 32;
constexpr double kSkew = 4.0;
// Default widths one bucket spans.  Sweeps are short, so wide buckets pay;
// graphs of few edges a vertex, whose frontier stays thin, hardly repeat work
// at any width (64 x 100 grid, kernel us: 4 310, 8 254, 64 215).  R-MAT of
// 8,192 vertices: 1 267, 4 217, 8 203, 64 243; a pack keeps every SM busy and
// repeats less at 4 (256 graphs: 2 284, 4 288, 8 304).
constexpr uint32_t kScale = 8, kScaleBatch = 4, kScaleSparse = 64;
constexpr uint32_t kSparse = 8;             // average degree up to which kScaleSparse holds

uint32_t words_of(uint32_t n) { return (n + 31u) / 32u; }

__host__ __device__ inline uint32_t width_scale(uint32_t n, uint64_t m, bool batch) {
    return m <= (uint64_t)kSparse * n ? kScaleSparse : batch ? kScaleBatch : kScale;
}

struct RowSlot;
struct Small {
    // graph
    const uint32_t *row;
    const uint2 *adj;
    uint32_t n, words, src;
    uint32_t width;        // uint32 width or float32 bits
    // shared memory
    uint32_t *dist, *pred, *near, *far, *pieces;
    uint16_t *queue;
    RowSlot *slots;  // 32 per warp
    uint32_t *qn, *hn, *lo; // double-buffered counters of the sweeps and advances
    uint32_t hi;
};

template <bool F32>
__device__ __forceinline__ uint32_t add_bits(uint32_t d, uint32_t w) {
    if (F32) return __float_as_uint(__fadd_rn(__uint_as_float(d), __uint_as_float(w)));
    return d + w;   // the caller has ruled out sums of 2^32 - 1 and more
}

// The next bound past the smallest far distance; always above it.
template <bool F32>
__device__ __forceinline__ uint32_t advance_bits(uint32_t d, uint32_t width) {
    if (F32) return max(add_bits<true>(d, width), d + 1u);
    return d > kFar - width ? kFar : d + width;
}

// One edge u -> v.  Relaxing: lowers dist[v] and queues v.  Predecessors: u
// is a candidate of v if the edge is tight.
template <bool F32, bool Pred>
__device__ __forceinline__ void small_edge(const Small &s, uint32_t u, uint32_t du, uint2 e, uint32_t &imp) {
    const uint32_t v = e.x, d = add_bits<F32>(du, e.y);
    if (Pred) {
        if (d == s.dist[v] && v != s.src && u < s.pred[v]) atomicMin(s.pred + v, u);
        return;
    }
    if (d >= s.dist[v]) return;
    if (d >= atomicMin(s.dist + v, d)) return;
    ++imp;
    const uint32_t bit = 1u << (v & 31u);
    uint32_t *set = (d < s.hi ? s.near : s.far) + (v >> 5);
    if (!(*reinterpret_cast<volatile uint32_t *>(set) & bit)) atomicOr(set, bit);
}

// The non-empty rows of a chunk of up to 32 vertices, in lane order.
struct RowSlot {
    uint32_t at;    // first edge minus the edges of the chunk's earlier rows
    uint32_t du, u;
};

// Edges [k0, k0 + 32 U) of a chunk's `total`, U per lane, all loads before any
// is used.  What bounds the solver is instructions per edge (one SM), so the
// row an edge belongs to is found without a search: a bit per row start in
// each window of 32 edges, one warp reduction, a population count.
template <bool F32, bool Pred, int U>
__device__ __forceinline__ void small_round(const Small &s, const RowSlot *slot, uint32_t start, uint32_t total,
                                            uint32_t k0, uint32_t &before, uint32_t &imp) {
    const uint32_t lane = lane_id(), upto = (2u << lane) - 1u;
    uint2 e[U];
    uint32_t own[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
        const uint32_t off = start - (k0 + 32u * j);
        const uint32_t starts = __reduce_or_sync(kAll, off < 32u ? 1u << off : 0u);
        own[j] = before + (uint32_t)__popc(starts & upto) - 1u;
        before += (uint32_t)__popc(starts);
        const uint32_t k = k0 + 32u * j + lane;
        // at + k wraps back to the edge where the row begins before the chunk's earlier edges
        const uint32_t at = k < total ? slot[own[j]].at + k : 0u;
        e[j] = k < total ? __ldg(s.adj + at) : make_uint2(kFar, 0u);
    }
#pragma unroll
    for (int j = 0; j < U; ++j)
        if (e[j].x != kFar) small_edge<F32, Pred>(s, Pred ? slot[own[j]].u : 0u, slot[own[j]].du, e[j], imp);
}

// The first `count` vertices of the queue (Pred: all vertices), a chunk of up
// to 32 per warp.  Rows longer than kPiece become pieces.
template <bool F32, bool Pred>
__device__ __forceinline__ void small_vertices(const Small &s, uint32_t *hn, uint32_t count, uint32_t &imp) {
    const uint32_t warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5, lane = lane_id();
    RowSlot *slot = s.slots + warp * 32u;
    uint32_t deal = (count + nwarps - 1u) / nwarps;
    if (deal > 32u) deal = 32u;
    for (uint32_t base = warp * deal; base < count; base += nwarps * deal) {
        uint32_t u = 0, du = 0, beg = 0, len = 0;
        if (lane < deal && base + lane < count) {
            u = Pred ? base + lane : s.queue[base + lane];
            du = *reinterpret_cast<volatile uint32_t *>(s.dist + u);
            beg = __ldg(s.row + u);
            len = Pred && du == kFar ? 0u : __ldg(s.row + u + 1) - beg;
            if (len > kPiece) {
                const uint32_t np = (len + kPiece - 1u) / kPiece, at = atomicAdd(hn, np);
                for (uint32_t q = 0; q < np; ++q) s.pieces[at + q] = u | (q << 16);
                len = 0;
            }
        }
        uint32_t incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, incl, o);
            if ((int)lane >= o) incl += y;
        }
        const uint32_t total = __shfl_sync(kAll, incl, 31), excl = incl - len;
        const unsigned rows = __ballot_sync(kAll, len != 0u);
        if (len) slot[__popc(rows & ((1u << lane) - 1u))] = RowSlot{beg - excl, du, u};
        __syncwarp();
        const uint32_t start = len ? excl : kFar;
        uint32_t before = 0, k0 = 0;
        for (; k0 + 32u < total; k0 += 128u) small_round<F32, Pred, 4>(s, slot, start, total, k0, before, imp);
        if (k0 < total) small_round<F32, Pred, 1>(s, slot, start, total, k0, before, imp);
        __syncwarp();
    }
}

// The pieces of the sweep's long rows, a warp each.
template <bool F32, bool Pred>
__device__ __forceinline__ void small_pieces(const Small &s, uint32_t count, uint32_t &imp) {
    const uint32_t nwarps = blockDim.x >> 5, lane = lane_id();
    for (uint32_t i = threadIdx.x >> 5; i < count; i += nwarps) {
        const uint32_t p = s.pieces[i], u = p & 0xFFFFu;
        const uint32_t du = *reinterpret_cast<volatile uint32_t *>(s.dist + u);
        const uint32_t beg = __ldg(s.row + u) + (p >> 16) * kPiece;
        const uint32_t end = min(__ldg(s.row + u + 1), beg + kPiece);
        uint2 e[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t k = beg + 32u * j + lane;
            e[j] = k < end ? __ldg(s.adj + k) : make_uint2(kFar, 0u);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (e[j].x != kFar) small_edge<F32, Pred>(s, u, du, e[j], imp);
    }
}

// The result words of a run, from the whole CTA.
struct SmallCounts {
    unsigned long long reached, edges, imp;
    uint32_t buckets, sweeps;
};

// Solves one instance.  Every thread of the CTA calls it; c is filled in
// thread 0.  s.dist .. s.lo point into shared memory.
template <bool F32>
__device__ void small_solve(Small &s, uint32_t *dist_out, int32_t *pred_out, unsigned long long *s_sum, SmallCounts &c) {
    const uint32_t tid = threadIdx.x, T = blockDim.x, lane = lane_id(), warp = tid >> 5, nwarps = T >> 5;
    for (uint32_t v = tid; v < s.n; v += T) s.dist[v] = v == s.src ? 0u : kFar;
    for (uint32_t w = tid; w < s.words; w += T) {
        s.near[w] = w == (s.src >> 5) ? 1u << (s.src & 31u) : 0u;
        s.far[w] = 0u;
    }
    if (tid < 2) s.qn[tid] = s.hn[tid] = 0u, s.lo[tid] = kFar;
    if (tid < 3) s_sum[tid] = 0ull;
    s.hi = advance_bits<F32>(0u, s.width);
    uint32_t imp = 0, sweeps = 0, buckets = 1, parity = 0;
    __syncthreads();
    for (;;) {
        // the near vertices, compacted
        for (uint32_t w = tid; w < s.words; w += T) {
            uint32_t bits = s.near[w];
            if (!bits) continue;
            s.near[w] = 0u;
            uint32_t at = atomicAdd(s.qn + parity, (uint32_t)__popc(bits));
            for (; bits; bits &= bits - 1u) s.queue[at++] = (uint16_t)(w * 32u + (uint32_t)__ffs(bits) - 1u);
        }
        __syncthreads();
        const uint32_t count = s.qn[parity];
        if (tid == 0) s.qn[parity ^ 1u] = s.hn[parity ^ 1u] = 0u;
        if (count == 0u) {
            // no near vertex left: the smallest far distance bounds the next bucket
            uint32_t *lo = s.lo + (buckets & 1u);
            uint32_t m = kFar;
            for (uint32_t w = warp; w < s.words; w += nwarps) {
                const uint32_t bits = s.far[w];
                if (!bits) continue;
                const uint32_t d = ((bits >> lane) & 1u) ? s.dist[w * 32u + lane] : 0u;
                const uint32_t live = __ballot_sync(kAll, d >= s.hi);   // the others were relaxed since
                if (lane == 0) s.far[w] = live;
                if (d >= s.hi) m = min(m, d);
            }
            m = __reduce_min_sync(kAll, m);
            if (lane == 0 && m != kFar) atomicMin(lo, m);
            __syncthreads();
            m = *lo;
            if (m == kFar) break;
            if (tid == 0) s.lo[(buckets & 1u) ^ 1u] = kFar;
            s.hi = advance_bits<F32>(m, s.width);
            for (uint32_t w = warp; w < s.words; w += nwarps) {
                const uint32_t bits = s.far[w];
                if (!bits) continue;
                const bool in = ((bits >> lane) & 1u) && s.dist[w * 32u + lane] < s.hi;
                const uint32_t take = __ballot_sync(kAll, in);
                if (lane == 0 && take) {
                    s.near[w] = take;
                    s.far[w] = bits & ~take;
                }
            }
            ++buckets;
            parity ^= 1u;
            __syncthreads();
            continue;
        }
        ++sweeps;
        small_vertices<F32, false>(s, s.hn + parity, count, imp);
        __syncthreads();
        const uint32_t pieces = s.hn[parity];
        if (pieces) {
            small_pieces<F32, false>(s, pieces, imp);
            __syncthreads();
        }
        parity ^= 1u;
    }
    // here qn and hn of the other parity are zero, and every thread sees the final distances
    if (pred_out) {
        uint32_t *hn = s.hn + (parity ^ 1u);
        for (uint32_t v = tid; v < s.n; v += T) s.pred[v] = 0x7FFFFFFFu;
        __syncthreads();
        small_vertices<F32, true>(s, hn, s.n, imp);
        __syncthreads();
        const uint32_t pieces = *hn;
        if (pieces) small_pieces<F32, true>(s, pieces, imp);
        __syncthreads();
    }
    unsigned long long reached = 0, edges = 0, im = imp;
    for (uint32_t v = tid; v < s.n; v += T) {
        const uint32_t d = s.dist[v];
        const bool ok = d != kFar;
        if (dist_out) dist_out[v] = ok ? d : (F32 ? 0x7F800000u : kFar);
        if (pred_out) pred_out[v] = ok ? (v == s.src ? (int32_t)v : (int32_t)s.pred[v]) : -1;
        if (ok) {
            ++reached;
            edges += __ldg(s.row + v + 1) - __ldg(s.row + v);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        reached += __shfl_down_sync(kAll, reached, o);
        edges += __shfl_down_sync(kAll, edges, o);
        im += __shfl_down_sync(kAll, im, o);
    }
    if (lane == 0) {
        atomicAdd(s_sum + 0, reached);
        atomicAdd(s_sum + 1, edges);
        atomicAdd(s_sum + 2, im);
    }
    __syncthreads();
    if (tid == 0) c = SmallCounts{s_sum[0], s_sum[1], s_sum[2], buckets, sweeps};
}

__device__ __forceinline__ void carve_small(Small &s, unsigned char *mem, uint32_t n_cap) {
    const uint32_t words = (n_cap + 31u) / 32u;
    s.dist = reinterpret_cast<uint32_t *>(mem);
    s.pred = s.dist + n_cap;
    s.near = s.pred + n_cap;
    s.far = s.near + words;
    s.pieces = s.far + words;
}

template <bool F32>
__global__ void __launch_bounds__(kSmallTPB, 1) sssp_small(const uint32_t *row, const uint2 *adj, uint32_t n,
                                                           uint32_t src, uint32_t width, uint32_t n_cap,
                                                           uint32_t piece_cap, uint32_t *dist_out, int32_t *pred_out,
                                                           InstResult *res) {
    extern __shared__ __align__(16) unsigned char mem[];
    __shared__ uint32_t s_ctr[6];
    __shared__ RowSlot s_slots[kSmallTPB];
    __shared__ unsigned long long s_sum[3];
    Small s;
    carve_small(s, mem, n_cap);
    s.queue = reinterpret_cast<uint16_t *>(s.pieces + piece_cap);
    s.slots = s_slots;
    s.qn = s_ctr;
    s.hn = s_ctr + 2;
    s.lo = s_ctr + 4;
    s.row = row;
    s.adj = adj;
    s.n = n;
    s.words = (n + 31u) / 32u;
    s.src = src;
    s.width = width;
    SmallCounts c;
    small_solve<F32>(s, dist_out, pred_out, s_sum, c);
    if (threadIdx.x == 0) {
        res->done = 1u;
        res->phases = c.sweeps;
        res->buckets = c.buckets;
        res->reached = c.reached;
        res->edges_reached = c.edges;
        res->improvements = c.imp;
    }
}

template <bool F32>
__global__ void __launch_bounds__(kSmallTPB, 1) sssp_small_batch(const InstDesc *__restrict__ inst,
                                                                      InstResult *__restrict__ out, uint32_t count,
                                                                      uint32_t *queue, uint32_t n_cap,
                                                                      uint32_t piece_cap) {
    extern __shared__ __align__(16) unsigned char mem[];
    __shared__ uint32_t s_ctr[6], s_inst;
    __shared__ RowSlot s_slots[kSmallTPB];
    __shared__ unsigned long long s_sum[3];
    Small s;
    carve_small(s, mem, n_cap);
    s.queue = reinterpret_cast<uint16_t *>(s.pieces + piece_cap);
    s.slots = s_slots;
    s.qn = s_ctr;
    s.hn = s_ctr + 2;
    s.lo = s_ctr + 4;
    for (;;) {
        __syncthreads();   // the last instance's shared state has been read
        if (threadIdx.x == 0) s_inst = atomicAdd(queue, 1u);
        __syncthreads();
        const uint32_t i = s_inst;
        if (i >= count) return;
        const unsigned long long t0 = globaltimer();
        const InstDesc d = inst[i];
        s.row = d.g.row;
        s.adj = d.g.adj;
        s.n = d.g.n;
        s.words = (d.g.n + 31u) / 32u;
        s.src = d.source;
        const uint32_t scale = width_scale(d.g.n, d.g.m, true);
        s.width = F32 ? __float_as_uint(__fdiv_rn((float)scale, d.inv_delta_f))
                      : (uint32_t)min((unsigned long long)d.delta_u * scale, 0xFFFFFFFFull);
        SmallCounts c;
        small_solve<F32>(s, d.dist, d.pred, s_sum, c);
        if (threadIdx.x == 0) {
            InstResult r;
            r.done = 1u;
            r.error = 0u;
            r.group = blockIdx.x;
            r.phases = c.sweeps;
            r.buckets = c.buckets;
            r.pending_scans = 0u;
            r.solo_phases = c.sweeps;
            r.pad = 0u;
            r.reached = c.reached;
            r.edges_reached = c.edges;
            r.improvements = c.imp;
            r.start_ns = t0;
            r.end_ns = globaltimer();
            out[i] = r;
        }
    }
}

const void *kernel_of(bool f32, bool batch) {
    if (batch) return f32 ? (const void *)sssp_small_batch<true> : (const void *)sssp_small_batch<false>;
    return f32 ? (const void *)sssp_small<true> : (const void *)sssp_small<false>;
}

}  // namespace

SmallShape small_shape(uint32_t n, uint64_t m) {
    SmallShape s{};
    s.n_cap = (n + 31u) & ~31u;
    // a row of more than kPiece edges has at most twice its share of pieces
    s.piece_cap = (uint32_t)(2u * (m / kPiece) + 1u);
    s.bytes = 4ull * s.n_cap * 2u + 4ull * words_of(s.n_cap) * 2u + 4ull * s.piece_cap + 2ull * s.n_cap;
    return s;
}

bool small_call(const gbs_graph *g, const gbs_params *p) {
    if (!small_graph(g->wtype, g->n, g->m, g->max_w, g->mean_w, 0)) return false;
    if (!p) return true;
    if ((p->flags & ~GBS_F_NO_STATS) || p->solo_entries || p->solo_descs || p->inline_edges || p->full_items ||
        p->fuse_rounds)
        return false;
    return !(p->delta > 0) || resolve_schedule(g->wtype, g->max_w, g->n, g->m, p->delta, -1.0).delta ==
                                  resolve_schedule(g->wtype, g->max_w, g->n, g->m, 0.0, -1.0).delta;
}

bool small_graph(gbs_weight_type wt, uint32_t n, uint64_t m, double max_w, double mean_w, uint32_t instances) {
    if (n == 0 || n > kSmallN || m > (instances ? kSmallBatchM : kSmallM)) return false;
    if (small_shape(n, m).bytes > kSmallBytes) return false;
    if (m > kSmallWideM) {
        const bool wide = resolve_schedule(wt, max_w, n, m, 0.0, -1.0).delta >= kWideRatio * mean_w;
        const bool large = m > kSmallM, skewed = max_w > kSkew * mean_w;
        const uint32_t least = kWideStep * (1u + (large ? 1u : 0u) + (skewed ? 0u : 1u));
        if ((wide || (large && skewed)) && instances < least) return false;
    }
    if (wt == GBS_WEIGHT_U32) return (double)n * max_w < 4294967295.0;
    return wt == GBS_WEIGHT_F32;
}

uint32_t small_grid(bool f32, const SmallShape &shape, int sms, uint32_t count) {
    int per_sm = 0;
    const void *k = kernel_of(f32, true);
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmallBytes) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kSmallTPB, shape.bytes) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return std::min<uint32_t>((uint32_t)(per_sm * sms), count);
}

gbs_status small_launch(bool f32, const SmallShape &shape, uint32_t grid, const InstDesc *inst, InstResult *res,
                        uint32_t count, uint32_t *queue, cudaStream_t s) {
    if (f32)
        sssp_small_batch<true><<<grid, kSmallTPB, shape.bytes, s>>>(inst, res, count, queue, shape.n_cap,
                                                                         shape.piece_cap);
    else
        sssp_small_batch<false><<<grid, kSmallTPB, shape.bytes, s>>>(inst, res, count, queue, shape.n_cap,
                                                                          shape.piece_cap);
    GBS_CUDA(cudaGetLastError());
    return GBS_OK;
}

gbs_status small_run(gbs_graph *g, uint32_t src, void *dist, int32_t *pred, double light, bool want_stats,
                     gbs_stats *stats) {
    if (src >= g->n) return fail(GBS_ERR_INVALID_ARG, "source out of range");
    const SmallShape shape = small_shape(g->n, g->m);
    const bool f32 = g->wtype == GBS_WEIGHT_F32;
    if (!g->h_small) {
        GBS_CUDA(cudaMallocHost(&g->h_small, sizeof(InstResult)));
        GBS_CUDA(cudaFuncSetAttribute(kernel_of(f32, false), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)kSmallBytes));
    }
    const Resolved r = resolve_schedule(g->wtype, g->max_w, g->n, g->m, 0.0, light);
    double wide = r.delta * width_scale(g->n, g->m, false);
    uint32_t width;
    if (f32) {
        const float w = (float)wide;
        std::memcpy(&width, &w, 4);
    } else {
        wide = std::min(wide, 4294967295.0);
        width = (uint32_t)wide;
    }
    GBS_CUDA(cudaEventRecord(g->ev[0], g->stream));
    if (f32)
        sssp_small<true><<<1, kSmallTPB, shape.bytes, g->stream>>>(g->d_row, g->d_adj, g->n, src, width, shape.n_cap,
                                                                   shape.piece_cap, static_cast<uint32_t *>(dist),
                                                                   pred, g->h_small);
    else
        sssp_small<false><<<1, kSmallTPB, shape.bytes, g->stream>>>(g->d_row, g->d_adj, g->n, src, width, shape.n_cap,
                                                                    shape.piece_cap, static_cast<uint32_t *>(dist),
                                                                    pred, g->h_small);
    GBS_CUDA(cudaGetLastError());
    GBS_CUDA(cudaEventRecord(g->ev[1], g->stream));
    GBS_CUDA(cudaStreamSynchronize(g->stream));
    g->trace_n = g->feat_n = 0;   // as after any run that recorded neither
    if (stats) {
        const InstResult &x = *g->h_small;
        float ms = 0.f;
        std::memset(stats, 0, sizeof(*stats));
        GBS_CUDA(cudaEventElapsedTime(&ms, g->ev[0], g->ev[1]));
        stats->device_ms = stats->kernel_ms = ms;
        stats->reached = want_stats ? x.reached : 0;
        stats->edges_reached = want_stats ? x.edges_reached : 0;
        stats->improvements = x.improvements;
        stats->buckets = x.buckets;
        stats->phases = stats->solo_phases = x.phases;
        stats->blocks = 1u;
        stats->delta_used = wide;
        stats->light_used = r.light;
    }
    return GBS_OK;
}

}  // namespace gbs
