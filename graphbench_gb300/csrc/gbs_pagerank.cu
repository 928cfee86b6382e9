// gbs_pagerank.cu -- PageRank on the GPU (sm_103a): the reference's iteration
// (pagerank/pagerank_mpi.c:667-1043, one node, constants RDM_JMP and THRESH
// of include/graph.h:17-18) as a pull over the in-edge CSR, replacing the MPI
// message exchange.
//
//   weight = 1, recip = 1 / out-degree, wb = rj, diff = weight * recip
//   per iteration:  wb[v] += sum over in-edges u of (1 - rj) * diff[u]
//                   diff'[v] = (wb[v] - weight[v]) * recip[v]
//                   weight[v] = wb[v]; stop when no |diff'| exceeds thresh
//
// diff is double-buffered (iteration t reads t-1's); after the first iteration
// wb and weight hold the same number, so one array stands for both.  The
// per-iteration sum of a row has a fixed order shared with the oracle: the
// row's CSR positions in 32-position words, each word summed from its lowest
// position up, the word sums of each block of 32 words combined by a butterfly,
// the block sums added in order.
//
// Rows of at most 32 edges (two words) are summed by one thread (their
// butterfly is the plain sum of the two word sums); the words of longer rows are
// summed one per thread into a buffer, and a second kernel combines them (a
// thread per row of up to kMid words, with a shorter chain for those of up to
// kFew, a warp per longer row).
//
// What bounds the pull is the load unit, which looks up one cache line per
// clock: the gather of an edge's diff is a line of its own whatever the order,
// and a thread that reads its word's columns one by one takes another for each.
// Columns are therefore read four at a time (aligned groups, masked at the
// ends).  Coalesced column reads through shared memory, with a word summed per
// lane afterwards, were slower (335 us an iteration): fewer lookups, but the
// 32 dependent adds of a word (55 cycles each) then run with nothing in flight.
//
// Rows are put into classes on the device (one per degree up to 32, rows of up
// to kFew words, of up to kMid, longer ones).  Iterations are enqueued kAhead at
// a time: each leaves a word that says whether some |diff'| exceeded thresh, the
// kernels of the next return at once where it does not, and the host reads the
// words back once per batch.  R-MAT of 1,048,576 vertices and 31 M edges: the
// pull 0.220 -> 0.178 ms an iteration, the call 18.6 -> 7.1 ms.
#include <algorithm>
#include <cmath>
#include <vector>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "gbs_host.hpp"

namespace gbs {
namespace {

constexpr uint32_t kShort = 32;   // rows up to this many edges are summed by one thread

// Long rows of up to kFew or kMid words are combined by one thread (31 adds
// for a block of 32; a warp's butterfly runs 5 x 32), longer ones by a warp.
constexpr uint32_t kFew = 8, kMid = 32;
constexpr uint32_t kClasses = kShort + 4;       // rows by degree 0..kShort, of at most kFew words, kMid words, longer
constexpr uint32_t kClsFew = kShort + 1, kClsMid = kShort + 2, kClsBig = kShort + 3;
constexpr int kPrTPB = 256;
constexpr uint32_t kAhead = 8;    // iterations enqueued between two looks at their flags

struct PrArgs {
    const unsigned long long *row;
    const uint32_t *col;
    unsigned long long m;
    double pj;          // 1 - random jump
    double rj;
    double thresh;
    const double *recip;
    double *weight;
    const double *diff;     // this iteration's input, times (1 - rj)
    double *diff_next;      // its output, times (1 - rj)
    const uint32_t *srow;    // the rows of at most kShort edges, grouped by degree
    uint32_t n_short;
    const uint2 *lw;         // words of the long rows: row, mask word
    uint32_t n_lw, lw_blocks;
    double *part;            // one sum per long-row word
    const uint32_t *lr_row;  // long rows: those of at most kFew words, of at most kMid, the others
    const uint2 *lr_words;   // their first word and number of words
    uint32_t n_few, n_mid, n_big;
    uint32_t big_blocks, mid_blocks;
    bool first;              // first iteration: wb = rj, weight = 1
    const uint32_t *run;     // zero: the iteration before this one was the last
    uint32_t *flag;          // set when some |diff'| > thresh
};

// Rows of every class, and words of the long rows.
struct PrCounts {
    uint32_t rows[kClasses];
    uint32_t words;
};

__device__ __forceinline__ uint32_t words_of(unsigned long long beg, unsigned long long end) {
    return (uint32_t)(((end + 31ull) >> 5) - (beg >> 5));
}
__device__ __forceinline__ uint32_t class_of(unsigned long long beg, unsigned long long end) {
    if (end - beg <= kShort) return (uint32_t)(end - beg);
    const uint32_t w = words_of(beg, end);
    return w <= kFew ? kClsFew : w <= kMid ? kClsMid : kClsBig;
}

__global__ void __launch_bounds__(256) k_pr_count(const unsigned long long *__restrict__ row, uint32_t n,
                                                  PrCounts *cnt) {
    __shared__ uint32_t s[kClasses + 1];
    for (uint32_t i = threadIdx.x; i <= kClasses; i += blockDim.x) s[i] = 0u;
    __syncthreads();
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const unsigned long long beg = row[v], end = row[v + 1];
        const uint32_t c = class_of(beg, end);
        atomicAdd(s + c, 1u);
        if (c >= kClsFew) atomicAdd(s + kClasses, words_of(beg, end));
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i <= kClasses; i += blockDim.x)
        if (s[i]) atomicAdd(i < kClasses ? cnt->rows + i : &cnt->words, s[i]);
}

// Every row at its class's place (`at` counts up from the class's first), the
// words of long rows listed.  The order inside a class is arbitrary: a row's
// sum does not depend on it.
__global__ void __launch_bounds__(256) k_pr_place(const unsigned long long *__restrict__ row, uint32_t n, PrCounts *at,
                                                  uint32_t n_short, uint32_t *__restrict__ list,
                                                  uint2 *__restrict__ lr_words, uint2 *__restrict__ lw) {
    __shared__ uint32_t s[kClasses + 1], base[kClasses + 1];
    const unsigned lane = threadIdx.x & 31u;
    for (uint32_t v0 = blockIdx.x * blockDim.x; v0 < n; v0 += gridDim.x * blockDim.x) {
        for (uint32_t i = threadIdx.x; i <= kClasses; i += blockDim.x) s[i] = 0u;
        __syncthreads();
        const uint32_t v = v0 + threadIdx.x;
        unsigned long long beg = 0;
        uint32_t c = 0, rank = 0, nw = 0, wrank = 0;
        if (v < n) {
            const unsigned long long end = row[v + 1];
            beg = row[v];
            c = class_of(beg, end);
            rank = atomicAdd(s + c, 1u);
            if (c >= kClsFew) {
                nw = words_of(beg, end);
                wrank = atomicAdd(s + kClasses, nw);
            }
        }
        __syncthreads();
        for (uint32_t i = threadIdx.x; i <= kClasses; i += blockDim.x)
            base[i] = s[i] ? atomicAdd(i < kClasses ? at->rows + i : &at->words, s[i]) : 0u;
        __syncthreads();
        const uint32_t w0 = base[kClasses] + wrank;
        if (v < n) {
            const uint32_t pos = base[c] + rank;
            list[pos] = v;
            if (nw) lr_words[pos - n_short] = make_uint2(w0, nw);
        }
        unsigned lng = __ballot_sync(0xffffffffu, nw != 0u);
        while (lng) {
            const int q = __ffs(lng) - 1;
            lng &= lng - 1u;
            const uint32_t qv = __shfl_sync(0xffffffffu, v, q), qn = __shfl_sync(0xffffffffu, nw, q);
            const uint32_t qw = __shfl_sync(0xffffffffu, w0, q);
            const uint32_t qb = __shfl_sync(0xffffffffu, (uint32_t)(beg >> 5), q);
            for (uint32_t i = lane; i < qn; i += 32u) lw[qw + i] = make_uint2(qv, qb + i);
        }
        __syncthreads();   // s and base are written again
    }
}

__global__ void k_outdeg(const uint32_t *__restrict__ col, unsigned long long m, uint32_t *__restrict__ deg) {
    for (unsigned long long e = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; e < m;
         e += (unsigned long long)gridDim.x * blockDim.x)
        atomicAdd(deg + col[e], 1u);
}

// diff is kept multiplied by (1 - rj): every edge term (1 - rj) * diff[u] is
// then a load, the same product computed once per vertex instead of per edge.
__global__ void k_pr_init(const uint32_t *__restrict__ deg, uint32_t n, double rj, double *__restrict__ recip,
                          double *__restrict__ weight, double *__restrict__ diff) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const double r = __ddiv_rn(1.0, (double)deg[v]);   // 1/0 = +inf, as the reference's 1.0 / 0
        recip[v] = r;
        weight[v] = 1.0;
        diff[v] = __dmul_rn(1.0 - rj, __dmul_rn(1.0, r));
    }
}

// Returns whether |diff'| exceeds the threshold.
__device__ __forceinline__ bool pr_update(const PrArgs &a, uint32_t v, double s) {
    const double old = a.weight[v];
    const double w = __dadd_rn(a.first ? a.rj : old, s);
    const double d = __dmul_rn(__dadd_rn(w, -old), a.recip[v]);
    a.weight[v] = w;
    a.diff_next[v] = __dmul_rn(a.pj, d);
    return fabs(d) > a.thresh;   // NaN compares false, as in the reference
}

// Four columns from an aligned position; past the last edge one by one.
__device__ __forceinline__ uint4 four_cols(const PrArgs &a, unsigned long long e) {
    if (e + 4ull <= a.m) return __ldg(reinterpret_cast<const uint4 *>(a.col + e));
    return make_uint4(e < a.m ? __ldg(a.col + e) : 0u, e + 1 < a.m ? __ldg(a.col + e + 1) : 0u,
                      e + 2 < a.m ? __ldg(a.col + e + 2) : 0u, 0u);
}

// The terms of positions [lo, hi) in order, eight gathers in flight, handed to
// add(position, term).
template <typename Add>
__device__ __forceinline__ void pull_range(const PrArgs &a, unsigned long long lo, unsigned long long hi, Add add) {
    for (unsigned long long e0 = lo & ~3ull; e0 < hi; e0 += 8ull) {
        uint32_t u[8];
        double t[8];
        const uint4 x = four_cols(a, e0);
        const uint4 y = e0 + 4ull < hi ? four_cols(a, e0 + 4ull) : make_uint4(0u, 0u, 0u, 0u);
        u[0] = x.x, u[1] = x.y, u[2] = x.z, u[3] = x.w;
        u[4] = y.x, u[5] = y.y, u[6] = y.z, u[7] = y.w;
#pragma unroll
        for (int k = 0; k < 8; ++k) t[k] = e0 + k >= lo && e0 + k < hi ? __ldg(a.diff + u[k]) : 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (e0 + k >= lo && e0 + k < hi) add(e0 + k, t[k]);
    }
}

// Blocks of word sums of the long rows, then blocks of short rows, one item a
// thread.  A short row has at most two words: each edge is one add into its
// word's sum, chosen by a select, because a branch at the word boundary runs in
// almost every step of a warp (its rows start anywhere) and repeats the adds.
__global__ void __launch_bounds__(kPrTPB, 6) k_pr_pull(PrArgs a) {
    if (*a.run == 0u) return;
    if (blockIdx.x < a.lw_blocks) {
        const uint32_t x = blockIdx.x * kPrTPB + threadIdx.x;
        if (x >= a.n_lw) return;
        const uint2 w = __ldg(a.lw + x);
        const unsigned long long at = (unsigned long long)w.y << 5;
        const unsigned long long lo = max(a.row[w.x], at), hi = min(a.row[w.x + 1], at + 32ull);
        double p = 0.0;
        pull_range(a, lo, hi, [&](unsigned long long, double t) { p = __dadd_rn(p, t); });
        a.part[x] = p;
        return;
    }
    // a warp's short rows have equal degrees, so its adds run with every lane busy
    const uint32_t i = (blockIdx.x - a.lw_blocks) * kPrTPB + threadIdx.x;
    bool over = false;
    if (i < a.n_short) {
        const uint32_t v = __ldg(a.srow + i);
        const unsigned long long beg = a.row[v], end = a.row[v + 1], cut = (beg | 31ull) + 1ull;
        double p0 = 0.0, p1 = 0.0;
        pull_range(a, beg, end, [&](unsigned long long e, double t) {
            const bool low = e < cut;
            const double p = __dadd_rn(low ? p0 : p1, t);
            p0 = low ? p : p0;
            p1 = low ? p1 : p;
        });
        over = pr_update(a, v, __dadd_rn(p0, p1));
    }
    // one store per block: every thread's own store queues up at one address
    if (__syncthreads_or(over) && threadIdx.x == 0) *a.flag = 1u;
}

__device__ __forceinline__ double butterfly32(double t) {
    for (int h = 16; h > 0; h >>= 1) t = __dadd_rn(t, __shfl_down_sync(0xffffffffu, t, h));
    return t;
}

// The butterfly over N slots in one thread; slots past w.y hold zeros.
template <int N>
__device__ __forceinline__ double thread_row(const PrArgs &a, uint2 w) {
    double q[N];
#pragma unroll
    for (uint32_t k = 0; k < N; ++k) q[k] = k < w.y ? a.part[w.x + k] : 0.0;
#pragma unroll
    for (uint32_t h = N / 2; h > 0; h >>= 1)
#pragma unroll
        for (uint32_t k = 0; k < h; ++k) q[k] = __dadd_rn(q[k], q[k + h]);
    return q[0];
}

// Long rows: blocks of 32 word sums by the butterfly, block sums in order.
// Blocks of rows of more than kMid words first (a warp each: a hub's chain of
// block sums is the longest piece of work), then of rows of kFew..kMid words
// and of fewer, a thread each.
__global__ void __launch_bounds__(kPrTPB) k_pr_long(PrArgs a) {
    if (*a.run == 0u) return;
    const unsigned lane = threadIdx.x & 31u;
    bool over = false;
    if (blockIdx.x < a.big_blocks) {
        const uint32_t i = blockIdx.x * (kPrTPB / 32) + (threadIdx.x >> 5);
        if (i < a.n_big) {
            const uint32_t at = a.n_few + a.n_mid + i;
            const uint2 w = __ldg(a.lr_words + at);
            double r = 0.0;
            double cur = lane < w.y ? a.part[w.x + lane] : 0.0;
            for (uint32_t t0 = 0; t0 < w.y; t0 += 32u) {
                const uint32_t nx = t0 + 32u + lane;
                const double next = nx < w.y ? a.part[w.x + nx] : 0.0;
                r = __dadd_rn(r, __shfl_sync(0xffffffffu, butterfly32(cur), 0));
                cur = next;
            }
            if (lane == 0) over = pr_update(a, __ldg(a.lr_row + at), r);
        }
    } else if (blockIdx.x < a.big_blocks + a.mid_blocks) {
        const uint32_t i = (blockIdx.x - a.big_blocks) * kPrTPB + threadIdx.x;
        if (i < a.n_mid) {
            const uint32_t at = a.n_few + i;
            over = pr_update(a, __ldg(a.lr_row + at), thread_row<kMid>(a, __ldg(a.lr_words + at)));
        }
    } else {
        const uint32_t i = (blockIdx.x - a.big_blocks - a.mid_blocks) * kPrTPB + threadIdx.x;
        if (i < a.n_few) over = pr_update(a, __ldg(a.lr_row + i), thread_row<kFew>(a, __ldg(a.lr_words + i)));
    }
    if (__syncthreads_or(over) && threadIdx.x == 0) *a.flag = 1u;
}

__global__ void k_src_of(const unsigned long long *__restrict__ row, uint32_t n, uint32_t *__restrict__ src) {
    const unsigned lane = threadIdx.x & 31u;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n; v += warps)
        for (unsigned long long e = row[v] + lane; e < row[v + 1]; e += 32ull) src[e] = v;
}

__global__ void k_iota32(uint32_t *__restrict__ id, unsigned long long m) {
    for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < m;
         k += (unsigned long long)gridDim.x * blockDim.x)
        id[k] = (uint32_t)k;
}

__global__ void k_transpose_place(const uint32_t *__restrict__ idx, const uint32_t *__restrict__ src,
                                  const double *__restrict__ w, unsigned long long m, uint32_t *__restrict__ col,
                                  double *__restrict__ wout) {
    for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < m;
         p += (unsigned long long)gridDim.x * blockDim.x) {
        col[p] = src[idx[p]];
        wout[p] = w[idx[p]];
    }
}

__global__ void k_hist64(const uint32_t *__restrict__ col, unsigned long long m, unsigned long long *__restrict__ cnt) {
    for (unsigned long long e = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; e < m;
         e += (unsigned long long)gridDim.x * blockDim.x)
        atomicAdd(cnt + col[e], 1ull);
}

int grid_of(unsigned long long items, int sms) {
    return (int)std::max<unsigned long long>(1, std::min<unsigned long long>((items + 255) / 256, (unsigned long long)sms * 16));
}

// Device buffers of one call.
struct Pool {
    std::vector<void *> p;
    ~Pool() {
        for (void *q : p) cudaFree(q);
    }
    template <typename T> cudaError_t get(T **out, size_t count) {
        void *q = nullptr;
        const cudaError_t e = cudaMalloc(&q, sizeof(T) * (count ? count : 1));
        if (e == cudaSuccess) p.push_back(q);
        *out = static_cast<T *>(q);
        return e;
    }
};

}  // namespace

gbs_status run_pagerank(const gbs_device_csr *c, const gbs_pagerank_params *params, double *rank_out,
                        gbs_pagerank_stats *stats) {
    const uint32_t n = c->n;
    const unsigned long long m = c->m;
    const double rj = (params && params->random_jump > 0) ? params->random_jump : 0.3;
    const double thresh = (params && params->threshold > 0) ? params->threshold : 1e-6;
    const uint32_t max_iters = (params && params->max_iters) ? params->max_iters : 10000u;
    if (!(rj < 1.0)) return fail(GBS_ERR_INVALID_ARG, "random_jump must be in (0, 1)");
    int dev = 0, sms = 0;
    GBS_CUDA(cudaGetDevice(&dev));
    GBS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    cudaStream_t s;
    GBS_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct StreamFree {
        cudaStream_t s;
        ~StreamFree() { cudaStreamDestroy(s); }
    } sf{s};
    cudaEvent_t e0, e1;
    GBS_CUDA(cudaEventCreate(&e0));
    GBS_CUDA(cudaEventCreate(&e1));
    struct EvFree {
        cudaEvent_t a, b;
        ~EvFree() {
            cudaEventDestroy(a);
            cudaEventDestroy(b);
        }
    } ef{e0, e1};
    Pool pool;
    // one allocation for everything whose size is known: a row of more than
    // kShort edges has at most 2 words more than a 32nd of them
    const size_t max_lr = std::min<size_t>(n, (size_t)(m / (kShort + 1)) + 1);
    const size_t max_lw = (size_t)(m / 32) + 2 * max_lr;
    char *mem = nullptr;
    size_t used = 0;
    auto take = [&](size_t bytes) {
        const size_t at = used;
        used += (bytes + 255) & ~(size_t)255;
        return at;
    };
    const size_t o_recip = take(8ull * n), o_weight = take(8ull * n), o_d0 = take(8ull * n), o_d1 = take(8ull * n);
    const size_t o_deg = take(4ull * n), o_list = take(4ull * n), o_lrw = take(8ull * max_lr), o_lw = take(8ull * max_lw);
    const size_t o_part = take(8ull * max_lw), o_cnt = take(sizeof(PrCounts)), o_flag = take(4ull * (kAhead + 1));
    GBS_CUDA(pool.get(&mem, used));
    double *recip = (double *)(mem + o_recip), *weight = (double *)(mem + o_weight);
    double *diff[2] = {(double *)(mem + o_d0), (double *)(mem + o_d1)};
    uint32_t *deg = (uint32_t *)(mem + o_deg), *list = (uint32_t *)(mem + o_list), *flag = (uint32_t *)(mem + o_flag);
    uint2 *lr_words = (uint2 *)(mem + o_lrw), *lw = (uint2 *)(mem + o_lw);
    PrCounts *d_cnt = (PrCounts *)(mem + o_cnt);
    GBS_CUDA(cudaEventRecord(e0, s));
    GBS_CUDA(cudaMemsetAsync(deg, 0, 4ull * (n ? n : 1), s));
    GBS_CUDA(cudaMemsetAsync(d_cnt, 0, sizeof(PrCounts), s));
    k_pr_count<<<grid_of(n, sms), 256, 0, s>>>(c->d_row, n, d_cnt);
    GBS_CUDA(cudaGetLastError());
    PrCounts cnt{}, at{};
    GBS_CUDA(cudaMemcpyAsync(&cnt, d_cnt, sizeof(cnt), cudaMemcpyDeviceToHost, s));
    k_outdeg<<<grid_of(m, sms), 256, 0, s>>>(c->d_col, m, deg);
    k_pr_init<<<grid_of(n, sms), 256, 0, s>>>(deg, n, rj, recip, weight, diff[0]);
    GBS_CUDA(cudaGetLastError());
    GBS_CUDA(cudaStreamSynchronize(s));
    for (uint32_t k = 1; k < kClasses; ++k) at.rows[k] = at.rows[k - 1] + cnt.rows[k - 1];
    const uint32_t n_short = at.rows[kClsFew];
    GBS_CUDA(cudaMemcpyAsync(d_cnt, &at, sizeof(at), cudaMemcpyHostToDevice, s));
    k_pr_place<<<grid_of(n, sms), 256, 0, s>>>(c->d_row, n, d_cnt, n_short, list, lr_words, lw);
    GBS_CUDA(cudaGetLastError());
    PrArgs a{};
    a.row = c->d_row;
    a.col = c->d_col;
    a.m = m;
    a.pj = 1.0 - rj;
    a.rj = rj;
    a.thresh = thresh;
    a.recip = recip;
    a.weight = weight;
    a.lw = lw;
    a.n_lw = cnt.words;
    a.part = (double *)(mem + o_part);
    a.lr_row = list + n_short;
    a.lr_words = lr_words;
    a.n_few = cnt.rows[kClsFew];
    a.n_mid = cnt.rows[kClsMid];
    a.n_big = cnt.rows[kClsBig];
    auto blocks = [](uint32_t items, uint32_t per) { return (items + per - 1u) / per; };
    a.lw_blocks = blocks(a.n_lw, kPrTPB);
    a.big_blocks = blocks(a.n_big, kPrTPB / 32);
    a.mid_blocks = blocks(a.n_mid, kPrTPB);
    const uint32_t g2 = a.big_blocks + a.mid_blocks + blocks(a.n_few, kPrTPB);
    uint32_t it = 0, more = 1, word[kAhead + 1];
    while (more && it < max_iters) {
        const uint32_t batch = std::min(kAhead, max_iters - it);
        std::fill(word, word + kAhead + 1, 0u);
        word[0] = 1u;
        GBS_CUDA(cudaMemcpyAsync(flag, word, sizeof(word), cudaMemcpyHostToDevice, s));
        for (uint32_t k = 0; k < batch; ++k) {
            const uint32_t t = it + k;
            a.diff = diff[t & 1u];
            a.diff_next = diff[(t + 1u) & 1u];
            a.first = t == 0u;
            a.run = flag + k;
            a.flag = flag + k + 1;
            // a row without in-edges keeps its weight after the first iteration
            // and its diff (0, or NaN for 0 * inf) after the second; the third
            // writes it to the other buffer
            const uint32_t skip = t >= 3u ? cnt.rows[0] : 0u;
            a.srow = list + skip;
            a.n_short = n_short - skip;
            const uint32_t g1 = a.lw_blocks + blocks(a.n_short, kPrTPB);
            if (g1) k_pr_pull<<<g1, kPrTPB, 0, s>>>(a);
            if (g2) k_pr_long<<<g2, kPrTPB, 0, s>>>(a);
        }
        GBS_CUDA(cudaGetLastError());
        GBS_CUDA(cudaMemcpyAsync(word, flag, sizeof(word), cudaMemcpyDeviceToHost, s));
        GBS_CUDA(cudaStreamSynchronize(s));
        uint32_t ran = 1;
        while (ran < batch && word[ran]) ++ran;
        it += ran;
        more = word[ran];
    }
    GBS_CUDA(cudaEventRecord(e1, s));
    if (rank_out) GBS_CUDA(cudaMemcpyAsync(rank_out, weight, 8ull * n, cudaMemcpyDeviceToHost, s));
    GBS_CUDA(cudaStreamSynchronize(s));
    if (stats) {
        float ms = 0.f;
        GBS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        stats->iterations = it;
        stats->converged = more ? 0u : 1u;
        stats->device_ms = ms;
        stats->edges = m;
    }
    return GBS_OK;
}

gbs_status transpose_csr(const gbs_device_csr *c, gbs_device_csr *t) {
    const uint32_t n = c->n;
    const unsigned long long m = c->m;
    int dev = 0, sms = 0;
    GBS_CUDA(cudaGetDevice(&dev));
    GBS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    Pool pool;
    uint32_t *src = nullptr, *id = nullptr, *id_s = nullptr, *key_s = nullptr;
    unsigned long long *cnt = nullptr;
    GBS_CUDA(pool.get(&src, m));
    GBS_CUDA(pool.get(&id, m));
    GBS_CUDA(pool.get(&id_s, m));
    GBS_CUDA(pool.get(&key_s, m));
    GBS_CUDA(pool.get(&cnt, (size_t)n + 1));
    k_src_of<<<std::max(1, std::min<int>((n + 7) / 8, sms * 16)), 256>>>(c->d_row, n, src);
    k_iota32<<<grid_of(m, sms), 256>>>(id, m);
    GBS_CUDA(cudaGetLastError());
    size_t tmp = 0;
    GBS_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, c->d_col, key_s, id, id_s, (int64_t)m));
    char *t_mem = nullptr;
    GBS_CUDA(pool.get(&t_mem, tmp));
    GBS_CUDA(cub::DeviceRadixSort::SortPairs(t_mem, tmp, c->d_col, key_s, id, id_s, (int64_t)m));
    GBS_CUDA(cudaMemset(cnt, 0, 8ull * (n + 1ull)));
    k_hist64<<<grid_of(m, sms), 256>>>(c->d_col, m, cnt);
    GBS_CUDA(cudaGetLastError());
    GBS_CUDA(cudaMalloc(&t->d_row, 8ull * (n + 1ull)));
    size_t tmp2 = 0;
    GBS_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp2, cnt, t->d_row, (int64_t)n + 1));
    char *t2 = nullptr;
    GBS_CUDA(pool.get(&t2, tmp2));
    GBS_CUDA(cub::DeviceScan::ExclusiveSum(t2, tmp2, cnt, t->d_row, (int64_t)n + 1));
    GBS_CUDA(cudaMalloc(&t->d_col, 4ull * (m ? m : 1)));
    GBS_CUDA(cudaMalloc(&t->d_w, 8ull * (m ? m : 1)));
    k_transpose_place<<<grid_of(m, sms), 256>>>(id_s, src, c->d_w, m, t->d_col, t->d_w);
    GBS_CUDA(cudaGetLastError());
    GBS_CUDA(cudaDeviceSynchronize());
    t->n = n;
    t->m = m;
    return GBS_OK;
}

}  // namespace gbs

extern "C" {

gbs_status gbs_pagerank(const gbs_device_csr *in_edges, const gbs_pagerank_params *params, double *rank_out,
                        gbs_pagerank_stats *stats) {
    if (!in_edges) return gbs::fail(GBS_ERR_INVALID_ARG, "csr is NULL");
    return gbs::run_pagerank(in_edges, params, rank_out, stats);
}

gbs_status gbs_device_csr_transpose(const gbs_device_csr *c, gbs_device_csr **out) {
    if (!c || !out) return gbs::fail(GBS_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    gbs_device_csr *t = new gbs_device_csr();
    const gbs_status st = gbs::transpose_csr(c, t);
    if (st != GBS_OK) {
        gbs_device_csr_destroy(t);
        return st;
    }
    *out = t;
    return GBS_OK;
}

}  // extern "C"
