// gbs_ingest.cu -- graph ingest on the GPU (sm_103a): the reference's text
// and binary CSR readers (graph/csr.c:4-299), duplicate-edge removal
// (partition/csr_partition_bin_mpi.c:47-105) and the build of a resident
// graph, all on the device.
//
// Text (scan_csr_idx + read_graph_csr, graph/csr.c:4-202): "p <name> v_num
// e_num offset g_v_size" then "a v_id v_to weight" lines (other lines, e.g.
// "c" comments, are skipped); the first e_num "a" lines are read.  SEND:
// row = v_id - offset, column = v_to - 1; RECV: row = v_to - offset, column =
// v_id - 1.  Rows keep their edges in file order (the reference fills them in
// file order).  The weight is (double)v_to / (double)v_num with the file's
// v_to, and the reference stores the k-th line's weight at CSR position k
// (edge_info[e_num_read], :46), not at that edge's position: the two agree
// only for a file sorted by row.  Both are kept here as the reference has
// them; the third number of an "a" line is read and ignored, as there.
//
// Binary (read_csr_bin, graph/csr.c:211-299): int64 v_num, e_num, offset,
// g_v_size, then e_num int64 (from, to) pairs.  SEND: row = from - offset,
// column = to - target_offset; RECV: row = to - offset, column = from -
// target_offset (target_offset is the reference's OFFSET: 1, or 0 in its
// Graph500 build).  The weight of CSR position p is 0.1 for even p and 0.2 for
// odd p (:293-298).  With dedup, a (from, to) pair seen earlier in the file is
// dropped first, as remove_duplicate does.
//
// Device work: the text is cut into 512-byte chunks; a warp counts and then
// lists the "a" lines of a chunk, 16 bytes a lane (one exclusive scan between),
// and one thread per line parses its numbers into a row, a column and a weight.
// The CSR is a stable radix sort of the columns by row (CUB), so rows keep file
// order; a file already in row order is not sorted.  The row offsets are
// searched for in the sorted rows.  Duplicate removal sorts the pairs by the
// bits their largest ids use.  Every call takes its buffers from one
// allocation: a cudaMalloc of a few MB takes 35 us here, its cudaFree 35-140,
// and a call has more than ten.  R-MAT of 65,536 vertices, 30 MB of text: copy,
// lines and numbers 0.76 -> 0.27 ms (a thread per chunk read byte by byte),
// build 0.68 -> 0.15, the call 1.9 -> 0.67; 3.1 M pairs with duplicates: 3.0 ->
// 1.3.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <chrono>
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "gbs_host.hpp"

namespace gbs {
namespace {

constexpr uint64_t kChunk = 512;     // bytes of text per counting warp

enum IngestErr : uint32_t {
    kIngOk = 0,
    kIngSyntax = 1,      // an "a" line without three integers
    kIngRange = 2,       // a row or column outside [0, v_num)
    kIngDupRange = 3,    // a pair outside [0, 2^32) (duplicate removal)
};

struct DevErr {
    uint32_t code;
    uint32_t pad;
    unsigned long long where;   // edge index (file order)
};

__device__ __forceinline__ void set_err(DevErr *e, uint32_t code, unsigned long long where) {
    if (atomicCAS(&e->code, 0u, code) == 0u) e->where = where;
}

__device__ __forceinline__ bool is_blank(char c) { return c == ' ' || c == '\t' || c == '\r'; }

// An "a" record starts at byte i: i is the start of a line (after optional
// blanks) whose first token is exactly "a".
__device__ __forceinline__ bool a_line_at(const char *buf, unsigned long long len, unsigned long long i) {
    if (i != 0 && buf[i - 1] != '\n') return false;
    while (i < len && is_blank(buf[i])) ++i;
    return i + 1 < len && buf[i] == 'a' && (buf[i + 1] == ' ' || buf[i + 1] == '\t');
}

// The "a" records whose preceding newline (or the start of the file) lies in a
// chunk: counted, or listed from base[chunk] on.  A warp takes a chunk, a lane
// 16 bytes of it (buf is padded to whole 16-byte groups).
template <bool List>
__global__ void __launch_bounds__(256) k_lines(const char *__restrict__ buf, unsigned long long len,
                                               unsigned long long chunks, unsigned long long *__restrict__ cnt,
                                               const unsigned long long *__restrict__ base,
                                               unsigned long long *__restrict__ pos, unsigned long long cap) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned long long warp = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5;
    const unsigned long long warps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
    for (unsigned long long c = warp; c < chunks; c += warps) {
        const unsigned long long at = c * kChunk + 16ull * lane;
        uint32_t starts = 0;   // bit j: a record starts at at + j + 1; bit 16: at 0
        if (at < len) {
            const uint4 x = *reinterpret_cast<const uint4 *>(buf + at);
            const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (((w[j >> 2] >> (8 * (j & 3))) & 0xFFu) == '\n' && at + j < len) starts |= 1u << j;
            for (uint32_t b = starts; b; b &= b - 1u) {
                const int j = __ffs((int)b) - 1;
                if (!a_line_at(buf, len, at + j + 1ull)) starts &= ~(1u << j);
            }
            if (at == 0ull && a_line_at(buf, len, 0ull)) starts |= 1u << 16;
        }
        const uint32_t n = (uint32_t)__popc(starts);
        if (!List) {
            const uint32_t total = __reduce_add_sync(0xffffffffu, n);
            if (lane == 0) cnt[c] = total;
        } else {
            uint32_t incl = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if ((int)lane >= o) incl += y;
            }
            unsigned long long k = base[c] + incl - n;
            if (starts & (1u << 16)) {   // the start of the file comes before its first newline
                if (k < cap) pos[k] = 0ull;
                ++k;
            }
            for (uint32_t b = starts & 0xFFFFu; b; b &= b - 1u, ++k)
                if (k < cap) pos[k] = at + (unsigned long long)__ffs((int)b);
        }
    }
}

// Reads a decimal integer (optional sign) after blanks; false if none.
__device__ __forceinline__ bool read_int(const char *buf, unsigned long long len, unsigned long long &i,
                                         long long &out) {
    while (i < len && is_blank(buf[i])) ++i;
    bool neg = false;
    if (i < len && (buf[i] == '-' || buf[i] == '+')) {
        neg = buf[i] == '-';
        ++i;
    }
    if (i >= len || buf[i] < '0' || buf[i] > '9') return false;
    unsigned long long v = 0;
    while (i < len && buf[i] >= '0' && buf[i] <= '9') v = v * 10ull + (unsigned long long)(buf[i++] - '0');
    out = neg ? -(long long)v : (long long)v;
    return true;
}

// Row and column of an edge, checked against [0, v_num).
__device__ __forceinline__ void put_edge(long long r, long long c, long long v_num, unsigned long long k,
                                         uint32_t *__restrict__ row, uint32_t *__restrict__ col, DevErr *err) {
    if (r < 0 || r >= v_num || c < 0 || c >= v_num) {
        set_err(err, kIngRange, k);
        r = c = 0;
    }
    row[k] = (uint32_t)r;
    col[k] = (uint32_t)c;
}

// One thread per "a" record, at most cap of them: row, column, and the weight
// of CSR position k, the k-th line's v_to / v_num (the weight token is checked
// and ignored, as the reference ignores it).  err[0]: a malformed line, err[1]:
// an edge out of range.
__global__ void k_parse_lines(const char *__restrict__ buf, unsigned long long len,
                              const unsigned long long *__restrict__ pos, const unsigned long long *__restrict__ lines,
                              unsigned long long cap, long long row_shift, bool by_to, long long v_num,
                              uint32_t *__restrict__ row, uint32_t *__restrict__ col, double *__restrict__ wout,
                              DevErr *err) {
    const unsigned long long count = min(*lines, cap);
    for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < count;
         k += (unsigned long long)gridDim.x * blockDim.x) {
        unsigned long long i = pos[k];
        while (is_blank(buf[i])) ++i;
        ++i;   // the 'a'
        long long a = 0, b = 0, w = 0;
        if (!read_int(buf, len, i, a) || !read_int(buf, len, i, b) || !read_int(buf, len, i, w)) {
            set_err(err, kIngSyntax, k);
            row[k] = col[k] = 0u;
            continue;
        }
        put_edge((by_to ? b : a) - row_shift, (by_to ? a : b) - 1, v_num, k, row, col, err + 1);
        wout[k] = (double)b / (double)v_num;
    }
}

// Binary pairs: all of them, or (keep given) pair k as edge at[k] where keep[k] is set.
__global__ void k_pair_rows(const longlong2 *__restrict__ pairs, unsigned long long m, const uint32_t *__restrict__ keep,
                            const uint32_t *__restrict__ at, long long row_shift, long long col_shift, bool by_to,
                            long long v_num, uint32_t *__restrict__ row, uint32_t *__restrict__ col, DevErr *err) {
    for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < m;
         k += (unsigned long long)gridDim.x * blockDim.x) {
        if (keep && !keep[k]) continue;
        const longlong2 p = pairs[k];
        put_edge((by_to ? p.y : p.x) - row_shift, (by_to ? p.x : p.y) - col_shift, v_num, keep ? at[k] : k, row, col, err);
    }
}

// Whether the rows are not in ascending order.
__global__ void k_row_order(const uint32_t *__restrict__ row, unsigned long long m, uint32_t *unsorted) {
    bool bad = false;
    for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x + 1ull; k < m;
         k += (unsigned long long)gridDim.x * blockDim.x)
        bad |= row[k] < row[k - 1ull];
    if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31u) == 0) *unsorted = 1u;
}

// out[v] = the first position of row v or a later one.
__global__ void k_row_starts(const uint32_t *__restrict__ row, unsigned long long m, uint32_t n,
                             unsigned long long *__restrict__ out) {
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x) {
        unsigned long long lo = 0ull, hi = m;
        while (lo < hi) {
            const unsigned long long mid = lo + (hi - lo) / 2ull;
            if (row[mid] < v) lo = mid + 1ull;
            else hi = mid;
        }
        out[v] = lo;
    }
}

// Binary files: the weight of CSR position p is 0.1 for even p, 0.2 for odd p.
__global__ void k_parity_weights(unsigned long long m, double *__restrict__ out) {
    for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < m;
         p += (unsigned long long)gridDim.x * blockDim.x)
        out[p] = (p & 1ull) ? 0.2 : 0.1;
}

// Duplicate removal: the largest ids of the raw pairs, which must be in
// [0, 2^32); then key = from << to_bits | to.
__global__ void k_pair_max(const longlong2 *__restrict__ pairs, unsigned long long m, uint32_t *mx, DevErr *err) {
    uint32_t a = 0, b = 0;
    for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < m;
         k += (unsigned long long)gridDim.x * blockDim.x) {
        const longlong2 p = pairs[k];
        if (p.x < 0 || p.y < 0 || p.x > 0xFFFFFFFFll || p.y > 0xFFFFFFFFll) {
            set_err(err, kIngDupRange, k);
        } else {
            a = max(a, (uint32_t)p.x);
            b = max(b, (uint32_t)p.y);
        }
    }
    a = __reduce_max_sync(0xffffffffu, a);
    b = __reduce_max_sync(0xffffffffu, b);
    if ((threadIdx.x & 31u) == 0) {
        atomicMax(mx, a);
        atomicMax(mx + 1, b);
    }
}
__global__ void k_pair_keys(const longlong2 *__restrict__ pairs, unsigned long long m, int to_bits,
                            unsigned long long *__restrict__ key, uint32_t *__restrict__ idx) {
    for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < m;
         k += (unsigned long long)gridDim.x * blockDim.x) {
        const longlong2 p = pairs[k];
        key[k] = ((unsigned long long)p.x << to_bits) | (unsigned long long)p.y;
        idx[k] = (uint32_t)k;
    }
}

// keep[original index] = 1 for the first occurrence of each pair (the sort is
// stable, so the first of a run of equal keys is the earliest in the file).
__global__ void k_first_of_run(const unsigned long long *__restrict__ key, const uint32_t *__restrict__ idx,
                               unsigned long long m, uint32_t *__restrict__ keep) {
    for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < m;
         p += (unsigned long long)gridDim.x * blockDim.x)
        keep[idx[p]] = (p == 0 || key[p] != key[p - 1]) ? 1u : 0u;
}

// ------------------------------------------------- resident graph build
// What the pass over the edges finds.
struct EdgeStats {
    unsigned long long bad;       // 4 x the first bad edge + what is wrong (kBad*); ~0: none
    unsigned long long max_bits;  // largest weight, bits of its type
    double sum;                   // of the weights
    uint32_t unsorted;            // a row's columns are not in ascending order
    uint32_t zero;                // a weight is zero
    uint32_t rows_bad;            // row offsets decrease
    uint32_t max_deg;             // longest row
};
enum : uint32_t { kBadCol = 0, kBadWeight = 1, kBadInteger = 2 };

// Weight bits of type WT (0 uint32, 1 float32, 2 float64) from a source of the
// same type or from a device CSR's doubles; -0 as +0.  Returns kBad* or ~0u.
template <int WT, typename Src>
__device__ __forceinline__ uint32_t weight_bits(Src w, unsigned long long &bits) {
    if constexpr (sizeof(Src) == 4 && WT == 0) {
        bits = w;
        return ~0u;
    } else {
        if (!(w >= Src(0)) || isinf(w)) {
            bits = 0ull;
            return kBadWeight;
        }
        if (w == Src(0)) w = Src(0);
        if constexpr (WT == 2) {
            bits = (unsigned long long)__double_as_longlong(w);
        } else if constexpr (WT == 1) {
            bits = __float_as_uint((float)w);
        } else {
            bits = (unsigned long long)(uint32_t)w;
            if (w != floor(w) || w > Src(4294967295.0)) return kBadInteger;
        }
        return ~0u;
    }
}

// One pass over the edges in CSR order: every edge's row, checks, the sort key
// (uint32 / float32: row << 32 | weight bits; float64: weight bits, the row
// beside it) and the statistics.  A warp takes 1,024 consecutive edges, a lane
// every 32nd of them: its row is found by a search once and then by walking on.
// A search stays inside the offsets even where they decrease (the caller looks
// at rows_bad first).
constexpr uint32_t kEdgeTile = 1024;
template <int WT, typename Src>
__global__ void __launch_bounds__(256) k_edges(const unsigned long long *__restrict__ row, const uint32_t *__restrict__ col,
                                               const Src *__restrict__ w, uint32_t n, unsigned long long m,
                                               unsigned long long *__restrict__ key, uint32_t *__restrict__ row_of,
                                               double *__restrict__ part, EdgeStats *st) {
    const unsigned lane = threadIdx.x & 31u;
    const unsigned long long warp = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) >> 5;
    const unsigned long long warps = ((unsigned long long)gridDim.x * blockDim.x) >> 5;
    unsigned long long mx = 0ull, bad = ~0ull;
    double sum = 0.0;
    bool unsorted = false, zero = false;
    for (unsigned long long t = warp * kEdgeTile; t < m; t += warps * kEdgeTile) {
        uint32_t v = 0, top = n - 1u;   // the last row that starts at or before the lane's first edge
        while (v < top) {
            const uint32_t mid = v + (top - v + 1u) / 2u;
            if (row[mid] <= t + lane) v = mid;
            else top = mid - 1u;
        }
        for (unsigned long long e = t + lane; e < min(m, t + kEdgeTile); e += 32u) {
            v = row_at(row, n, v, e);
            const uint32_t c = col[e];
            unsigned long long bits;
            const Src x = w[e];
            const uint32_t why = weight_bits<WT, Src>(x, bits);
            if (c >= n) bad = min(bad, 4ull * e + kBadCol);
            else if (why != ~0u) bad = min(bad, 4ull * e + why);
            unsorted |= e > row[v] && col[e - 1u] > c;
            zero |= bits == 0ull;
            mx = max(mx, bits);
            sum += (double)x;
            if (WT == 2) {
                key[e] = bits;
                row_of[e] = v;
            } else {
                key[e] = ((unsigned long long)v << 32) | bits;
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        mx = max(mx, __shfl_down_sync(0xffffffffu, mx, o));
        bad = min(bad, __shfl_down_sync(0xffffffffu, bad, o));
        sum += __shfl_down_sync(0xffffffffu, sum, o);
    }
    if (__any_sync(0xffffffffu, unsorted) && lane == 0) st->unsorted = 1u;
    if (__any_sync(0xffffffffu, zero) && lane == 0) st->zero = 1u;
    if (lane == 0) {
        if (mx) atomicMax(&st->max_bits, mx);
        if (bad != ~0ull) atomicMin(&st->bad, bad);
        part[warp] = sum;
    }
}

// The warps' sums of weights, always in one order: the mean weight is an input
// of the learned controller, and builds of one graph must agree in it.
constexpr int kSumTPB = 256;
__global__ void __launch_bounds__(kSumTPB) k_weight_sum(const double *__restrict__ part, uint32_t count, EdgeStats *st) {
    __shared__ double s[kSumTPB];
    double x = 0.0;
    for (uint32_t i = threadIdx.x; i < count; i += kSumTPB) x += part[i];
    s[threadIdx.x] = x;
    for (int h = kSumTPB / 2; h > 0; h >>= 1) {
        __syncthreads();
        if ((int)threadIdx.x < h) s[threadIdx.x] += s[threadIdx.x + h];
    }
    if (threadIdx.x == 0) st->sum = s[0];
}

__global__ void k_edge_stats_init(EdgeStats *st) { *st = EdgeStats{~0ull, 0ull, 0.0, 0u, 0u, 0u, 0u}; }

template <typename K>
__global__ void k_gather_key(const K *__restrict__ src, const uint32_t *__restrict__ id, unsigned long long m,
                             K *__restrict__ key) {
    for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < m;
         p += (unsigned long long)gridDim.x * blockDim.x)
        key[p] = src[id[p]];
}

// Sorted (row, weight) keys and the columns that came with them.
__global__ void k_adj32(const unsigned long long *__restrict__ key, const uint32_t *__restrict__ col,
                        unsigned long long m, uint2 *__restrict__ adj) {
    for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < m;
         p += (unsigned long long)gridDim.x * blockDim.x)
        adj[p] = make_uint2(col[p], (uint32_t)key[p]);
}

__global__ void k_adj64(const uint32_t *__restrict__ id, const uint32_t *__restrict__ col,
                        const unsigned long long *__restrict__ wbits, unsigned long long m, uint2 *__restrict__ adj,
                        unsigned long long *__restrict__ w64) {
    for (unsigned long long p = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; p < m;
         p += (unsigned long long)gridDim.x * blockDim.x) {
        const uint32_t e = id[p];
        adj[p] = make_uint2(col[e], 0u);
        w64[p] = wbits[e];
    }
}

// uint32 offsets, whether the offsets decrease, the longest row.
__global__ void k_row32(const unsigned long long *__restrict__ row, uint32_t n, uint32_t *__restrict__ row32,
                        EdgeStats *st) {
    uint32_t d = 0;
    bool bad = false;
    for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v <= n; v += gridDim.x * blockDim.x) {
        row32[v] = (uint32_t)row[v];
        if (v < n) {
            d = max(d, (uint32_t)(row[v + 1] - row[v]));
            bad |= row[v + 1] < row[v];
        }
    }
    d = __reduce_max_sync(0xffffffffu, d);
    if ((threadIdx.x & 31u) == 0) atomicMax(&st->max_deg, d);
    if (bad) st->rows_bad = 1u;
}

// ----------------------------------------------------------------- host
// Device buffers of one call, released on every exit path: taken from one
// block where it was reserved and holds them (a stack: reset gives back what was
// taken since the mark, for later work on the same stream), allocated one by one
// otherwise.  Calls beyond kMaxBlock do not reserve: freeing each buffer when
// it is done keeps their peak lower.
constexpr size_t kMaxBlock = 8ull << 30;
// What a block has room for beside the buffers of `items` that are counted one by
// one: sort scratch, alignment.  Small blocks stay below the size from which a
// cudaMalloc and its cudaFree are slow (35 us and more): a file of 64 vertices
// 0.361 -> 0.259 ms, a graph of it 0.200 -> 0.104.
constexpr size_t slack(unsigned long long items) {
    return (size_t)std::min<unsigned long long>(16ull << 20, (96ull << 10) + 16ull * items);
}
// Failure-path tests: bytes one call may hold on this thread, and whether it fails
// beyond them for want of memory (gbs_test_buffer_limit).
thread_local size_t t_buffer_limit = SIZE_MAX;
thread_local bool t_limit_is_memory = true;
struct Bufs {
    std::vector<std::pair<void *, size_t>> own;
    char *block = nullptr;
    size_t cap = 0, used = 0, held = 0;
    // memory that runs out is a size no device has: the runtime's own error
    cudaError_t alloc(void **p, size_t bytes) {
        const bool over = held + bytes > t_buffer_limit;
        if (over && !t_limit_is_memory) return cudaErrorUnknown;
        const cudaError_t e = cudaMalloc(p, over ? (size_t)1 << 62 : bytes);
        if (e == cudaSuccess) held += bytes;
        return e;
    }
    void reserve(size_t bytes) {
        if (block || bytes > kMaxBlock) return;
        if (alloc(reinterpret_cast<void **>(&block), bytes) == cudaSuccess) cap = bytes;
        else cudaGetLastError();
    }
    template <typename T> cudaError_t get(T **out, size_t count) {
        const size_t bytes = (sizeof(T) * (count ? count : 1) + 255) & ~(size_t)255;
        if (used + bytes <= cap) {
            *out = reinterpret_cast<T *>(block + used);
            used += bytes;
            return cudaSuccess;
        }
        void *q = nullptr;
        const cudaError_t e = alloc(&q, bytes);
        if (e == cudaSuccess) own.push_back({q, bytes});
        *out = static_cast<T *>(q);
        return e;
    }
    struct Mark {
        size_t used, own;
    };
    Mark mark() const { return {used, own.size()}; }
    void reset(Mark m) {
        used = m.used;
        for (; own.size() > m.own; own.pop_back()) {
            cudaFree(own.back().first);
            held -= own.back().second;
        }
    }
    ~Bufs() {
        reset({0, 0});
        cudaFree(block);
    }
};

#define ING_CUDA(call)                                                                       \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            return fail(e_ == cudaErrorMemoryAllocation ? GBS_ERR_NO_MEMORY : GBS_ERR_CUDA,  \
                        std::string(#call) + ": " + cudaGetErrorString(e_));                 \
    } while (0)

int grid_for(unsigned long long items, int sms) {
    const unsigned long long b = (items + 255) / 256;
    return (int)std::max<unsigned long long>(1, std::min<unsigned long long>(b, (unsigned long long)sms * 16));
}

double ms_since(std::chrono::steady_clock::time_point t0) {
    return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
}

gbs_status check_err(const DevErr &e, const char *what) {
    if (e.code == kIngOk) return GBS_OK;
    const char *why = e.code == kIngSyntax    ? "an \"a\" line without three integers"
                      : e.code == kIngRange   ? "a row or column outside [0, v_num)"
                                              : "a vertex id outside [0, 2^32)";
    return fail(GBS_ERR_INVALID_ARG, std::string(what) + ": edge " + std::to_string(e.where) + ": " + why);
}

// CUB radix sort of (key, value) pairs, stable; out buffers given.
template <typename K>
gbs_status sort_pairs(const K *kin, K *kout, const uint32_t *vin, uint32_t *vout, unsigned long long m,
                      cudaStream_t s, Bufs &bufs, int end_bit = (int)sizeof(K) * 8) {
    const Bufs::Mark at = bufs.mark();
    size_t tmp = 0;
    ING_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, kin, kout, vin, vout, (int64_t)m, 0, end_bit, s));
    void *t = nullptr;
    ING_CUDA(bufs.get(reinterpret_cast<char **>(&t), tmp));
    ING_CUDA(cub::DeviceRadixSort::SortPairs(t, tmp, kin, kout, vin, vout, (int64_t)m, 0, end_bit, s));
    bufs.reset(at);
    return GBS_OK;
}

template <typename T>
gbs_status excl_sum(const T *in, T *out, unsigned long long count, cudaStream_t s, Bufs &bufs) {
    const Bufs::Mark at = bufs.mark();
    size_t tmp = 0;
    ING_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tmp, in, out, (int64_t)count, s));
    void *t = nullptr;
    ING_CUDA(bufs.get(reinterpret_cast<char **>(&t), tmp));
    ING_CUDA(cub::DeviceScan::ExclusiveSum(t, tmp, in, out, (int64_t)count, s));
    bufs.reset(at);
    return GBS_OK;
}

int bits_of(unsigned long long most) {   // bits of the values 0 .. most, at least 1
    int b = 1;
    while (b < 64 && (most >> b)) ++b;
    return b;
}

// Edges (row, col) in file order -> the CSR's offsets and columns, rows in file
// order.  `unsorted`: a device word the call may use.
gbs_status build_csr(const uint32_t *row, const uint32_t *col, unsigned long long m, uint32_t n, uint32_t *unsorted,
                     cudaStream_t s, int sms, Bufs &bufs, gbs_device_csr *out) {
    uint32_t hu = 0;
    ING_CUDA(cudaMemsetAsync(unsorted, 0, sizeof(uint32_t), s));
    k_row_order<<<grid_for(m, sms), 256, 0, s>>>(row, m, unsorted);
    ING_CUDA(cudaGetLastError());
    ING_CUDA(cudaMemcpyAsync(&hu, unsorted, sizeof(hu), cudaMemcpyDeviceToHost, s));
    ING_CUDA(cudaMalloc(&out->d_row, sizeof(unsigned long long) * ((size_t)n + 1)));
    ING_CUDA(cudaMalloc(&out->d_col, sizeof(uint32_t) * (m ? m : 1)));
    ING_CUDA(cudaStreamSynchronize(s));
    if (hu) {
        uint32_t *row_s = nullptr;
        ING_CUDA(bufs.get(&row_s, m));
        const gbs_status st = sort_pairs<uint32_t>(row, row_s, col, out->d_col, m, s, bufs, bits_of(n - 1u));
        if (st != GBS_OK) return st;
        row = row_s;
    } else {
        ING_CUDA(cudaMemcpyAsync(out->d_col, col, sizeof(uint32_t) * m, cudaMemcpyDeviceToDevice, s));
    }
    k_row_starts<<<grid_for((unsigned long long)n + 1, sms), 256, 0, s>>>(row, m, n, out->d_row);
    ING_CUDA(cudaGetLastError());
    out->n = n;
    out->m = m;
    return GBS_OK;
}

// File bytes into a pinned host buffer.
gbs_status read_file(const char *path, std::vector<char> &host, char **pinned, size_t &len) {
    FILE *f = std::fopen(path, "rb");
    if (!f) return fail(GBS_ERR_INVALID_ARG, std::string("cannot open ") + path);
    std::fseek(f, 0, SEEK_END);
    const long sz = std::ftell(f);
    std::fseek(f, 0, SEEK_SET);
    if (sz < 0) {
        std::fclose(f);
        return fail(GBS_ERR_INVALID_ARG, std::string("cannot size ") + path);
    }
    len = (size_t)sz;
    char *p = nullptr;
    if (cudaHostAlloc(reinterpret_cast<void **>(&p), len ? len : 1, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        host.resize(len ? len : 1);
        p = host.data();
    } else {
        *pinned = p;
    }
    const size_t got = len ? std::fread(p, 1, len, f) : 0;
    std::fclose(f);
    if (got != len) return fail(GBS_ERR_INVALID_ARG, std::string("short read of ") + path);
    if (!*pinned) *pinned = nullptr;
    return GBS_OK;
}

struct PinnedFree {
    char *p = nullptr;
    ~PinnedFree() {
        if (p) cudaFreeHost(p);
    }
};

// The "p" record: the first line whose first token is "p", before any "a".
gbs_status text_header(const char *buf, size_t len, long long hdr[4]) {
    size_t i = 0;
    while (i < len) {
        size_t j = i;
        while (j < len && (buf[j] == ' ' || buf[j] == '\t' || buf[j] == '\r')) ++j;
        size_t e = j;
        while (e < len && buf[e] != '\n') ++e;
        if (j + 1 < len && buf[j] == 'a' && (buf[j + 1] == ' ' || buf[j + 1] == '\t'))
            return fail(GBS_ERR_INVALID_ARG, "text graph: an \"a\" line before the \"p\" line");
        if (j + 1 < len && buf[j] == 'p' && (buf[j + 1] == ' ' || buf[j + 1] == '\t')) {
            std::string line(buf + j + 1, buf + e);
            char name[64] = {0};
            long long v[4];
            if (std::sscanf(line.c_str(), " %63s %lld %lld %lld %lld", name, &v[0], &v[1], &v[2], &v[3]) != 5)
                return fail(GBS_ERR_INVALID_ARG, "text graph: malformed \"p\" line");
            for (int k = 0; k < 4; ++k) hdr[k] = v[k];
            return GBS_OK;
        }
        i = e + 1;
    }
    return fail(GBS_ERR_INVALID_ARG, "text graph: no \"p\" line");
}

gbs_status check_header(const long long h[4]) {
    if (h[0] < 1 || h[0] > 0x7FFFFFFFll) return fail(GBS_ERR_INVALID_ARG, "v_num must be in [1, 2^31)");
    if (h[1] < 0 || h[1] >= 0xFFFFFFFFll) return fail(GBS_ERR_UNSUPPORTED, "e_num must be in [0, 2^32 - 1)");
    return GBS_OK;
}

}  // namespace

// Parses text already in memory (host bytes).
gbs_status ingest_text(const char *bytes, size_t len, int direction, gbs_device_csr *out, gbs_ingest_info *info) {
    long long hdr[4];
    gbs_status st = text_header(bytes, len, hdr);
    if (st != GBS_OK) return st;
    st = check_header(hdr);
    if (st != GBS_OK) return st;
    int dev = 0, sms = 0;
    ING_CUDA(cudaGetDevice(&dev));
    ING_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    cudaStream_t s;
    ING_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct StreamFree {
        cudaStream_t s;
        ~StreamFree() { cudaStreamDestroy(s); }
    } sf{s};
    Bufs bufs;
    cudaEvent_t ev[3];
    for (auto &e : ev) ING_CUDA(cudaEventCreate(&e));
    struct EvFree {
        cudaEvent_t *e;
        ~EvFree() {
            for (int i = 0; i < 3; ++i) cudaEventDestroy(e[i]);
        }
    } ef{ev};
    // the reference stops after e_num records, and none is shorter than "a 1 1 1"
    const unsigned long long cap = std::min<unsigned long long>((unsigned long long)hdr[1], len / 7 + 1);
    const unsigned long long chunks = (len + kChunk - 1) / kChunk;
    bufs.reserve(len + 16 * chunks + 36 * cap + slack(cap));
    char *dbuf = nullptr;
    unsigned long long *cnt = nullptr, *base = nullptr, *pos = nullptr;
    uint32_t *row = nullptr, *col = nullptr, *word = nullptr;
    DevErr *d_err = nullptr;
    ING_CUDA(bufs.get(&word, 1));
    ING_CUDA(bufs.get(&d_err, 2));
    ING_CUDA(bufs.get(&row, cap));
    ING_CUDA(bufs.get(&col, cap));
    ING_CUDA(cudaMalloc(&out->d_w, sizeof(double) * (cap ? cap : 1)));
    const Bufs::Mark parse = bufs.mark();
    ING_CUDA(bufs.get(&dbuf, len + 16));
    ING_CUDA(bufs.get(&cnt, chunks + 1));
    ING_CUDA(bufs.get(&base, chunks + 1));
    ING_CUDA(bufs.get(&pos, cap));
    ING_CUDA(cudaEventRecord(ev[0], s));
    ING_CUDA(cudaMemcpyAsync(dbuf, bytes, len, cudaMemcpyHostToDevice, s));
    ING_CUDA(cudaMemsetAsync(cnt + chunks, 0, sizeof(unsigned long long), s));
    ING_CUDA(cudaMemsetAsync(d_err, 0, 2 * sizeof(DevErr), s));
    const int gc = grid_for(chunks * 32, sms);
    k_lines<false><<<gc, 256, 0, s>>>(dbuf, len, chunks, cnt, nullptr, nullptr, 0);
    ING_CUDA(cudaGetLastError());
    st = excl_sum(cnt, base, chunks + 1, s, bufs);
    if (st != GBS_OK) return st;
    // SEND: row = v_id - offset, col = v_to - 1; RECV: row = v_to - offset, col = v_id - 1
    const bool send = direction != GBS_DIR_RECV;
    k_lines<true><<<gc, 256, 0, s>>>(dbuf, len, chunks, nullptr, base, pos, cap);
    k_parse_lines<<<grid_for(cap, sms), 256, 0, s>>>(dbuf, len, pos, base + chunks, cap, hdr[2], !send, hdr[0], row, col,
                                                     out->d_w, d_err);
    ING_CUDA(cudaGetLastError());
    unsigned long long lines = 0;
    DevErr he[2] = {};
    ING_CUDA(cudaMemcpyAsync(&lines, base + chunks, sizeof(lines), cudaMemcpyDeviceToHost, s));
    ING_CUDA(cudaMemcpyAsync(he, d_err, sizeof(he), cudaMemcpyDeviceToHost, s));
    ING_CUDA(cudaEventRecord(ev[1], s));
    ING_CUDA(cudaStreamSynchronize(s));
    for (const DevErr &e : he)
        if ((st = check_err(e, "text graph")) != GBS_OK) return st;
    const unsigned long long m = std::min(lines, cap);
    bufs.reset(parse);
    st = build_csr(row, col, m, (uint32_t)hdr[0], word, s, sms, bufs, out);
    if (st != GBS_OK) return st;
    ING_CUDA(cudaEventRecord(ev[2], s));
    ING_CUDA(cudaEventSynchronize(ev[2]));
    if (info) {
        float a = 0.f, b = 0.f;
        ING_CUDA(cudaEventElapsedTime(&a, ev[0], ev[1]));
        ING_CUDA(cudaEventElapsedTime(&b, ev[1], ev[2]));
        info->v_num = hdr[0];
        info->e_num = hdr[1];
        info->offset = hdr[2];
        info->g_v_size = hdr[3];
        info->records = lines;
        info->edges = m;
        info->duplicates = 0;
        info->parse_ms = a;
        info->build_ms = b;
    }
    return GBS_OK;
}

gbs_status ingest_bin(const char *bytes, size_t len, int direction, long long target_offset, int dedup,
                      gbs_device_csr *out, gbs_ingest_info *info) {
    if (len < 32) return fail(GBS_ERR_INVALID_ARG, "binary graph: shorter than its 32-byte header");
    long long hdr[4];
    std::memcpy(hdr, bytes, 32);
    gbs_status st = check_header(hdr);
    if (st != GBS_OK) return st;
    const unsigned long long m0 = (unsigned long long)hdr[1];
    if (len < 32 + 16 * m0) return fail(GBS_ERR_INVALID_ARG, "binary graph: fewer pairs than e_num");
    int dev = 0, sms = 0;
    ING_CUDA(cudaGetDevice(&dev));
    ING_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    cudaStream_t s;
    ING_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    struct StreamFree {
        cudaStream_t s;
        ~StreamFree() { cudaStreamDestroy(s); }
    } sf{s};
    Bufs bufs;
    cudaEvent_t ev[3];
    for (auto &e : ev) ING_CUDA(cudaEventCreate(&e));
    struct EvFree {
        cudaEvent_t *e;
        ~EvFree() {
            for (int i = 0; i < 3; ++i) cudaEventDestroy(e[i]);
        }
    } ef{ev};
    bufs.reserve((dedup ? 70 : 38) * m0 + slack(m0));
    longlong2 *pairs = nullptr;
    uint32_t *row = nullptr, *col = nullptr, *word = nullptr, *keep = nullptr, *at = nullptr;
    DevErr *d_err = nullptr, he{};
    ING_CUDA(bufs.get(&word, 2));
    ING_CUDA(bufs.get(&d_err, 1));
    ING_CUDA(bufs.get(&row, m0));
    ING_CUDA(bufs.get(&col, m0));
    const Bufs::Mark raw = bufs.mark();
    ING_CUDA(bufs.get(&pairs, m0));
    ING_CUDA(cudaEventRecord(ev[0], s));
    ING_CUDA(cudaMemcpyAsync(pairs, bytes + 32, 16 * m0, cudaMemcpyHostToDevice, s));
    ING_CUDA(cudaMemsetAsync(d_err, 0, sizeof(DevErr), s));
    const int gb = grid_for(m0, sms);
    unsigned long long m = m0;
    if (dedup && m0) {
        uint32_t mx[2] = {0, 0}, kept = 0;
        ING_CUDA(cudaMemsetAsync(word, 0, 2 * sizeof(uint32_t), s));
        k_pair_max<<<gb, 256, 0, s>>>(pairs, m0, word, d_err);
        ING_CUDA(cudaGetLastError());
        ING_CUDA(cudaMemcpyAsync(&he, d_err, sizeof(he), cudaMemcpyDeviceToHost, s));
        ING_CUDA(cudaMemcpyAsync(mx, word, sizeof(mx), cudaMemcpyDeviceToHost, s));
        ING_CUDA(cudaStreamSynchronize(s));
        st = check_err(he, "binary graph");
        if (st != GBS_OK) return st;
        ING_CUDA(bufs.get(&keep, m0 + 1));   // one more slot for the total
        ING_CUDA(bufs.get(&at, m0 + 1));
        const Bufs::Mark keys = bufs.mark();
        unsigned long long *key = nullptr, *key_s = nullptr;
        uint32_t *idx = nullptr, *idx_s = nullptr;
        ING_CUDA(bufs.get(&key, m0));
        ING_CUDA(bufs.get(&key_s, m0));
        ING_CUDA(bufs.get(&idx, m0));
        ING_CUDA(bufs.get(&idx_s, m0));
        const int to_bits = bits_of(mx[1]);
        k_pair_keys<<<gb, 256, 0, s>>>(pairs, m0, to_bits, key, idx);
        ING_CUDA(cudaGetLastError());
        st = sort_pairs<unsigned long long>(key, key_s, idx, idx_s, m0, s, bufs, bits_of(mx[0]) + to_bits);
        if (st != GBS_OK) return st;
        k_first_of_run<<<gb, 256, 0, s>>>(key_s, idx_s, m0, keep);
        ING_CUDA(cudaGetLastError());
        bufs.reset(keys);
        ING_CUDA(cudaMemsetAsync(keep + m0, 0, sizeof(uint32_t), s));
        st = excl_sum(keep, at, m0 + 1, s, bufs);
        if (st != GBS_OK) return st;
        ING_CUDA(cudaMemcpyAsync(&kept, at + m0, sizeof(kept), cudaMemcpyDeviceToHost, s));
        ING_CUDA(cudaStreamSynchronize(s));
        m = kept;
    }
    const unsigned long long dups = m0 - m;
    ING_CUDA(cudaEventRecord(ev[1], s));
    // SEND: row = from - offset, col = to - target_offset; RECV: row = to - offset, col = from - target_offset
    const bool send = direction != GBS_DIR_RECV;
    k_pair_rows<<<gb, 256, 0, s>>>(pairs, m0, keep, at, hdr[2], target_offset, !send, hdr[0], row, col, d_err);
    ING_CUDA(cudaGetLastError());
    ING_CUDA(cudaMemcpyAsync(&he, d_err, sizeof(he), cudaMemcpyDeviceToHost, s));
    ING_CUDA(cudaStreamSynchronize(s));
    st = check_err(he, "binary graph");
    if (st != GBS_OK) return st;
    bufs.reset(raw);
    ING_CUDA(cudaMalloc(&out->d_w, sizeof(double) * (m ? m : 1)));
    k_parity_weights<<<grid_for(m, sms), 256, 0, s>>>(m, out->d_w);
    ING_CUDA(cudaGetLastError());
    st = build_csr(row, col, m, (uint32_t)hdr[0], word, s, sms, bufs, out);
    if (st != GBS_OK) return st;
    ING_CUDA(cudaEventRecord(ev[2], s));
    ING_CUDA(cudaEventSynchronize(ev[2]));
    if (info) {
        float a = 0.f, b = 0.f;
        ING_CUDA(cudaEventElapsedTime(&a, ev[0], ev[1]));
        ING_CUDA(cudaEventElapsedTime(&b, ev[1], ev[2]));
        info->v_num = hdr[0];
        info->e_num = hdr[1];
        info->offset = hdr[2];
        info->g_v_size = hdr[3];
        info->records = m0;
        info->edges = m;
        info->duplicates = dups;
        info->parse_ms = a;
        info->build_ms = b;
    }
    return GBS_OK;
}

__global__ void k_iota(uint32_t *__restrict__ id, unsigned long long m) {
    for (unsigned long long k = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; k < m;
         k += (unsigned long long)gridDim.x * blockDim.x)
        id[k] = (uint32_t)k;
}

// A resident graph from device arrays: rows sorted by (weight, column) with
// stable radix passes, the columns first where some row does not have them in
// ascending order.  `host`: the arrays come from gbs_graph_create (its
// messages); else from a device CSR.  gbs_graph_create, checked and sorted by 16
// host cores -> here, ms: R-MAT 16 6.5 -> 1.1 (float64 10.8 -> 1.7), 20 116 ->
// 5.6, 22 475 -> 20.
size_t build_bytes(unsigned long long m, bool f64) { return (f64 ? 52 : 36) * m + slack(m); }

template <int WT, typename Src>
gbs_status build_graph(uint32_t n, unsigned long long m, const unsigned long long *row, const uint32_t *col, const Src *w,
                       bool host, int sms, cudaStream_t s, Bufs &bufs, gbs_graph **out) {
    constexpr gbs_weight_type wtype = WT == 2 ? GBS_WEIGHT_F64 : WT == 1 ? GBS_WEIGHT_F32 : GBS_WEIGHT_U32;
    constexpr bool f64 = WT == 2;
    const int gb = grid_for(m, sms);
    bufs.reserve(build_bytes(m, f64));
    EdgeStats *st = nullptr, hs{};
    unsigned long long *key = nullptr, *key_s = nullptr;
    uint32_t *row_of = nullptr, *row32 = nullptr;
    const int ge = grid_for((m + kEdgeTile - 1) / kEdgeTile * 32, sms);
    const uint32_t edge_warps = (uint32_t)ge * 8u;   // of 256 threads a block
    double *part = nullptr;
    ING_CUDA(bufs.get(&st, 1));
    ING_CUDA(bufs.get(&part, edge_warps));
    ING_CUDA(bufs.get(&key, m));
    ING_CUDA(bufs.get(&key_s, m));
    if (f64) ING_CUDA(bufs.get(&row_of, m));
    ING_CUDA(cudaMalloc(&row32, sizeof(uint32_t) * ((size_t)n + 1)));
    struct Guard {   // row32 becomes the graph's; until then it is freed here
        uint32_t *p;
        ~Guard() { cudaFree(p); }
    } guard{row32};
    k_edge_stats_init<<<1, 1, 0, s>>>(st);
    k_row32<<<std::max(1, std::min<int>((int)(((unsigned long long)n + 256) / 256), sms * 8)), 256, 0, s>>>(row, n, row32, st);
    k_edges<WT, Src><<<ge, 256, 0, s>>>(row, col, w, n, m, key, row_of, part, st);
    k_weight_sum<<<1, kSumTPB, 0, s>>>(part, edge_warps, st);
    ING_CUDA(cudaGetLastError());
    ING_CUDA(cudaMemcpyAsync(&hs, st, sizeof(hs), cudaMemcpyDeviceToHost, s));
    ING_CUDA(cudaStreamSynchronize(s));
    if (hs.rows_bad) return fail(GBS_ERR_INVALID_ARG, "row_offsets decrease");
    if (hs.bad != ~0ull) {
        const uint32_t why = (uint32_t)(hs.bad & 3ull);
        if (why == kBadCol) return fail(GBS_ERR_INVALID_ARG, "column index out of range");
        if (why == kBadInteger) return fail(GBS_ERR_INVALID_ARG, "uint32 graphs need integer weights below 2^32");
        return fail(GBS_ERR_INVALID_ARG, !host ? "weights must be finite and >= 0"
                                         : f64 ? "float64 weights must be finite and >= 0"
                                               : "float32 weights must be finite and >= 0");
    }
    double max_w = 0.0;
    if (WT == 0) {
        max_w = (double)hs.max_bits;
    } else if (WT == 1) {
        const uint32_t bits = (uint32_t)hs.max_bits;
        float f;
        std::memcpy(&f, &bits, 4);
        max_w = f;
    } else {
        std::memcpy(&max_w, &hs.max_bits, 8);
    }
    int bits_n = 1;
    while (bits_n < 32 && (1ull << bits_n) < n) ++bits_n;
    // columns into order first, if they are not: id then lists the edges
    uint32_t *id0 = nullptr, *id1 = nullptr, *col_s = nullptr;
    const uint32_t *cols = col;   // the columns in the order of the keys
    gbs_status r;
    if (!f64 || hs.unsorted) ING_CUDA(bufs.get(&col_s, m));
    if (f64 || hs.unsorted) {
        ING_CUDA(bufs.get(&id0, m));
        ING_CUDA(bufs.get(&id1, m));
        k_iota<<<gb, 256, 0, s>>>(id0, m);
        ING_CUDA(cudaGetLastError());
    }
    if (hs.unsorted) {
        if ((r = sort_pairs<uint32_t>(col, col_s, id0, id1, m, s, bufs, bits_n)) != GBS_OK) return r;
        std::swap(id0, id1);
        k_gather_key<unsigned long long><<<gb, 256, 0, s>>>(key, id0, m, key_s);
        ING_CUDA(cudaGetLastError());
        if (!f64) {
            std::swap(key, key_s);
            cols = col_s;
        }
    }
    gbs_graph *g = nullptr;
    if (f64) {
        // by weight, then by row; key keeps the weights in edge order.  The rows'
        // keys lie where the weights' were, so that a build holds 40 bytes an
        // edge at most
        unsigned long long *a = key_s;
        uint32_t *rk_s = reinterpret_cast<uint32_t *>(key_s);
        if (hs.unsorted) ING_CUDA(bufs.get(&a, m));
        else ING_CUDA(bufs.get(&rk_s, m));
        if ((r = sort_pairs<unsigned long long>(hs.unsorted ? key_s : key, a, id0, id1, m, s, bufs)) != GBS_OK) return r;
        uint32_t *rk = reinterpret_cast<uint32_t *>(a);
        k_gather_key<uint32_t><<<gb, 256, 0, s>>>(row_of, id1, m, rk);
        ING_CUDA(cudaGetLastError());
        if ((r = sort_pairs<uint32_t>(rk, rk_s, id1, id0, m, s, bufs, bits_n)) != GBS_OK) return r;
    } else {
        uint32_t *c_out = cols == col_s ? nullptr : col_s;
        if (!c_out) ING_CUDA(bufs.get(&c_out, m));
        if ((r = sort_pairs<unsigned long long>(key, key_s, cols, c_out, m, s, bufs, 32 + bits_n)) != GBS_OK) return r;
        cols = c_out;
    }
    if ((r = graph_shell(n, m, wtype, max_w, m ? hs.sum / (double)m : 0.0, hs.zero != 0u, &g)) != GBS_OK) return r;
    cudaError_t e = cudaMalloc(&g->d_adj, sizeof(uint2) * (m ? m : 1));
    if (e == cudaSuccess && f64) e = cudaMalloc(&g->d_w64, sizeof(unsigned long long) * (m ? m : 1));
    if (e != cudaSuccess) {
        cudaGetLastError();
        free_graph(g);
        return fail(e == cudaErrorMemoryAllocation ? GBS_ERR_NO_MEMORY : GBS_ERR_CUDA, cudaGetErrorString(e));
    }
    if (f64) k_adj64<<<gb, 256, 0, s>>>(id0, col, key, m, g->d_adj, g->d_w64);
    else k_adj32<<<gb, 256, 0, s>>>(key_s, cols, m, g->d_adj);
    if ((e = cudaGetLastError()) != cudaSuccess || (e = cudaStreamSynchronize(s)) != cudaSuccess) {
        free_graph(g);
        return fail(GBS_ERR_CUDA, cudaGetErrorString(e));
    }
    g->d_row = row32;
    guard.p = nullptr;
    g->max_deg = hs.max_deg;
    *out = g;
    return GBS_OK;
}

struct StreamOf {
    cudaStream_t s = nullptr;
    ~StreamOf() {
        if (s) cudaStreamDestroy(s);
    }
};

gbs_status graph_from_csr(const gbs_device_csr *c, gbs_weight_type wtype, gbs_graph **out) {
    if (wtype != GBS_WEIGHT_U32 && wtype != GBS_WEIGHT_F32 && wtype != GBS_WEIGHT_F64)
        return fail(GBS_ERR_INVALID_ARG, "unknown weight type");
    int dev = 0, sms = 0;
    ING_CUDA(cudaGetDevice(&dev));
    ING_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    StreamOf so;
    ING_CUDA(cudaStreamCreateWithFlags(&so.s, cudaStreamNonBlocking));
    Bufs bufs;
    if (wtype == GBS_WEIGHT_F64) return build_graph<2, double>(c->n, c->m, c->d_row, c->d_col, c->d_w, false, sms, so.s, bufs, out);
    if (wtype == GBS_WEIGHT_F32) return build_graph<1, double>(c->n, c->m, c->d_row, c->d_col, c->d_w, false, sms, so.s, bufs, out);
    return build_graph<0, double>(c->n, c->m, c->d_row, c->d_col, c->d_w, false, sms, so.s, bufs, out);
}

gbs_status graph_from_host(uint32_t n, uint64_t m, const uint64_t *row, const uint32_t *cols, const void *weights,
                           gbs_weight_type wtype, gbs_graph **out) {
    int dev = 0, sms = 0;
    ING_CUDA(cudaGetDevice(&dev));
    ING_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    StreamOf so;
    ING_CUDA(cudaStreamCreateWithFlags(&so.s, cudaStreamNonBlocking));
    Bufs bufs;
    const size_t wb = dist_bytes(wtype);
    unsigned long long *d_row = nullptr;
    uint32_t *d_col = nullptr;
    char *d_w = nullptr;
    bufs.reserve(8ull * n + (4 + wb) * m + build_bytes(m, wtype == GBS_WEIGHT_F64));
    ING_CUDA(bufs.get(&d_row, (size_t)n + 1));
    ING_CUDA(bufs.get(&d_col, m));
    ING_CUDA(bufs.get(&d_w, wb * m));
    ING_CUDA(cudaMemcpyAsync(d_row, row, 8ull * ((size_t)n + 1), cudaMemcpyHostToDevice, so.s));
    if (m) {
        ING_CUDA(cudaMemcpyAsync(d_col, cols, 4ull * m, cudaMemcpyHostToDevice, so.s));
        ING_CUDA(cudaMemcpyAsync(d_w, weights, wb * m, cudaMemcpyHostToDevice, so.s));
    }
    if (wtype == GBS_WEIGHT_F64)
        return build_graph<2, double>(n, m, d_row, d_col, reinterpret_cast<double *>(d_w), true, sms, so.s, bufs, out);
    if (wtype == GBS_WEIGHT_F32)
        return build_graph<1, float>(n, m, d_row, d_col, reinterpret_cast<float *>(d_w), true, sms, so.s, bufs, out);
    return build_graph<0, uint32_t>(n, m, d_row, d_col, reinterpret_cast<uint32_t *>(d_w), true, sms, so.s, bufs, out);
}

}  // namespace gbs

// ===================================================================== C ABI
extern "C" {

// Not part of the public header: makes a reader or a graph build on this thread
// that would hold more bytes fail as on a full device, or (memory 0) with
// another error (bytes 0: no limit).
void gbs_test_buffer_limit(size_t bytes, int memory) {
    gbs::t_buffer_limit = bytes ? bytes : SIZE_MAX;
    gbs::t_limit_is_memory = memory != 0;
}

gbs_status gbs_parse_text(const char *bytes, size_t len, int direction, gbs_device_csr **out, gbs_ingest_info *info) {
    if (!out || (len && !bytes)) return gbs::fail(GBS_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    gbs_device_csr *c = new gbs_device_csr();
    const gbs_status st = gbs::ingest_text(bytes, len, direction, c, info);
    if (st != GBS_OK) {
        gbs_device_csr_destroy(c);
        return st;
    }
    *out = c;
    return GBS_OK;
}

gbs_status gbs_parse_bin(const void *bytes, size_t len, int direction, int64_t target_offset, int dedup,
                         gbs_device_csr **out, gbs_ingest_info *info) {
    if (!out || (len && !bytes)) return gbs::fail(GBS_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    gbs_device_csr *c = new gbs_device_csr();
    const gbs_status st = gbs::ingest_bin(static_cast<const char *>(bytes), len, direction, target_offset, dedup, c, info);
    if (st != GBS_OK) {
        gbs_device_csr_destroy(c);
        return st;
    }
    *out = c;
    return GBS_OK;
}

static gbs_status read_whole(const char *path, char **pinned, std::vector<char> &host, size_t &len, double &ms) {
    const auto t0 = std::chrono::steady_clock::now();
    const gbs_status st = gbs::read_file(path, host, pinned, len);
    ms = gbs::ms_since(t0);
    return st;
}

gbs_status gbs_read_text(const char *path, int direction, gbs_device_csr **out, gbs_ingest_info *info) {
    if (!path || !out) return gbs::fail(GBS_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    gbs::PinnedFree pf;
    std::vector<char> host;
    size_t len = 0;
    double ms = 0.0;
    gbs_status st = read_whole(path, &pf.p, host, len, ms);
    if (st != GBS_OK) return st;
    st = gbs_parse_text(pf.p ? pf.p : host.data(), len, direction, out, info);
    if (st == GBS_OK && info) info->read_ms = ms;
    return st;
}

gbs_status gbs_read_bin(const char *path, int direction, int64_t target_offset, int dedup, gbs_device_csr **out,
                        gbs_ingest_info *info) {
    if (!path || !out) return gbs::fail(GBS_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    gbs::PinnedFree pf;
    std::vector<char> host;
    size_t len = 0;
    double ms = 0.0;
    gbs_status st = read_whole(path, &pf.p, host, len, ms);
    if (st != GBS_OK) return st;
    st = gbs_parse_bin(pf.p ? pf.p : host.data(), len, direction, target_offset, dedup, out, info);
    if (st == GBS_OK && info) info->read_ms = ms;
    return st;
}

gbs_status gbs_device_csr_info(const gbs_device_csr *c, uint32_t *n, uint64_t *m) {
    if (!c) return gbs::fail(GBS_ERR_INVALID_ARG, "csr is NULL");
    if (n) *n = c->n;
    if (m) *m = c->m;
    return GBS_OK;
}

gbs_status gbs_device_csr_export(const gbs_device_csr *c, uint64_t *row_offsets, uint32_t *cols, double *weights) {
    if (!c) return gbs::fail(GBS_ERR_INVALID_ARG, "csr is NULL");
    if (row_offsets)
        GBS_CUDA(cudaMemcpy(row_offsets, c->d_row, sizeof(uint64_t) * ((size_t)c->n + 1), cudaMemcpyDeviceToHost));
    if (cols && c->m) GBS_CUDA(cudaMemcpy(cols, c->d_col, sizeof(uint32_t) * c->m, cudaMemcpyDeviceToHost));
    if (weights && c->m) GBS_CUDA(cudaMemcpy(weights, c->d_w, sizeof(double) * c->m, cudaMemcpyDeviceToHost));
    return GBS_OK;
}

gbs_status gbs_graph_from_device_csr(const gbs_device_csr *c, gbs_weight_type wtype, gbs_graph **out) {
    if (!c || !out) return gbs::fail(GBS_ERR_INVALID_ARG, "NULL argument");
    *out = nullptr;
    return gbs::graph_from_csr(c, wtype, out);
}

gbs_status gbs_device_csr_destroy(gbs_device_csr *c) {
    if (!c) return gbs::fail(GBS_ERR_INVALID_ARG, "csr is NULL");
    cudaFree(c->d_row);
    cudaFree(c->d_col);
    cudaFree(c->d_w);
    delete c;
    return GBS_OK;
}

}  // extern "C"
