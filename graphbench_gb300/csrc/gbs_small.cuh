// gbs_small.cuh -- host interface of the one-CTA solver for graphs whose whole
// search state fits in shared memory (gbs_small.cu).
#pragma once

#include "gbs_host.hpp"

namespace gbs {

// Shared-memory limits of a launch that solves graphs of at most n vertices
// and m edges.
struct SmallShape {
    uint32_t n_cap;        // vertices
    uint32_t piece_cap;    // pieces of long rows in one sweep
    size_t bytes;          // dynamic shared memory of a CTA
};
SmallShape small_shape(uint32_t n, uint64_t m);

// Whether a graph is solved by one CTA when the caller left every knob of the
// schedule at its default: uint32 or float32 weights, the size below for its
// weights (mean_w: their mean) and, in a plan, the number of instances (0: a
// call of its own), and (for uint32) no path sum that could pass 2^32 - 1.
bool small_graph(gbs_weight_type wt, uint32_t n, uint64_t m, double max_w, double mean_w, uint32_t instances);

// Whether this call runs on one CTA: a small graph and no knob set that would
// shape the run (a delta that resolves to the default width is the default; the
// light bound shapes only runs that set full_items, as in the persistent kernel).
bool small_call(const gbs_graph *g, const gbs_params *p);

// One source of a resident graph: dist / pred (device or mapped host memory,
// either may be null) and the statistics, in one launch on g->stream.  `light`:
// the caller's bound, for the statistics.
gbs_status small_run(gbs_graph *g, uint32_t src, void *dist, int32_t *pred, double light, bool want_stats,
                     gbs_stats *stats);

// Instances of a plan: one CTA per instance, taken from `queue` until `count`
// are done.  The grid for a shape, and the launch (capturable).
uint32_t small_grid(bool f32, const SmallShape &shape, int sms, uint32_t count);
gbs_status small_launch(bool f32, const SmallShape &shape, uint32_t grid, const InstDesc *inst, InstResult *res,
                        uint32_t count, uint32_t *queue, cudaStream_t s);

}  // namespace gbs
