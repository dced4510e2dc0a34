// gg_internal.h -- declarations shared by the library's translation units (not
// part of the C ABI; hidden symbols).
#pragma once
#include <cstdint>
#include <string>
#include <vector>
#include <cuda_runtime.h>

#include "gg.h"

namespace gg {

// Options of an evaluation that only the library's own modules use.
struct EvalExtra {
    const int32_t *inv = nullptr;  // device [rows]: source index of each vertex (-1: none)
    int ns = 0;                    // sources in that list
    uint4 *planes = nullptr;       // distance bit-planes to write (every source, in order)
    int nplanes = 0;
    bool no_graph = false;         // launch directly, neither capture nor replay
    uint64_t *within = nullptr;    // host [2]: total distance and number of the pairs whose vertex is a
                                   // source of the list too (diagonal included); needs `inv`, and a
                                   // plain-graph table that is range-checked already (read in place)
};

__attribute__((visibility("hidden"))) void set_last_error(const char *msg);

// Autotuner cache (gg_tune.cpp): key = GPU name and SM count, evaluator, shape.
__attribute__((visibility("hidden"))) std::string tune_key(int device, const char *what,
                                                         const std::vector<long long> &dims);
__attribute__((visibility("hidden"))) bool tune_get(const std::string &key, std::vector<int> *vals);
__attribute__((visibility("hidden"))) void tune_put(const std::string &key, const std::vector<int> &vals);

// gg_graph_create for an engine that only engine_eval runs, with options that need the level loop.
__attribute__((visibility("hidden"))) gg_status graph_engine(int n, int d, int device, gg_engine **out);

// One evaluation of `e` on the device table `d_table` (on stream `st`, blocking),
// with the extra options `x` (nullptr: none).
__attribute__((visibility("hidden"))) gg_status engine_eval(gg_engine *e, const int32_t *d_table,
                                                          const gg_eval_opts *o, gg_result *r,
                                                          cudaStream_t st, const EvalExtra *x);

// Columns (chunks of 128 sources) of the distance planes an evaluation of every
// source writes, and the engine's rows.
__attribute__((visibility("hidden"))) int engine_plane_cols(const gg_engine *e);

}  // namespace gg
