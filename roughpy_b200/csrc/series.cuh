// Row-resident Horner series: exp, fmexp and log of dense free tensors in one
// launch, for shapes whose lower levels fit in shared memory.
#pragma once

#include "common.cuh"

namespace rpyb {

enum SeriesKind { kSeriesExp = 0, kSeriesFmexp = 1, kSeriesLog = 2 };

struct SeriesRows {
    void* out = nullptr;          // levels 0..top are written
    const void* arg = nullptr;
    const void* mult = nullptr;   // fmexp only
    int64_t ld_out = 0, ld_arg = 0, ld_mult = 0;
    int64_t batch = 0;
    bool fresh = false;           // log: take out[0] as zero
};

// Whether series of `top` levels of this shape run in the row-resident kernel.
bool series_available(const Geometry& g, int top);

// Whether one product launch a step is faster there for this batch.
bool series_slower(int dtype, SeriesKind kind, const Geometry& g, int top, int64_t batch);

// out <- exp(arg), mult exp(arg) or log(arg), truncated at level `top` (>= 1);
// levels of arg above arg_max count as zero (log).  The level-0 rules are
// those of the product-launch drivers: exp writes 1, fmexp the multiplier's
// scalar, log 0 (its incoming out[0] joins the first coefficient).
int launch_series(int dtype, SeriesKind kind, const Geometry& g, int top, int arg_max,
                  const SeriesRows& rows, cudaStream_t stream);

}  // namespace rpyb
