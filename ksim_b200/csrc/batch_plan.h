// batch_plan.h — what a batch's items cost (host code only, free of
// CUDA, so the CPU tests check it directly).
#pragma once

#include <algorithm>
#include <cstdint>

namespace ksim {

// Microseconds of an item, roughly, whichever body runs it: the items of one
// list go longest first, and the groups' kernels by their longest item.
// A sliced tile of 1,024 shots takes about 0.9 us a term, one of 512 shots
// 0.83 and one of 256 0.75 of that.
inline double slice_item_us(int64_t terms, int shots)
{
    return 0.9 * (double)terms * (shots >= 1024 ? 1.0 : shots >= 512 ? 0.83 : 0.75);
}
// A term-record tile goes by its stream's bytes and its shots: 256 shots of a
// term of about 2 KB take 3.0 us with the SMs full (306 terms 0.92 ms).
inline double record_item_us(double stream_bytes, int64_t shots)
{
    return 3.0 / (2088.0 * 256.0) * stream_bytes * (double)shots;
}

}  // namespace ksim
