// heavy_parts.h — which of kSub parts of a square's extent a coordinate lies in (the heavy pairs'
// search of basins_ref.cu; host code too, for its test).
#pragma once

#ifdef __CUDACC__
#define UCB_PARTS_FN __host__ __device__ __forceinline__
#else
#define UCB_PARTS_FN inline
#endif

namespace ucbbr {

constexpr int kSub = 16;

// Parts a unit of an extent of `width`. 0 (everything in part 0, whose box then covers the whole
// extent) for an extent without width, and where the quotient overflows, below 16 / DBL_MAX: there
// the lowest cell's 0 x infinity would have no part.
UCB_PARTS_FN double part_scale(double width) {
    const double s = kSub / width;
    return width > 0 && s <= 1.7976931348623157e308 ? s : 0;
}

UCB_PARTS_FN int part_index(double offset, double scale) {
    const int i = (int)(offset * scale);
    return i < 0 ? 0 : i < kSub ? i : kSub - 1;
}

}  // namespace ucbbr
