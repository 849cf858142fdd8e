// The bucket layouts of two-byte slots.
#include "sqf_layout.cuh"

namespace gqf {

template int launch_layout<2>(const LayoutPlan &, const SqfGeom &, uint8_t *, const BucketSrc &, const BucketSrc &, int,
                              int, bool, const uint32_t *, Scratch &, uint32_t *, cudaStream_t, const uint32_t *);

}  // namespace gqf
