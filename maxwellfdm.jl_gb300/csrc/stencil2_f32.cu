// The second operator kernel in complex64 (a translation unit per precision, so that
// both compile at the same time).
#include "stencil2.cuh"

namespace fdfd {

template int launch_apply_v2<float>(fdfd_handle *, const float2 *, float2 *, int, const float2 *, int, KScalars *, int, bool);

}  // namespace fdfd
