// The second operator kernel in complex128 (a translation unit per precision, so that
// both compile at the same time).
#include "stencil2.cuh"

namespace fdfd {

template int launch_apply_v2<double>(fdfd_handle *, const double2 *, double2 *, int, const double2 *, int, KScalars *, int, bool);

}  // namespace fdfd
