// march_ny2.cu -- instantiation of the column march for NY = 2, 3x3 blocks
#include "march.cuh"

namespace cb {
template int run_x1march<2, 3>(const Geom &, const canoe_thermo_t &, int, int, int,
                               const double *, const double *, double *, const double *,
                               const Stage &, int, cudaStream_t);
}  // namespace cb
