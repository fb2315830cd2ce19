// march5_ny0.cu -- instantiation of the column march for NY = 0, 5x5 blocks
#include "march.cuh"

namespace cb {
template int run_x1march<0, 5>(const Geom &, const canoe_thermo_t &, int, int, int,
                               const double *, const double *, double *, const double *,
                               const Stage &, int, cudaStream_t);
}  // namespace cb
