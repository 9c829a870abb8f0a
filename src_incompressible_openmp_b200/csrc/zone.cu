// The zone kernels, apart from capi.cu so that the two compile side by side.
#include "zone_body.cuh"

namespace mpcd_dev {

template __global__ void k_zone_pass<false>(ZoneArgs);
template __global__ void k_zone_pass<true>(ZoneArgs);
template __global__ void k_zone_pass_sync<false, 4>(ZoneArgs, int);
template __global__ void k_zone_pass_sync<false, 8>(ZoneArgs, int);
template __global__ void k_zone_pass_sync<false, 16>(ZoneArgs, int);
template __global__ void k_zone_pass_sync<true, 4>(ZoneArgs, int);
template __global__ void k_zone_pass_sync<true, 8>(ZoneArgs, int);
template __global__ void k_zone_pass_sync<true, 16>(ZoneArgs, int);
template __global__ void k_zone_pass_batch<false>(const ZoneArgs* __restrict__, const int* __restrict__, int);
template __global__ void k_zone_overflow<false>(ZoneArgs, char*, size_t, int*, double*);
template __global__ void k_zone_overflow<true>(ZoneArgs, char*, size_t, int*, double*);

}  // namespace mpcd_dev
