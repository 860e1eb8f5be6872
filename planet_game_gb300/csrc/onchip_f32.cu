// The on-chip solves in FP32: see onchip_kernel.cuh.
#include "onchip_kernel.cuh"

namespace psgb {

template bool onchip_has<float>(int);
template int onchip_active_clusters<float>(int, unsigned, unsigned, std::size_t);
template void onchip_launch<float>(const OnchipArgs<float>&, int, unsigned, std::size_t, cudaStream_t);

}  // namespace psgb
