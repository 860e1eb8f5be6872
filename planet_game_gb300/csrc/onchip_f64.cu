// The on-chip solves in FP64: see onchip_kernel.cuh.
#include "onchip_kernel.cuh"

namespace psgb {

template bool onchip_has<double>(int);
template int onchip_active_clusters<double>(int, unsigned, unsigned, std::size_t);
template void onchip_launch<double>(const OnchipArgs<double>&, int, unsigned, std::size_t, cudaStream_t);

}  // namespace psgb
