// st_zmetro_k3.cu -- Metropolis pass for K classes 16, 20, 24, 32.
#include "st_zmetro.cuh"

namespace st {
namespace zmetro {
template cudaError_t launch_zmetro_k<16>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<20>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<24>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<32>(const LaunchSet&, int, size_t);
}  // namespace zmetro
}  // namespace st
