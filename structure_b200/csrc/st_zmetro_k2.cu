// st_zmetro_k2.cu -- Metropolis pass for K classes 7, 8, 9, 10, 11, 12.
#include "st_zmetro.cuh"

namespace st {
namespace zmetro {
template cudaError_t launch_zmetro_k<7>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<8>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<9>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<10>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<11>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<12>(const LaunchSet&, int, size_t);
}  // namespace zmetro
}  // namespace st
