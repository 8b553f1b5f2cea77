// st_zmetro_k1.cu -- Metropolis pass for K classes 1, 2, 3, 4, 5, 6.
#include "st_zmetro.cuh"

namespace st {
namespace zmetro {
template cudaError_t launch_zmetro_k<1>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<2>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<3>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<4>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<5>(const LaunchSet&, int, size_t);
template cudaError_t launch_zmetro_k<6>(const LaunchSet&, int, size_t);

size_t layout_total(int kt, int T) { return (size_t)layout(kt, T).total; }
}  // namespace zmetro
}  // namespace st
