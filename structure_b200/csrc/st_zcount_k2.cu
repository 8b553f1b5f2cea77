// st_zcount_k2.cu -- counting Z pass for K classes 5, 6.
#include "st_zcount.cuh"

namespace st {
namespace zcount {
template cudaError_t launch_zcount_k<5>(const LaunchSet&, int, int, size_t);
template cudaError_t launch_zcount_k<6>(const LaunchSet&, int, int, size_t);
}  // namespace zcount
}  // namespace st
