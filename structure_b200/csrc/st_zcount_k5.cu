// st_zcount_k5.cu -- counting Z pass for K classes 11, 12.
#include "st_zcount.cuh"

namespace st {
namespace zcount {
template cudaError_t launch_zcount_k<11>(const LaunchSet&, int, int, size_t);
template cudaError_t launch_zcount_k<12>(const LaunchSet&, int, int, size_t);
}  // namespace zcount
}  // namespace st
