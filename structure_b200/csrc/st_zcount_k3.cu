// st_zcount_k3.cu -- counting Z pass for K classes 7, 8.
#include "st_zcount.cuh"

namespace st {
namespace zcount {
template cudaError_t launch_zcount_k<7>(const LaunchSet&, int, int, size_t);
template cudaError_t launch_zcount_k<8>(const LaunchSet&, int, int, size_t);
}  // namespace zcount
}  // namespace st
