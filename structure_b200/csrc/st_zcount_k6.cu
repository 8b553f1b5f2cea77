// st_zcount_k6.cu -- counting Z pass for K classes 16, 20.
#include "st_zcount.cuh"

namespace st {
namespace zcount {
template cudaError_t launch_zcount_k<16>(const LaunchSet&, int, int, size_t);
template cudaError_t launch_zcount_k<20>(const LaunchSet&, int, int, size_t);
}  // namespace zcount
}  // namespace st
