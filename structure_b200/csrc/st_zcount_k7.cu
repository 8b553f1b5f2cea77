// st_zcount_k7.cu -- counting Z pass for K classes 24, 32.
#include "st_zcount.cuh"

namespace st {
namespace zcount {
template cudaError_t launch_zcount_k<24>(const LaunchSet&, int, int, size_t);
template cudaError_t launch_zcount_k<32>(const LaunchSet&, int, int, size_t);
}  // namespace zcount
}  // namespace st
