// st_zcount_k4.cu -- counting Z pass for K classes 9, 10.
#include "st_zcount.cuh"

namespace st {
namespace zcount {
template cudaError_t launch_zcount_k<9>(const LaunchSet&, int, int, size_t);
template cudaError_t launch_zcount_k<10>(const LaunchSet&, int, int, size_t);
}  // namespace zcount
}  // namespace st
