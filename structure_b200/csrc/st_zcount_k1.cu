// st_zcount_k1.cu -- counting Z pass for K classes 1, 2, 3, 4.
#include "st_zcount.cuh"

namespace st {
namespace zcount {
template cudaError_t launch_zcount_k<1>(const LaunchSet&, int, int, size_t);
template cudaError_t launch_zcount_k<2>(const LaunchSet&, int, int, size_t);
template cudaError_t launch_zcount_k<3>(const LaunchSet&, int, int, size_t);
template cudaError_t launch_zcount_k<4>(const LaunchSet&, int, int, size_t);

size_t zc_layout_total(int kt, int T) { return (size_t)zc_layout(kt, T).total; }
int zc_ctas_of(int kt) { return zc_ctas(kt); }
}  // namespace zcount
}  // namespace st
