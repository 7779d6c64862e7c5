// Eikonal solve kernels: the second order scheme (see families.cuh).
#include "solve.cuh"

namespace agd {
template int solve<fam::O2>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::O3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
}  // namespace agd
