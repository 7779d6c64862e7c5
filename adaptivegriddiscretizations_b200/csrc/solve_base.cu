// Eikonal solve kernels: plans that mix the plain variants (see families.cuh).
#include "solve.cuh"

namespace agd {
template int solve<fam::BASE2>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::BASE3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
}  // namespace agd
