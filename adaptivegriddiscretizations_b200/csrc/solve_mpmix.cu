// Eikonal solve kernels: plans that mix multiprecision and plain variants (see families.cuh).
#include "solve.cuh"

namespace agd {
template int solve<fam::MP2>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::MP3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
}  // namespace agd
