// Eikonal solve kernels: Riemann2, plain and with walls (see families.cuh).
#include "solve.cuh"

namespace agd {
template int solve<fam::R2>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::R2L>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::R2W>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
}  // namespace agd
