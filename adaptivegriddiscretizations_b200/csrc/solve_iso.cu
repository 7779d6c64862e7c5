// Eikonal solve kernels: Isotropic2 and Isotropic3 (see families.cuh).
#include "solve.cuh"

namespace agd {
template int solve<fam::I16>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::I8>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::I3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
}  // namespace agd
