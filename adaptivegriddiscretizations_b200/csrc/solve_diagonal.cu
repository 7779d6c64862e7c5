// Eikonal solve kernels: the Diagonal models (see families.cuh).
#include "solve.cuh"

namespace agd {
template int solve<fam::D2>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::D3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::DMP2>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::DMP3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::DF2>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::DF3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::DO2>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
template int solve<fam::DO3>(const WsLayout &, void *, int, agd_stats *, const agd_launch *, cudaStream_t);
}  // namespace agd
