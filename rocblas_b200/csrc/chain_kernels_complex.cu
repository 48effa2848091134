// The chain solve's kernels for complex types (trsm_chain.cuh), compiled apart from the entry points
// so that the library's parts build in parallel.
#include "trsm_chain.cuh"

namespace rb200
{

template void launch_chain_w<cplx<double>, 8, false>(const ChainParams<cplx<double>>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<cplx<double>, 16, false>(const ChainParams<cplx<double>>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<cplx<double>, 32, false>(const ChainParams<cplx<double>>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<cplx<double>, 64, false>(const ChainParams<cplx<double>>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<cplx<float>, 8, false>(const ChainParams<cplx<float>>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<cplx<float>, 16, false>(const ChainParams<cplx<float>>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<cplx<float>, 32, false>(const ChainParams<cplx<float>>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<cplx<float>, 64, false>(const ChainParams<cplx<float>>&, bool, bool, int, int64_t, cudaStream_t, bool);

} // namespace rb200
