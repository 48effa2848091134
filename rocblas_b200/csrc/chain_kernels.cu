// The chain solve's kernels (trsm_chain.cuh), compiled apart from the entry points so that the
// library's parts build in parallel.
#include "trsm_chain.cuh"

namespace rb200
{

template void launch_chain_w<double, 8, false>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<double, 16, false>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<double, 32, false>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<double, 64, false>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<double, 32, true>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<double, 64, true>(const ChainParams<double>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<float, 8, false>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<float, 16, false>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<float, 32, false>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<float, 64, false>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<float, 32, true>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);
template void launch_chain_w<float, 64, true>(const ChainParams<float>&, bool, bool, int, int64_t, cudaStream_t, bool);

} // namespace rb200
