// The FP64 GEMM tiles (gemm_dmma.cuh), compiled apart from the entry points so that the
// library's parts build in parallel.
#include "gemm_dmma.cuh"

namespace rb200
{

template void launch_dmma_tile<false, false>(DmmaTile, const GemmParams<double>&, int, cudaStream_t);
template void launch_dmma_tile<false, true>(DmmaTile, const GemmParams<double>&, int, cudaStream_t);
template void launch_dmma_tile<true, false>(DmmaTile, const GemmParams<double>&, int, cudaStream_t);
template void launch_dmma_tile<true, true>(DmmaTile, const GemmParams<double>&, int, cudaStream_t);

} // namespace rb200
