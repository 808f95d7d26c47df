// Ragged-pencil kernels, EXACT policy (see mhd_ragged.cuh); compiled with --fmad=false
#include "mhd_ragged.cuh"

namespace mhd {

cudaError_t fluidx_rag_exact(const FluidxArgs& a, const RagShape& sh, int pb, cudaStream_t s)
{
    return fluidx_rag_set<true>(a, sh, pb, s);
}

cudaError_t advect_rag_exact(const AdvectArgs& a, const RagShape& sh, int pb, bool wu, cudaStream_t s)
{
    return advect_rag_set<true>(a, sh, pb, wu, s);
}

}  // namespace mhd
