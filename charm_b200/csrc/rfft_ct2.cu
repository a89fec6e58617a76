// Row transforms of the compile-time plans M = 1152, 1536, 1728 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

cudaError_t launch_rfft_ct2(const RfftArgs &A, bool inverse, cudaStream_t st)
{
    switch (A.M)
    {
    case 1152: return rfft_ct_launch<1152>(A, inverse, st);
    case 1536: return rfft_ct_launch<1536>(A, inverse, st);
    case 1728: return rfft_ct_launch<1728>(A, inverse, st);
    default: return cudaErrorInvalidConfiguration;
    }
}

} // namespace cb
