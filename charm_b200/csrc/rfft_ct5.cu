// Row transforms of the compile-time plans M = 5184, 6912 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

cudaError_t launch_rfft_ct5(const RfftArgs &A, bool inverse, cudaStream_t st)
{
    switch (A.M)
    {
    case 5184: return rfft_ct_launch<5184>(A, inverse, st);
    case 6912: return rfft_ct_launch<6912>(A, inverse, st);
    default: return cudaErrorInvalidConfiguration;
    }
}

} // namespace cb
