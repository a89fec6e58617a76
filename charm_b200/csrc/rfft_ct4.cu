// Row transforms of the compile-time plans M = 3456, 4096, 4608 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

cudaError_t launch_rfft_ct4(const RfftArgs &A, bool inverse, cudaStream_t st)
{
    switch (A.M)
    {
    case 3456: return rfft_ct_launch<3456>(A, inverse, st);
    case 4096: return rfft_ct_launch<4096>(A, inverse, st);
    case 4608: return rfft_ct_launch<4608>(A, inverse, st);
    default: return cudaErrorInvalidConfiguration;
    }
}

} // namespace cb
