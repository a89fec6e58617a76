// Row transforms of the compile-time plans M = 2048, 2304, 3072 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

cudaError_t launch_rfft_ct3(const RfftArgs &A, bool inverse, cudaStream_t st)
{
    switch (A.M)
    {
    case 2048: return rfft_ct_launch<2048>(A, inverse, st);
    case 2304: return rfft_ct_launch<2304>(A, inverse, st);
    case 3072: return rfft_ct_launch<3072>(A, inverse, st);
    default: return cudaErrorInvalidConfiguration;
    }
}

} // namespace cb
