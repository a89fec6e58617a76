// Row transforms of the compile-time plans M = 8192, 9216 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

cudaError_t launch_rfft_ct6(const RfftArgs &A, bool inverse, cudaStream_t st)
{
    switch (A.M)
    {
    case 8192: return rfft_ct_launch<8192>(A, inverse, st);
    case 9216: return rfft_ct_launch<9216>(A, inverse, st);
    default: return cudaErrorInvalidConfiguration;
    }
}

} // namespace cb
