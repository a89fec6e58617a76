// Row transforms of the compile-time plans M = 512, 576, 768, 1024 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

cudaError_t launch_rfft_ct1(const RfftArgs &A, bool inverse, cudaStream_t st)
{
    switch (A.M)
    {
    case 512: return rfft_ct_launch<512>(A, inverse, st);
    case 576: return rfft_ct_launch<576>(A, inverse, st);
    case 768: return rfft_ct_launch<768>(A, inverse, st);
    case 1024: return rfft_ct_launch<1024>(A, inverse, st);
    default: return cudaErrorInvalidConfiguration;
    }
}

} // namespace cb
