// Row transforms of the compile-time plans M = 512, 576, 768, 1024 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

bool launch_rfft_ct1(const RfftArgs &A, bool inverse, cudaStream_t st,
                     cudaError_t *e)
{
    switch (A.M)
    {
    case 512: *e = rfft_ct_launch<512>(A, inverse, st); return true;
    case 576: *e = rfft_ct_launch<576>(A, inverse, st); return true;
    case 768: *e = rfft_ct_launch<768>(A, inverse, st); return true;
    case 1024: *e = rfft_ct_launch<1024>(A, inverse, st); return true;
    default: return false;
    }
}

} // namespace cb
