// Row transforms of the compile-time plans M = 1152, 1536, 1728 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

bool launch_rfft_ct2(const RfftArgs &A, bool inverse, cudaStream_t st,
                     cudaError_t *e)
{
    switch (A.M)
    {
    case 1152: *e = rfft_ct_launch<1152>(A, inverse, st); return true;
    case 1536: *e = rfft_ct_launch<1536>(A, inverse, st); return true;
    case 1728: *e = rfft_ct_launch<1728>(A, inverse, st); return true;
    default: return false;
    }
}

} // namespace cb
