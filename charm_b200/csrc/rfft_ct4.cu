// Row transforms of the compile-time plans M = 3456, 4096, 4608 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

bool launch_rfft_ct4(const RfftArgs &A, bool inverse, cudaStream_t st,
                     cudaError_t *e)
{
    switch (A.M)
    {
    case 3456: *e = rfft_ct_launch<3456>(A, inverse, st); return true;
    case 4096: *e = rfft_ct_launch<4096>(A, inverse, st); return true;
    case 4608: *e = rfft_ct_launch<4608>(A, inverse, st); return true;
    default: return false;
    }
}

} // namespace cb
