// Row transforms of the compile-time plans M = 5184, 6912 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

bool launch_rfft_ct5(const RfftArgs &A, bool inverse, cudaStream_t st,
                     cudaError_t *e)
{
    switch (A.M)
    {
    case 5184: *e = rfft_ct_launch<5184>(A, inverse, st); return true;
    case 6912: *e = rfft_ct_launch<6912>(A, inverse, st); return true;
    default: return false;
    }
}

} // namespace cb
