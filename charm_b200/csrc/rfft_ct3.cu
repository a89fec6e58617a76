// Row transforms of the compile-time plans M = 2048, 2304, 3072 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

bool launch_rfft_ct3(const RfftArgs &A, bool inverse, cudaStream_t st,
                     cudaError_t *e)
{
    switch (A.M)
    {
    case 2048: *e = rfft_ct_launch<2048>(A, inverse, st); return true;
    case 2304: *e = rfft_ct_launch<2304>(A, inverse, st); return true;
    case 3072: *e = rfft_ct_launch<3072>(A, inverse, st); return true;
    default: return false;
    }
}

} // namespace cb
