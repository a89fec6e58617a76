// Row transforms of the compile-time plans M = 8192, 9216 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

bool launch_rfft_ct6(const RfftArgs &A, bool inverse, cudaStream_t st,
                     cudaError_t *e)
{
    switch (A.M)
    {
    case 8192: *e = rfft_ct_launch<8192>(A, inverse, st); return true;
    case 9216: *e = rfft_ct_launch<9216>(A, inverse, st); return true;
    default: return false;
    }
}

} // namespace cb
