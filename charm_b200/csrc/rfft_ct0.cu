// Row transforms of the compile-time plans M = 64, 128, 192, 256, 384 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

bool launch_rfft_ct0(const RfftArgs &A, bool inverse, cudaStream_t st,
                     cudaError_t *e)
{
    switch (A.M)
    {
    case 64: *e = rfft_ct_launch<64>(A, inverse, st); return true;
    case 128: *e = rfft_ct_launch<128>(A, inverse, st); return true;
    case 192: *e = rfft_ct_launch<192>(A, inverse, st); return true;
    case 256: *e = rfft_ct_launch<256>(A, inverse, st); return true;
    case 384: *e = rfft_ct_launch<384>(A, inverse, st); return true;
    default: return false;
    }
}

} // namespace cb
