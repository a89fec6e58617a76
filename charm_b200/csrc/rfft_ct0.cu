// Row transforms of the compile-time plans M = 64, 128, 192, 256, 384 (rfft.cuh).
#include "rfft.cuh"

namespace cb
{

cudaError_t launch_rfft_ct0(const RfftArgs &A, bool inverse, cudaStream_t st)
{
    switch (A.M)
    {
    case 64: return rfft_ct_launch<64>(A, inverse, st);
    case 128: return rfft_ct_launch<128>(A, inverse, st);
    case 192: return rfft_ct_launch<192>(A, inverse, st);
    case 256: return rfft_ct_launch<256>(A, inverse, st);
    case 384: return rfft_ct_launch<384>(A, inverse, st);
    default: return cudaErrorInvalidConfiguration;
    }
}

} // namespace cb
