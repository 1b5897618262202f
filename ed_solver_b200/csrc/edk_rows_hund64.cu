// Row kernel with bulk-copy row staging: FP64 instances with Hund terms.
#include "edk_rows_tma_inst.cuh"

namespace edk {

cudaError_t launch_hund_f64(const HamDev &H, const RowArgs &a, int num_sms, const FastShape &s, cudaStream_t st)
{
    EDK_TMA_HUND_ALL(double)
    return cudaErrorInvalidValue;
}

}  // namespace edk
