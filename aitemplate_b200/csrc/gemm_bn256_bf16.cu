// Instantiations of the tcgen05 GEMM kernel for 256-column output tiles in bfloat16 (see gemm_kernel.cuh).
#include "gemm_kernel.cuh"

namespace b200ait {
#define B200AIT_CASE_BF16_256(CODE)                              \
  case (CODE):                                                  \
    launch_tc<256, true, (CODE)>(ta, tb, tout, p, grid, stream); \
    break;
B200AIT_DEFINE_LAUNCH_TC_WIDTH_BF16(256)
#undef B200AIT_CASE_BF16_256
}  // namespace b200ait
