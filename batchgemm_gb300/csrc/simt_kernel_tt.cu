// simt_kernel_tt.cu -- the persistent FP32 SIMT kernel, both operands stored transposed.
#define BGEMM_SIMT_TA true
#define BGEMM_SIMT_TB true
#define BGEMM_SIMT_LAUNCH simt_launch_tt
#include "simt_kernel_t.h"
