// simt_kernel_tn.cu -- the persistent FP32 SIMT kernel, A stored K x M.
#define BGEMM_SIMT_TA true
#define BGEMM_SIMT_TB false
#define BGEMM_SIMT_LAUNCH simt_launch_tn
#include "simt_kernel_t.h"
