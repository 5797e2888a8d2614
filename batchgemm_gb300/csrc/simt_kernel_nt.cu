// simt_kernel_nt.cu -- the persistent FP32 SIMT kernel, B stored N x K.
#define BGEMM_SIMT_TA false
#define BGEMM_SIMT_TB true
#define BGEMM_SIMT_LAUNCH simt_launch_nt
#include "simt_kernel_t.h"
