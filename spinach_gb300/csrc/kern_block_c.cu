// Instantiations of the coupled-state kernels for one value type.
#define SPX_INST_CPLX 1
#define SPX_INST_FN spx_block_kernel_c
#include "kern_block.inc"
