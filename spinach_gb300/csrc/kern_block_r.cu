// Instantiations of the coupled-state kernels for one value type.
#define SPX_INST_CPLX 0
#define SPX_INST_FN spx_block_kernel_r
#include "kern_block.inc"
