// Instantiations of the coupled-state kernels for real values.
#define SPX_INST_EXT 0
#define SPX_INST_FN spx_block_kernel_r
#include "kern_block.inc"
