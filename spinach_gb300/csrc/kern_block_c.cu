// Instantiations of the coupled-state kernels for complex values.
#define SPX_INST_EXT 1
#define SPX_INST_FN spx_block_kernel_c
#include "kern_block.inc"
