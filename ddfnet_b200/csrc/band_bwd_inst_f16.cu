// Band filter-gradient kernel instantiations for __half elements.
#define DDF_INST_T __half
#include "band_bwd_inst.inc"
