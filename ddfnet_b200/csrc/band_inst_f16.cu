// Band kernel instantiations for __half elements.
#define DDF_INST_T __half
#include "band_inst.inc"
