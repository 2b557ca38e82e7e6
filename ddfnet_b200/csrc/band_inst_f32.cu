// Band kernel instantiations for float elements.
#define DDF_INST_T float
#include "band_inst.inc"
