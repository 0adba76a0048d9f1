// mg_sweep32.cu — the float (mixed-precision) instances of mg_sweep.cu, built with fused multiply-add
// contraction; the double instances keep the reference's bits without it.
#define SGPU_FLOAT_UNIT 1
#include "mg_sweep.cu"
