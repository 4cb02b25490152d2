// Instantiations of dps16_kernel<GAP_LINEAR, *, *, *, false> (packed 16-bit twin pairs, scores alone).
#define PA_GAPK GAP_LINEAR
#define PA_TBK false
#define PA_FN(x) x##_dps16_linear
#include "pa_dps16_inst.inc"
