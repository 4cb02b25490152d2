// Instantiations of dps16_kernel<GAP_AFFINE, *, *, *, false> (packed 16-bit twin pairs, scores alone).
#define PA_GAPK GAP_AFFINE
#define PA_TBK false
#define PA_FN(x) x##_dps16_affine
#include "pa_dps16_inst.inc"
