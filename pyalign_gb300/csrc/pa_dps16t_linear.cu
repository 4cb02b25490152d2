// Instantiations of dps16_kernel<GAP_LINEAR, *, *, *, true> (packed 16-bit twin pairs, one traceback).
#define PA_GAPK GAP_LINEAR
#define PA_TBK true
#define PA_FN(x) x##_dps16t_linear
#include "pa_dps16_inst.inc"
