// Instantiations of dpf2_kernel<GAP_AFFINE, *, *, *> (two columns per lane step, float32).
#define PA_GAPK GAP_AFFINE
#define PA_DTW 0
#define PA_FN(x) x##_dpf2_affine
#include "pa_dpf2_inst.inc"
