// Instantiations of dpf2_kernel<GAP_DTW, *, *, *> (two columns per lane step, float32).
#define PA_GAPK GAP_DTW
#define PA_DTW 1
#define PA_FN(x) x##_dpf2_dtw
#include "pa_dpf2_inst.inc"
