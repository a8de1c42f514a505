// The pair instances of the backward kernels (PREC = 1 in bwd_sm100.cu) as a translation unit of their own, so that
// the two sets of instances compile side by side.
#define FA_PAIR_INSTANCES 1
#include "bwd_sm100.cu"
