// The pair instances of the forward kernel (PREC = 1 in fwd_sm100.cu) as a translation unit of their own, so that
// the two sets of instances compile side by side.
#define FA_PAIR_INSTANCES 1
#include "fwd_sm100.cu"
