// Degree-specialised FP32 stage-kernel variants for N = 12, 13 (split from the other
// degrees so that the variants compile in parallel).
#include "bbdg_stage_fast_impl.cuh"

template struct bbfast::FastKernel<12, BB_WAVE, 4, 128>;
template struct bbfast::FastKernel<12, BB_MAXWELL, 1, 256>;
template struct bbfast::FastKernel<13, BB_WAVE, 2, 256>;
template struct bbfast::FastKernel<13, BB_MAXWELL, 1, 384>;
