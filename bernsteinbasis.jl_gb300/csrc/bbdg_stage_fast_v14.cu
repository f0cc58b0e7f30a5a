// Degree-specialised FP32 stage-kernel variants for N = 14, 15 (split from the other
// degrees so that the variants compile in parallel).
#include "bbdg_stage_fast_impl.cuh"

template struct bbfast::FastKernel<14, BB_WAVE, 2, 256>;
template struct bbfast::FastKernel<14, BB_MAXWELL, 1, 384>;
template struct bbfast::FastKernel<15, BB_WAVE, 2, 256>;
template struct bbfast::FastKernel<15, BB_MAXWELL, 1, 448>;
