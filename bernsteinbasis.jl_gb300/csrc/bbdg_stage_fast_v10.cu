// Degree-specialised FP32 stage-kernel variants for N = 10, 11 (split from the other
// degrees so that the variants compile in parallel).
#include "bbdg_stage_fast_impl.cuh"

template struct bbfast::FastKernel<10, BB_WAVE, 2, 64>;
template struct bbfast::FastKernel<10, BB_MAXWELL, 2, 192>;
template struct bbfast::FastKernel<10, BB_MAXWELL, 2, 96>;
template struct bbfast::FastKernel<10, BB_MAXWELL, 2, 64>;
template struct bbfast::FastKernel<11, BB_WAVE, 2, 128>;
template struct bbfast::FastKernel<11, BB_WAVE, 2, 96>;
template struct bbfast::FastKernel<11, BB_MAXWELL, 2, 192>;
template struct bbfast::FastKernel<11, BB_MAXWELL, 2, 96>;
