// Degree-specialised FP32 stage-kernel variants for N = 7, 8 (split from the other
// degrees so that the variants compile in parallel).
#include "bbdg_stage_fast_impl.cuh"

template struct bbfast::FastKernel<7, BB_WAVE, 4, 32>;
template struct bbfast::FastKernel<7, BB_WAVE, 4, 64>;
template struct bbfast::FastKernel<7, BB_MAXWELL, 2, 64>;
template struct bbfast::FastKernel<8, BB_WAVE, 4, 64>;
template struct bbfast::FastKernel<8, BB_MAXWELL, 4, 64>;
template struct bbfast::FastKernel<8, BB_MAXWELL, 4, 32>;
template struct bbfast::FastKernel<7, BB_WAVE, 2, 64>;
