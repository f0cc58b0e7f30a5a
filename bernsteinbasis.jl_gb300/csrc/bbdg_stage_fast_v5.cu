// Degree-specialised FP32 stage-kernel variants for N = 3, 4, 5, 6 (split from the other
// degrees so that the variants compile in parallel).
#include "bbdg_stage_fast_impl.cuh"

template struct bbfast::FastKernel<5, BB_WAVE, 8, 32>;
template struct bbfast::FastKernel<5, BB_WAVE, 4, 32>;
template struct bbfast::FastKernel<5, BB_MAXWELL, 4, 32>;
template struct bbfast::FastKernel<5, BB_MAXWELL, 8, 32>;
template struct bbfast::FastKernel<4, BB_WAVE, 8, 32>;
template struct bbfast::FastKernel<4, BB_MAXWELL, 4, 32>;
template struct bbfast::FastKernel<6, BB_WAVE, 4, 32>;
template struct bbfast::FastKernel<6, BB_WAVE, 8, 32>;
template struct bbfast::FastKernel<6, BB_MAXWELL, 2, 64>;
template struct bbfast::FastKernel<3, BB_WAVE, 8, 32>;
template struct bbfast::FastKernel<3, BB_MAXWELL, 4, 32>;
template struct bbfast::FastKernel<5, BB_WAVE, 2, 32>;
template struct bbfast::FastKernel<6, BB_WAVE, 2, 64>;
template struct bbfast::FastKernel<5, BB_MAXWELL, 2, 32>;
