// Registry of the compiled degree-specialised stage-kernel variants:
// X(N, physics, elements per block, threads per element). The first variant matching a query
// is the default for that (N, physics), so each degree lists its fastest tile on a 16^3 x 6
// mesh first; the others are candidates of the autotuner. A mesh's last tile may be partial.
// Each variant is instantiated in one bbdg_stage_fast_v*.cu.
#pragma once
#define BB_FAST_VARIANTS(X) \
  X(9, BB_WAVE, 4, 64) \
  X(9, BB_WAVE, 4, 32) \
  X(9, BB_WAVE, 2, 64) \
  X(9, BB_MAXWELL, 2, 128) \
  X(9, BB_MAXWELL, 2, 64) \
  X(9, BB_MAXWELL, 2, 96) \
  X(5, BB_WAVE, 8, 32) \
  X(5, BB_WAVE, 4, 32) \
  X(5, BB_MAXWELL, 4, 32) \
  X(5, BB_MAXWELL, 8, 32) \
  X(10, BB_WAVE, 2, 64) \
  X(10, BB_MAXWELL, 2, 192) \
  X(10, BB_MAXWELL, 2, 96) \
  X(10, BB_MAXWELL, 2, 64) \
  X(4, BB_WAVE, 8, 32) \
  X(4, BB_MAXWELL, 4, 32) \
  X(6, BB_WAVE, 4, 32) \
  X(6, BB_WAVE, 8, 32) \
  X(6, BB_MAXWELL, 2, 64) \
  X(7, BB_WAVE, 4, 32) \
  X(7, BB_WAVE, 4, 64) \
  X(7, BB_MAXWELL, 2, 64) \
  X(8, BB_WAVE, 4, 64) \
  X(8, BB_MAXWELL, 4, 64) \
  X(8, BB_MAXWELL, 4, 32) \
  X(11, BB_WAVE, 2, 128) \
  X(11, BB_WAVE, 2, 96) \
  X(11, BB_MAXWELL, 2, 192) \
  X(11, BB_MAXWELL, 2, 96) \
  X(3, BB_WAVE, 8, 32) \
  X(3, BB_MAXWELL, 4, 32) \
  X(12, BB_WAVE, 4, 128) \
  X(12, BB_MAXWELL, 1, 256) \
  X(13, BB_WAVE, 2, 256) \
  X(13, BB_MAXWELL, 1, 384) \
  X(14, BB_WAVE, 2, 256) \
  X(14, BB_MAXWELL, 1, 384) \
  X(15, BB_WAVE, 2, 256) \
  X(15, BB_MAXWELL, 1, 448) \
  X(5, BB_WAVE, 2, 32) \
  X(6, BB_WAVE, 2, 64) \
  X(7, BB_WAVE, 2, 64) \
  X(5, BB_MAXWELL, 2, 32)
