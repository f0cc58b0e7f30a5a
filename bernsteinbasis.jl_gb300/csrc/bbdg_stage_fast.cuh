// Interface of the degree-specialised FP32 stage kernels (bbdg_stage_fast.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

constexpr int BB_VOL_GROUPS = 32;  // warp-rounds of the volume phase

struct FastStageParams {
  const void* tables;    // the variant's table image on the device (bb_fast_tables)
  int64_t K;
  int64_t tile_begin, tile_end;  // tiles [tile_begin, tile_end) of EPB elements (end 0 = all)
  int mode;              // 0: rhs only, 1: LSRK stage update
  float rkA, rkB, dt, tau;
  float* q;              // [NF][K][Np]
  float* res;            // [NF][K][Np]
  float* rhs;            // mode 0 output
  const float* trace_in; // [K][4][NF][Nfp], all faces that cross a tile boundary; nullptr
                         // (mode 0 only): neighbour nodes are read from q
  float* trace_out;      // [K][4][NF][Nfp] or nullptr
  const float* geo;      // [K][BB_GEO_STRIDE]
  const int32_t* conn;   // [K][4]
  int* status;
  uint32_t wait_iters;   // polls of a bounded mbarrier wait before it gives up (0 = 2^24)
  int fault;             // test only: 1 = one bulk copy is left out (a wait then runs out)
  int vec;               // floats per copy the field rows are aligned for: 4 = bulk copies, 2, 1
  // volume phase: warp-round g = r * (TPE / 32) + warp forms w(beta) for beta = vstart[g] +
  // lane, lane < vlen[g] (filled by the launcher)
  uint16_t vstart[BB_VOL_GROUPS];
  uint8_t vlen[BB_VOL_GROUPS];
};

struct FastLaunch {
  int num_sms;
  int device;           // CUDA device ordinal (the per-device launch set-up is cached)
  uint32_t wait_iters;  // copied into FastStageParams (the context's wait limit)
  int fault;            // copied into FastStageParams (the context's test-only fault mode)
};

// Index of the compiled variant for (N, physics, elements per block, threads), 0 = any; -1 if
// none. Any element count will do: the last tile may be partial.
int bb_fast_find(int N, int physics, int epb, int threads);
// The variant's constant tables on the context's device (whichever device is current), complete
// for any stream, made on first use and freed with the context; nullptr when out of memory.
struct bb_ctx;
const void* bb_fast_tables(bb_ctx* ctx, int idx);
int bb_fast_variant_info(int idx, int* epb, int* threads, size_t* smem);
int bb_fast_launch(int idx, const FastLaunch& fl, const FastStageParams& P, cudaStream_t st);
