#pragma once
// Degree-specialised FP32 lift operators (BernsteinLift mul! and face_lift_multiply!).
//
// One thread runs one face's whole lift chain (src/BernsteinLift.jl:139-164) in registers, with
// the degree a compile-time constant so that every multi-index is an immediate:
//   E_0 = L0 x, the 7-point stencil of (N+1)^2/2 R_{N+1} E_{N->N+1} on the face's Nfp inputs
//   E_d = R_{N-d+1} E_{d-1}, in place in registers (ascending order, as the reference)
//   layer d of the face's volume stack = l_d E_d (l_0 = 1)
//
// 4-face lift (BernsteinLift mul!): one warp per block and 8 elements per warp, one lane per
// (element, face) chain. Each chain writes its l_d-scaled stack to shared memory (odd lane stride:
// conflict-free; entries at the slots of lift_slot); the warp then forms every output coefficient as the sum of
// its four stack entries in the reference's face order (t=-1 face first, then faces 1, 2, 3 through
// the permutations of src/BernsteinLift.jl:207-218) and stores it coalesced. No atomics, so the
// result does not depend on scheduling. The next tile's inputs arrive while this tile is worked on:
// in registers (degrees up to 9), by a bulk copy into their own buffer (degrees 10 and 11), or
// from 12 on pulled into L2 a tile ahead and read with coalesced loads into the stack area at the
// start of the tile (no input buffer, so more elements per warp fit: 4 up to N = 13).
//
// Single-face lift (face_lift_multiply!): the t = -1 face's stack is already in volume order, so
// the chain writes the output tile directly.
#include <algorithm>

#include "bbdg_internal.cuh"
#include "bbdg_lift_slots.cuh"

namespace bblift {

__host__ __device__ constexpr int lf_tri(int n, int j) { return j * (2 * n + 3 - j) / 2; }
__host__ __device__ constexpr int lf_tet(int n, int k) {
  return ((n + 1) * (n + 2) * (n + 3) - (n + 1 - k) * (n + 2 - k) * (n + 3 - k)) / 6;
}
__host__ __device__ constexpr int lf_ij(int n, int i, int j) { return i + lf_tri(n, j); }
__host__ __device__ constexpr int lf_ijk(int n, int i, int j, int k) {
  return i + lf_tri(n, j) + lf_tet(n, k) - j * k;
}

// One face chain from the Nfp inputs X (registers) to the l_d-scaled stack g (shared memory,
// g[lf_ijk(N, i, j, d)] = F_d(i, j) = l_d E_d(i, j); for the t = -1 face this is the volume
// order). The chain carries F_d itself: l_d / l_{d-1} = -(N-d+1)/(d+1) and R_{N-d+1} divides by
// N-d+1, so F_d = -1/(d+1) [(i+1) F_{d-1}(i+1,j) + (j+1) F_{d-1}(i,j+1) + (N-d+1-i-j) F_{d-1}(i,j)]
// with F_0 = E_0 = L0 x.
template <int N, bool SLOTS>
__device__ __forceinline__ void lift_chain_stack(const float (&X)[(N + 1) * (N + 2) / 2],
                                                 float* g) {
  constexpr int NFP = (N + 1) * (N + 2) / 2;
  float E[NFP];
#pragma unroll
  for (int j = 0; j <= N; ++j) {
#pragma unroll
    for (int i = 0; i + j <= N; ++i) {
      const int k = N - i - j;
      float v = float((i + 1) * (i + 1) + (j + 1) * (j + 1) + (k + 1) * (k + 1)) * X[lf_ij(N, i, j)];
      if (j > 0) v = fmaf(float((i + 1) * j), X[lf_ij(N, i + 1, j - 1)], v);
      if (k > 0) v = fmaf(float((i + 1) * k), X[lf_ij(N, i + 1, j)], v);
      if (i > 0) v = fmaf(float((j + 1) * i), X[lf_ij(N, i - 1, j + 1)], v);
      if (k > 0) v = fmaf(float((j + 1) * k), X[lf_ij(N, i, j + 1)], v);
      if (i > 0) v = fmaf(float((k + 1) * i), X[lf_ij(N, i - 1, j)], v);
      if (j > 0) v = fmaf(float((k + 1) * j), X[lf_ij(N, i, j - 1)], v);
      E[lf_ij(N, i, j)] = 0.5f * v;
      g[SLOTS ? lift_slot<N>(lf_ij(N, i, j)) : lf_ij(N, i, j)] = E[lf_ij(N, i, j)];
    }
  }
#pragma unroll
  for (int d = 1; d <= N; ++d) {
    const int n = N - d + 1;  // input degree of this reduction
    const float inv = -1.0f / float(d + 1);
#pragma unroll
    for (int j = 0; j < n; ++j) {
#pragma unroll
      for (int i = 0; i + j < n; ++i) {
        // reduction_multiply! (src/BernsteinLift.jl:81-85) times l_d / l_{d-1}, in place,
        // ascending
        const float v = float(i + 1) * inv * E[lf_ij(N, i + 1, j)] +
                        (float(j + 1) * inv * E[lf_ij(N, i, j + 1)] +
                         float(n - i - j) * inv * E[lf_ij(N, i, j)]);
        E[lf_ij(N, i, j)] = v;
        g[SLOTS ? lift_slot<N>(lf_ijk(N, i, j, d)) : lf_ijk(N, i, j, d)] = v;
      }
    }
  }
}

__device__ __forceinline__ uint32_t lf_saddr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

template <int N>
struct Lift4 {
  static constexpr int NP = (N + 1) * (N + 2) * (N + 3) / 6;
  static constexpr int NFP = (N + 1) * (N + 2) / 2;
  static constexpr int NPS = NP | 1;    // stack stride: odd, conflict-free stack stores
  static constexpr int NFPP = NFP | 1;  // input row stride when staged from registers
  // elements per warp: 8 (32 chains) while the stacks leave room for several warps per SM;
  // 4 (16 chains, half the lanes idle in the chain phase) from N = 11 on and 2 from N = 14
  // on, which keeps several warps per SM for the loads and the gather (measured at N = 11
  // and 12: +16 %, +17 %; at N = 10 -15 %; at N = 13 with the staged inputs 4 beats 2 by 14 %,
  // at N = 14 and 15 2 beats 4 and 8)
  static constexpr int EPW = N >= 14 ? 2 : N >= 11 ? 4 : 8;
  // from N = 12: the next tile's inputs go to L2 (bulk prefetch), this tile's are read with
  // coalesced 16-byte loads and staged through the stack area (N = 12: 0.29 -> 0.31 of the
  // HBM copy rate, N = 13: 0.20 -> 0.235; slower at N = 10, 11 than the bulk-copy buffer)
  static constexpr bool STAGED = N >= 12;
  static constexpr int INW = EPW * 4 * NFP;  // input floats per tile
  // next tile in registers when they fit beside the chain, else a bulk copy
  static constexpr bool REG_PREFETCH = N <= 9;
  static constexpr int NV = (INW + 31) / 32;  // input floats per lane
  static constexpr int NR = (NP + 31) / 32;   // coefficients per lane
  // shared memory, bytes: [bulk input buffer][stacks (also the staged input)]
  static constexpr int IN_B = (REG_PREFETCH || STAGED) ? 0 : INW * 4;
  static constexpr int G_B = IN_B;
  // The gather. Up to degree 4 (35 coefficients), and at 10, the warp takes all elements'
  // coefficients in one run (FLAT), above coefficient by coefficient for every element. At degrees
  // 6 to 9 and 11 the stacks' entries lie at the slots of lift_slot, which share few banks (SLOTS),
  // with a table of positions; at the others in volume order, the positions in registers, because
  // the table would take the place of a warp. Large K, one run / as chosen: N = 5, 141 / 129 us;
  // N = 7, 150 / 129; N = 9, 153 / 151; N = 11, 190 / 167; N = 13, 280 / 227 (268 with slots); N = 15,
  // 340 / 310; N = 10, 176 / 172, but 5,245 columns 14.5 / 16.4.
  static constexpr bool FLAT = N <= 4 || N == 10, SLOTS = !FLAT && N >= 6 && N <= 11;
  static constexpr int P_B = G_B + (EPW * 4 * NPS * 4 + 15) / 16 * 16;  // [NP] positions
  static constexpr int BAR_B = P_B + ((FLAT ? NP * 4 : SLOTS ? NP * 8 : 0) + 15) / 16 * 16;
  static constexpr int SMEM = BAR_B + 16;
  static_assert(NFPP <= NPS, "staged inputs fit in the stack area");
  static_assert(REG_PREFETCH ? EPW == 8 : true, "the register path stages 32 chains");
  static_assert(EPW * 4 <= 32, "one chain per lane");
  static_assert(NP < 65536, "stack slots are packed in 16 bits");
  static_assert(INW % 4 == 0 && (INW * 4) % 16 == 0, "tiles are whole 16-byte chunks");
};

template <int N>
__global__ void __launch_bounds__(32) lift4_kernel(int64_t K, const uint4* __restrict__ gather,
                                                   const float* __restrict__ x,
                                                   float* __restrict__ out, int* status,
                                                   uint32_t wait_iters) {
  using L = Lift4<N>;
  constexpr int NP = L::NP, NFP = L::NFP, NPS = L::NPS, NFPP = L::NFPP, EPW = L::EPW;
  constexpr int NV = L::NV, NR = L::NR;
  extern __shared__ __align__(16) unsigned char smem[];
  float* sIn = reinterpret_cast<float*>(smem);  // bulk-copy input buffer (degrees > 9)
  float* sG = reinterpret_cast<float*>(smem + L::G_B);
  uint64_t* bar = reinterpret_cast<uint64_t*>(smem + L::BAR_B);
  const int t = threadIdx.x;
  // stack positions of coefficient n on faces f0 (i,k,j), f1 (j,k,l), f2 (j,k,i), f3 (i,j,k): from
  // the degree's gather table, or decoded where that takes less than a load (up to degree 4; 384
  // columns, table / decoded: N = 4, 2.5 / 2.3 us, N = 9, 6.6 / 7.6, N = 12, 7.6 / 11.5, N = 15,
  // 11.1 / 18.6)
  auto positions = [=](int n) {
    if constexpr (N <= 4) {
      int m = n, k = 0, j = 0;
      while (m >= (N - k + 1) * (N - k + 2) / 2) m -= (N - k + 1) * (N - k + 2) / 2, ++k;
      while (m >= N - k - j + 1) m -= N - k - j + 1, ++j;
      const int i = m, l = N - i - j - k;
      return make_uint2(lf_ijk(N, i, k, j) | (lf_ijk(N, j, k, l) << 16), lf_ijk(N, j, k, i) | (n << 16));
    } else {
      const uint4 ga = __ldg(gather + n);
      if constexpr (!L::SLOTS) return make_uint2(ga.z, ga.w);
      auto at = [](uint32_t q) { return (uint32_t)lift_slot_at<N>((int)q); };
      return make_uint2(at(ga.z & 0xffffu) | (at(ga.z >> 16) << 16),
                        at(ga.w & 0xffffu) | (at(ga.w >> 16) << 16));
    }
  };
  auto pack = [](uint2 p) {  // f0, f1, f2, 10 bits each (f3 is n itself in volume order)
    return (p.x & 0xffffu) | ((p.x >> 16) << 10) | ((p.y & 0xffffu) << 20);
  };
  uint2* sP = reinterpret_cast<uint2*>(smem + L::P_B);        // SLOTS
  uint32_t* sP10 = reinterpret_cast<uint32_t*>(smem + L::P_B);  // FLAT
  uint32_t pos[L::FLAT || L::SLOTS ? 1 : NR];
  if constexpr (L::FLAT || L::SLOTS) {
    for (int n = t; n < NP; n += 32) {
      if constexpr (L::FLAT) sP10[n] = pack(positions(n));
      else sP[n] = positions(n);
    }
  } else {
#pragma unroll
    for (int r = 0; r < NR; ++r) pos[r] = pack(positions(min(t + 32 * r, NP - 1)));
  }
  const int64_t ntile = (K + EPW - 1) / EPW;
  auto tile_ne = [&](int64_t tile) { return (int)(K - tile * EPW < EPW ? K - tile * EPW : EPW); };
  // Inputs are staged one float per lane: 32 lanes then store to 32 banks (chain rows are NFPP
  // apart), where 16-byte pieces meet four ways in a bank; those are still the better ones up to
  // degree 3 (a quarter of the loads).
  constexpr int VW = N <= 3 ? 4 : 1, NVW = (NV + VW - 1) / VW;  // floats per piece, pieces per lane
  float pf[L::REG_PREFETCH ? NVW : 1][VW];
  auto fetch = [&](int64_t tile) {  // registers path
    const float* xs = x + tile * EPW * 4 * NFP;
    const int nv = tile_ne(tile) * 4 * NFP;
#pragma unroll
    for (int r = 0; r < NVW; ++r) {
      const int g = VW * (t + 32 * r);
      if (g >= nv) continue;
      if constexpr (VW == 4)
        *reinterpret_cast<float4*>(pf[r]) = __ldg(reinterpret_cast<const float4*>(xs + g));
      else
        pf[r][0] = __ldg(xs + g);
    }
  };
  auto issue = [&](int64_t tile) {  // bulk-copy path, lane 0
    const uint32_t bytes = (uint32_t)(tile_ne(tile) * 4 * NFP * 4);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(lf_saddr(bar)),
                 "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            lf_saddr(sIn)),
        "l"(x + tile * EPW * 4 * NFP), "r"(bytes), "r"(lf_saddr(bar))
        : "memory");
  };
  // bounded wait for the bulk copy with the given phase parity (2^24 polls, about a second,
  // unless the context sets another limit)
  const uint32_t wlim = wait_iters ? wait_iters : (1u << 24);
  auto wait_in = [&](uint32_t parity) {
    for (uint32_t it = 0; it < wlim; ++it) {
      uint32_t ok;
      asm volatile(
          "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
          " selp.u32 %0, 1, 0, p;\n}\n"
          : "=r"(ok)
          : "r"(lf_saddr(bar)), "r"(parity)
          : "memory");
      if (ok) return true;
      if (it > 64) __nanosleep(64);
    }
    return false;
  };
  if constexpr (L::REG_PREFETCH) {
    if (blockIdx.x < ntile) fetch(blockIdx.x);
  } else if constexpr (!L::STAGED) {
    if (t == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(lf_saddr(bar)) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      if (blockIdx.x < ntile) issue(blockIdx.x);
    }
  }
  __syncwarp();
  uint32_t ph = 0;
  for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int ne = tile_ne(tile);
    const int64_t next = tile + gridDim.x;
    float X[NFP];
    if constexpr (L::REG_PREFETCH) {
      // stage this tile's inputs (chain c = element * 4 + face in rows of NFPP) and take each
      // lane's row into registers; then the next tile's loads go out
      const int nv = ne * 4 * NFP;
#pragma unroll
      for (int r = 0; r < NVW; ++r)
#pragma unroll
        for (int w = 0; w < VW; ++w) {
          const int g = VW * (t + 32 * r) + w;
          if (g < nv) sG[g + (NFPP - NFP) * (g / NFP)] = pf[r][w];
        }
      __syncwarp();
#pragma unroll
      for (int m = 0; m < NFP; ++m) X[m] = sG[t * NFPP + m];
      __syncwarp();  // every staged input is in registers before the stacks overwrite them
      if (next < ntile) fetch(next);
    } else if constexpr (L::STAGED) {
      // the tile's inputs, pulled into L2 a tile ago: coalesced 16-byte loads (one float per lane
      // was slower here: N = 12, 249 against 216 us), staged in the stack area (free until the
      // chains write it) in rows of NFPP, then one row per lane
      const float4* xs = reinterpret_cast<const float4*>(x + tile * EPW * 4 * NFP);
      const int nv = ne * NFP;  // float4s of the tile (4 NFP floats per element)
      constexpr int UNR = 8;
      for (int v0 = 0; v0 < nv; v0 += 32 * UNR) {
        float4 buf[UNR];
#pragma unroll
        for (int r = 0; r < UNR; ++r) {
          const int v = v0 + t + 32 * r;
          if (v < nv) buf[r] = __ldg(xs + v);
        }
#pragma unroll
        for (int r = 0; r < UNR; ++r) {
          const int v = v0 + t + 32 * r;
          if (v < nv) {
            const float qq[4] = {buf[r].x, buf[r].y, buf[r].z, buf[r].w};
#pragma unroll
            for (int w = 0; w < 4; ++w) {
              const int g = 4 * v + w;
              sG[g + (NFPP - NFP) * (g / NFP)] = qq[w];
            }
          }
        }
      }
      __syncwarp();
#pragma unroll
      for (int m = 0; m < NFP; ++m) X[m] = sG[(t < ne * 4 ? t : 0) * NFPP + m];
      __syncwarp();  // every staged input is in registers before the stacks overwrite them
      if (t == 0 && next < ntile) {
        // 16-byte aligned start and size: x is (checked by the caller) and a tile is
        // EPW * 4 * NFP floats, a multiple of 4
        const uint32_t bytes = (uint32_t)(tile_ne(next) * 4 * NFP * 4);
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(x + next * EPW * 4 * NFP),
                     "r"(bytes)
                     : "memory");
      }
    } else {
      if (!wait_in(ph)) {
        if (t == 0) {
          atomicOr(status, 2);
          wait_in(ph);  // let the copy in flight land before the block exits (bounded)
        }
        return;
      }
      ph ^= 1u;
#pragma unroll
      for (int m = 0; m < NFP; ++m) X[m] = sIn[(t < EPW * 4 ? t : 0) * NFP + m];
      __syncwarp();
      if (t == 0 && next < ntile) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        issue(next);
      }
    }
    if (t / 4 < ne) lift_chain_stack<N, L::SLOTS>(X, sG + t * NPS);
    __syncwarp();
    // out(n) = f3 stack + f0 stack + f1 stack + f2 stack at n's slots, coalesced stores
    float* os = out + tile * EPW * NP;
    auto gather = [&](const float* G, int n, uint32_t p) {
      return ((G[3 * NPS + n] + G[p & 1023u]) + G[NPS + ((p >> 10) & 1023u)]) +
             G[2 * NPS + (p >> 20)];
    };
    if constexpr (L::FLAT) {
      for (int v = t; v < ne * NP; v += 32) {
        const int e = v / NP, n = v - e * NP;
        os[v] = gather(sG + e * 4 * NPS, n, sP10[n]);
      }
    } else {
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const int n = t + 32 * r;
        if (n >= NP) continue;
        uint2 p = make_uint2(0u, 0u);
        if constexpr (L::SLOTS) p = sP[n];
#pragma unroll
        for (int e = 0; e < EPW; ++e) {
          if (e >= ne) continue;
          const float* G = sG + e * 4 * NPS;
          if constexpr (L::SLOTS)
            os[e * NP + n] = ((G[3 * NPS + (p.y >> 16)] + G[p.x & 0xffffu]) + G[NPS + (p.x >> 16)]) +
                             G[2 * NPS + (p.y & 0xffffu)];
          else
            os[e * NP + n] = gather(G, n, pos[r]);
        }
      }
    }
    __syncwarp();
  }
}

template <int N>
int launch_lift4(bb_ctx* ctx, const DegTables* t, int64_t K, const void* x, void* out,
                 cudaStream_t st) {
  using L = Lift4<N>;
  auto kern = lift4_kernel<N>;
  int* status = bb_ctx_status_word(ctx);
  if (!status) return bb_fail(ctx, BB_ERR_NOMEM, "status word allocation failed");
  BB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM));
  int per_sm = 0;
  BB_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32, L::SMEM));
  if (per_sm < 1) return bb_fail(ctx, BB_ERR_ARG, "lift tile does not fit");
  const int64_t ntile = (K + L::EPW - 1) / L::EPW;
  const int grid = (int)std::min<int64_t>(ntile, (int64_t)per_sm * ctx->num_sms);
  kern<<<grid, 32, L::SMEM, st>>>(K, reinterpret_cast<const uint4*>(t->d_words + t->o_gather),
                                  (const float*)x, (float*)out, status, ctx->wait_iters);
  return bb_check_launch(ctx, "lift4_kernel");
}

// Single face (the t = -1 face, k = 0): its stack is the output in volume order.
template <int N>
struct Lift1 {
  static constexpr int NP = (N + 1) * (N + 2) * (N + 3) / 6;
  static constexpr int NFP = (N + 1) * (N + 2) / 2;
  static constexpr int NFPP = NFP | 1;
  static constexpr int NPS = NP | 1;
  static constexpr int EPB = 32;
  static constexpr int SMEM = EPB * (NFPP + NPS) * 4;
};

template <int N>
__global__ void __launch_bounds__(32) lift1_kernel(int64_t K, const float* __restrict__ x,
                                                   float* __restrict__ out) {
  using L = Lift1<N>;
  constexpr int NP = L::NP, NFP = L::NFP, NFPP = L::NFPP, NPS = L::NPS, EPB = L::EPB;
  extern __shared__ __align__(16) float sm1[];
  float* sx = sm1;              // [EPB][NFPP]
  float* so = sm1 + EPB * NFPP;  // [EPB][NPS]
  const int t = threadIdx.x;
  const int64_t ntile = (K + EPB - 1) / EPB;
  for (int64_t tile = blockIdx.x; tile < ntile; tile += gridDim.x) {
    const int64_t e0 = tile * EPB;
    const int ne = (int)min64(EPB, K - e0);
    __syncwarp();
    for (int g = t; g < ne * NFP; g += 32) {
      const int ch = g / NFP, m = g - ch * NFP;
      sx[ch * NFPP + m] = __ldg(x + e0 * NFP + g);
    }
    __syncwarp();
    if (t < ne) {
      float X[NFP];
#pragma unroll
      for (int m = 0; m < NFP; ++m) X[m] = sx[t * NFPP + m];
      lift_chain_stack<N, false>(X, so + t * NPS);
    }
    __syncwarp();
    for (int v = t; v < ne * NP; v += 32) {
      const int e = v / NP, n = v - e * NP;
      out[e0 * NP + v] = so[e * NPS + n];
    }
  }
}

template <int N>
int launch_lift1(bb_ctx* ctx, int64_t K, const void* x, void* out, cudaStream_t st) {
  using L = Lift1<N>;
  auto kern = lift1_kernel<N>;
  BB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::SMEM));
  int per_sm = 0;
  BB_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32, L::SMEM));
  if (per_sm < 1) return bb_fail(ctx, BB_ERR_ARG, "lift tile does not fit");
  const int64_t ntile = (K + L::EPB - 1) / L::EPB;
  const int grid = (int)std::min<int64_t>(ntile, (int64_t)per_sm * ctx->num_sms);
  kern<<<grid, 32, L::SMEM, st>>>(K, (const float*)x, (float*)out);
  return bb_check_launch(ctx, "lift1_kernel");
}

}  // namespace bblift
