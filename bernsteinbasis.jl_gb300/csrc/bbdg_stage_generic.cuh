// Generic (runtime-degree) DG stage tile: shared by the per-solver stage kernel
// (bbdg_solver.cu) and the batched persistent kernel (bbdg_batch.cu).
//
// One thread block owns a tile of `epb` consecutive elements and does, per RK stage:
//   1. stage q (all fields), geometry and connectivity of its tile in shared memory
//   2. interface flux at every face node (examples/3d_wave.jl:41-56,
//      examples/3d_maxwell.jl:43-65): the neighbour trace comes from shared memory when
//      the neighbour is in the same tile, otherwise from the trace buffer written by the
//      previous stage (only faces that cross a tile boundary are ever written or read)
//   3. volume term (3d_wave.jl:59-79): the geometric combination of Dr, Ds, Dt is applied
//      as sum_b alpha_b w(alpha - e_b), w(beta) = sum_a g_a x(beta + e_a), g the barycentric
//      weights of the physical derivative (Dr = (D0 - D3)/2 etc.)
//   4. lift of the four face fluxes (src/BernsteinLift.jl:139-220): whole stacks where
//      they fit in shared memory, else accumulated level by level
//   5. gather of the stacks, divide by J, LSRK update res = A res + dt rhs, q += B res; write
//      q, res and the tile's outgoing traces
// q and res are updated in place: no block reads another tile's q, so there is no race.
#pragma once

#include "bbdg_internal.cuh"

template <int PHYS>
struct Phys;
template <>
struct Phys<BB_WAVE> {
  static constexpr int NF = 4;  // p, u, v, w
  static constexpr int NW = 4;  // div(u,v,w), dp/dx, dp/dy, dp/dz (scaled by J)
  static constexpr int NCH = 2;  // lift chains per face: pressure flux, scalar velocity flux
  static constexpr float vol_sign = -1.f;
};
template <>
struct Phys<BB_MAXWELL> {
  static constexpr int NF = 6;  // Hx, Hy, Hz, Ex, Ey, Ez
  static constexpr int NW = 6;  // curl terms
  static constexpr int NCH = 6;  // one lift chain per field
  static constexpr float vol_sign = 1.f;
};
// examples/3d_advec_scalar.jl: du = -(LIFT flux + J du/dx) / J; the flux is stored negated
// so that the shared "sign * volume + lift" combination gives the example's right-hand side.
template <>
struct Phys<BB_ADVECTION> {
  static constexpr int NF = 1;  // u
  static constexpr int NW = 1;  // J du/dx
  static constexpr int NCH = 1;
  static constexpr float vol_sign = -1.f;
};
// examples/3d_advec.jl: q = (u, v, w), fx(q) = (u, 0, 0), fy = fz = 0: the flux of the
// scalar example on each component, the volume term on u only; du = -(...) / J as above.
template <>
struct Phys<BB_ADVECTION3> {
  static constexpr int NF = 3;  // u, v, w
  static constexpr int NW = 1;  // J du/dx (v and w have no volume term)
  static constexpr int NCH = 3;
  static constexpr float vol_sign = -1.f;
};

template <class T>
struct StageParams {
  DegTables tab;
  const uint32_t* gtab;
  int64_t K;
  int64_t tile_begin, tile_end;  // stage_kernel's tiles [tile_begin, tile_end) (end 0 = all)
  int epb;
  int mode;             // 0: write rhs to `rhs`; 1: LSRK stage update of q and res
  T rkA, rkB, dt, tau;  // stage coefficients, time step, penalty (tau <= 0: as written)
  T* q;                 // [NF][K][Np]
  T* res;               // [NF][K][Np]
  T* rhs;               // mode 0 output [NF][K][Np]
  const T* trace_in;    // [K][4][NF][Nfp] or nullptr: gather neighbour traces from q
  T* trace_out;         // [K][4][NF][Nfp] or nullptr
  const T* geo;         // [K][BB_GEO_STRIDE]
  const int32_t* conn;  // [K][4]
  int* status;          // device error word
};

// Shared-memory layout of a tile (in units of T unless noted). stacks != 0: every chain of the
// tile keeps its whole lift stack (lift_stacks), and the gather, the volume term and the update
// are one pass (`out` is then the table of lift_stacks' weights); stacks == 0, where those do not
// fit: the lift goes face by face with two ping-pong rows and adds into `out`.
struct TileLayout {
  size_t q, out, flux, work, stack, geo, pen, gh, conn_bytes, tab_bytes, total;
  int work_elems;
  int stacks;
};
constexpr size_t kStackBytes = 224 * 1024;

// Lift chains per face for NF fields (Phys<PHYS>::NCH): the wave's velocity flux is a scalar
// times the face normal, so its three components share one chain.
__host__ __device__ inline int lift_chains(int NF) { return NF == 4 ? 2 : NF; }

// Layout for degree N with Np/Nfp/NpM1 coefficients, NF fields, NW volume terms, scalars of
// `tsize` bytes and `nwords` 32-bit table words: without whole stacks.
__host__ __device__ inline TileLayout tile_layout_rows(int N, int NF, int NW, size_t tsize,
                                                      int nwords, int epb) {
  TileLayout L;
  const size_t Np = np3(N), Nfp = np2(N), NpM1 = np3(N - 1), S = np2(N + 1);
  const size_t nch = (size_t)lift_chains(NF);
  size_t off = 0;
  L.q = off; off += (size_t)NF * epb * Np;
  L.out = off; off += (size_t)NF * epb * Np;
  L.flux = off; off += (size_t)epb * 4 * NF * Nfp;
  L.work = off;
  const size_t wvol = (size_t)NW * epb * NpM1, wlift = 2 * (size_t)epb * nch * S;
  L.work_elems = (int)(wvol > wlift ? wvol : wlift);
  off += L.work_elems;
  L.geo = off; off += (size_t)epb * BB_GEO_STRIDE;
  L.pen = off; off += (size_t)epb * 8;  // per face: tau |n|, tau / |n|
  L.gh = off; off += (size_t)epb * 9;   // per element: rxJ ... txJ / 2
  size_t bytes = align16(off * tsize);
  L.conn_bytes = bytes; bytes += align16((size_t)epb * 4 * sizeof(int32_t));
  L.tab_bytes = bytes; bytes += (size_t)nwords * 4;
  L.total = align16(bytes);
  L.stack = 0;
  L.stacks = 0;
  return L;
}

// The layout with whole stacks (row stride Np | 1, against bank conflicts).
__host__ __device__ inline TileLayout tile_layout_stacks(int N, int NF, int NW, size_t tsize,
                                                        int nwords, int epb) {
  TileLayout L;
  const size_t Np = np3(N), Nfp = np2(N), NpM1 = np3(N - 1);
  const size_t nch = (size_t)lift_chains(NF);
  size_t off = 0;
  L.q = off; off += (size_t)NF * epb * Np;
  L.flux = off; off += (size_t)epb * 4 * nch * Nfp;
  L.work = off; off += (size_t)NW * epb * NpM1;
  L.work_elems = (int)(NW * epb * NpM1);
  L.stack = off; off += (size_t)epb * 4 * nch * (Np | 1);
  L.geo = off; off += (size_t)epb * BB_GEO_STRIDE;
  L.pen = off; off += (size_t)epb * 8;
  L.gh = off; off += (size_t)epb * 9;
  L.out = off; off += tsize == 8 ? (size_t)(N + 1) * (N + 2) : 0;  // wred
  size_t bytes = align16(off * tsize);
  L.conn_bytes = bytes; bytes += align16((size_t)epb * 4 * sizeof(int32_t));
  L.tab_bytes = bytes; bytes += (size_t)nwords * 4;
  L.total = align16(bytes);
  L.stacks = 1;
  return L;
}

// Whole stacks where they fit. They take the place of one thread per (element, face, chain), which
// kept too few threads busy (FP32 scalar advection, N = 9, K = 10,368, 8 elements: 88 -> 56 us per
// stage; N = 15, K = 3,072: 227 -> 72), and in FP64 of the face-by-face lift (Maxwell N = 7,
// K = 4,374: 403 -> 301). Every form gives the same bits in FP32.
__host__ __device__ inline TileLayout tile_layout_for(int N, int NF, int NW, size_t tsize,
                                                     int nwords, int epb) {
  const TileLayout s = tile_layout_stacks(N, NF, NW, tsize, nwords, epb);
  return s.total <= kStackBytes ? s : tile_layout_rows(N, NF, NW, tsize, nwords, epb);
}

template <class T, int PHYS>
TileLayout tile_layout(const DegTables& t, int epb) {
  return tile_layout_for(t.N, Phys<PHYS>::NF, Phys<PHYS>::NW, sizeof(T), t.nwords, epb);
}

// The traces of the tile's faces whose neighbour lies outside it, from the updated q in sQ.
template <class T, int NF>
__device__ void write_traces(const StageParams<T>& P, const SmemTables& st, const T* sQ,
                             const int32_t* sConn, int64_t e0, int ne) {
  const int Np = P.tab.Np, Nfp = P.tab.Nfp, epb = P.epb;
  const FastDiv by_nfp(Nfp), by_nfnfp(NF * Nfp), by_4nfnfp(4 * NF * Nfp);
  for (int it = threadIdx.x; it < ne * 4 * NF * Nfp; it += blockDim.x) {
    const int le = by_4nfnfp.div(it);
    int rem = it - le * 4 * NF * Nfp;
    const int f = by_nfnfp.div(rem);
    rem -= f * NF * Nfp;
    const int fld = by_nfp.div(rem), a = rem - fld * Nfp;
    const int64_t nbr = (int64_t)((uint32_t)sConn[le * 4 + f] >> 5);
    if (nbr >= e0 && nbr < e0 + ne) continue;  // neighbour inside the tile
    P.trace_out[((size_t)(e0 + le) * 4 + f) * NF * Nfp + (size_t)fld * Nfp + a] =
        sQ[((size_t)fld * epb + le) * Np + st.fvol[f * Nfp + a]];
  }
}

// One tile of the generic stage (all threads of the block call it). The degree tables are in
// shared memory (st); the layout L matches P's degree, physics and tile.
template <class T, int PHYS>
__device__ void generic_stage_tile(const StageParams<T>& P, const TileLayout& L,
                                   const SmemTables& st, int64_t tile) {
  constexpr int NF = Phys<PHYS>::NF, NW = Phys<PHYS>::NW, NCH = Phys<PHYS>::NCH;
  extern __shared__ __align__(16) unsigned char smem[];
  T* sbase = reinterpret_cast<T*>(smem);
  T* sQ = sbase + L.q;
  T* sOut = sbase + L.out;
  T* sFlux = sbase + L.flux;
  T* sWork = sbase + L.work;
  T* sGeo = sbase + L.geo;
  T* sPen = sbase + L.pen;
  T* sGh = sbase + L.gh;
  int32_t* sConn = reinterpret_cast<int32_t*>(smem + L.conn_bytes);
  const int N = P.tab.N, Np = P.tab.Np, NpM1 = P.tab.NpM1, Nfp = P.tab.Nfp;
  const int64_t K = P.K;
  const int epb = P.epb;
  const bool use_res = P.mode != 0 && P.rkA != T(0);
  const FastDiv by_np(Np), by_npm1(NpM1), by_nfp(Nfp), by_4nfp(4 * Nfp);
    const int64_t e0 = tile * epb;
    const int ne = (int)min64(epb, K - e0);
    __syncthreads();
    // ---- 1. stage q, geometry, connectivity --------------------------------------------
    for (int fld = 0; fld < NF; ++fld)
      copy_g2s(sQ + (size_t)fld * epb * Np, P.q + ((size_t)fld * K + e0) * Np, ne * Np);
    copy_g2s(sGeo, P.geo + e0 * BB_GEO_STRIDE, ne * BB_GEO_STRIDE);
    for (int t = threadIdx.x; t < ne * 4; t += blockDim.x) {
      sConn[t] = __ldg(P.conn + e0 * 4 + t);
      // the face's penalty weights (tau |n|, tau / |n|; 1 and 1 with tau <= 0), once per face:
      // a square root and a division are long sequences on the FP64 pipe
      const T* g = P.geo + (e0 + (t >> 2)) * BB_GEO_STRIDE + 12 + (t & 3);
      const T nx = __ldg(g), ny = __ldg(g + 4), nz = __ldg(g + 8);
      T cp = T(1), cu = T(1);
      if (P.tau > T(0)) {
        const T Jf = sqrt(nx * nx + ny * ny + nz * nz);
        cp = P.tau * Jf;
        cu = P.tau / Jf;
      }
      sPen[2 * t] = cp;
      sPen[2 * t + 1] = cu;
    }
    if (sizeof(T) == 8 && L.stacks) {
      const T* w = reinterpret_cast<const T*>(P.gtab + P.tab.o_wred);
      for (int t = threadIdx.x; t < (N + 1) * (N + 2); t += blockDim.x) sbase[L.out + t] = __ldg(w + t);
    }
    // barycentric weights of J d/dx, J d/dy, J d/dz: g_a = (rxJ, sxJ, txJ, -sum) / 2, once
    // per element rather than per volume point
    for (int t = threadIdx.x; t < ne * 9; t += blockDim.x) {
      const int le = t / 9;
      sGh[t] = T(0.5) * __ldg(P.geo + (e0 + le) * BB_GEO_STRIDE + (t - le * 9));
    }
    __syncthreads();

    // ---- 2. interface flux -------------------------------------------------------------
    for (int it = threadIdx.x; it < ne * 4 * Nfp; it += blockDim.x) {
      const int le = by_4nfp.div(it);
      const int rem = it - le * 4 * Nfp;
      const int f = by_nfp.div(rem), a = rem - f * Nfp;
      const int32_t c = sConn[le * 4 + f];
      const int64_t nbr = (int64_t)((uint32_t)c >> 5);
      const int nface = (c >> 3) & 3, o = c & 7;
      T d[NF];
      const int vM = st.fvol[f * Nfp + a];
      if (nbr >= K || o > 5) {
        atomicOr(P.status, 1);
        for (int fld = 0; fld < NF; ++fld) d[fld] = T(0);
      } else if (!BB_DCHECK(vM < Np && st.fperm[o * Nfp + a] < Nfp, P.status)) {
        for (int fld = 0; fld < NF; ++fld) d[fld] = T(0);
      } else {
        const int ap = st.fperm[o * Nfp + a];
        if (nbr >= e0 && nbr < e0 + ne) {
          const int vP = BB_DCHECK(st.fvol[nface * Nfp + ap] < Np, P.status)
                             ? st.fvol[nface * Nfp + ap] : vM;
          const T* qP = sQ + (size_t)(nbr - e0) * Np + vP;
          const T* qM = sQ + (size_t)le * Np + vM;
#pragma unroll
          for (int fld = 0; fld < NF; ++fld) d[fld] = qP[(size_t)fld * epb * Np] - qM[(size_t)fld * epb * Np];
        } else if (P.trace_in) {
          const T* tp = P.trace_in + ((size_t)nbr * 4 + nface) * NF * Nfp + ap;
          const T* qM = sQ + (size_t)le * Np + vM;
#pragma unroll
          for (int fld = 0; fld < NF; ++fld) d[fld] = __ldg(tp + (size_t)fld * Nfp) - qM[(size_t)fld * epb * Np];
        } else {
          const int vP = BB_DCHECK(st.fvol[nface * Nfp + ap] < Np, P.status)
                             ? st.fvol[nface * Nfp + ap] : vM;
          const T* qP = P.q + (size_t)nbr * Np + vP;
          const T* qM = sQ + (size_t)le * Np + vM;
#pragma unroll
          for (int fld = 0; fld < NF; ++fld) d[fld] = __ldg(qP + (size_t)fld * K * Np) - qM[(size_t)fld * epb * Np];
        }
      }
      const T* g = sGeo + le * BB_GEO_STRIDE;
      const T nx = g[12 + f], ny = g[16 + f], nz = g[20 + f];
      const T cp = sPen[(le * 4 + f) * 2], cu = sPen[(le * 4 + f) * 2 + 1];
      T fl[NF];
      if constexpr (PHYS == BB_ADVECTION || PHYS == BB_ADVECTION3) {
        // 3d_advec_scalar.jl:24-29, 3d_advec.jl:44-45: 0.5 du nxJ - 0.5 du Jf per component
        // (negated, see Phys<BB_ADVECTION>)
        const T Jf = sqrt(nx * nx + ny * ny + nz * nz);
#pragma unroll
        for (int m = 0; m < NF; ++m) fl[m] = -(T(0.5) * d[m] * nx - T(0.5) * d[m] * Jf);
      } else if constexpr (PHYS == BB_WAVE) {
        // 3d_wave.jl:45-54
        // the velocity flux 0.5 B (nx, ny, nz) is stored as the scalar 0.5 B; the lift
        // multiplies its result by the normal
        if constexpr (sizeof(T) == 8) {  // the halves folded into n and cp (exact)
          const T h = fma(T(0.5) * nz, d[3], fma(T(0.5) * ny, d[2], T(0.5) * nx * d[1]));
          fl[0] = fma(T(0.5) * cp, d[0], -h);
          fl[1] = fma(cu, h, -T(0.5) * d[0]);
        } else {
        const T ndotdU = nx * d[1] + ny * d[2] + nz * d[3];
        const T A = cp * d[0] - ndotdU;
        const T B = cu * ndotdU - d[0];
        fl[0] = T(0.5) * A;
        fl[1] = T(0.5) * B;
        }
      } else if constexpr (sizeof(T) == 8) {
        maxwell_flux<T>(d, nx, ny, nz, cp, cu, fl);
      } else {
        // 3d_maxwell.jl:52-63: 0.5 (fx nx + fy ny + fz nz)(du) + 0.5 du - 0.5 n (n.d)
        const T Hx = d[0], Hy = d[1], Hz = d[2], Ex = d[3], Ey = d[4], Ez = d[5];
        const T ndH = nx * Hx + ny * Hy + nz * Hz;
        const T ndE = nx * Ex + ny * Ey + nz * Ez;
        const T ax[6] = {T(0), Ez, -Ey, T(0), -Hz, Hy};
        const T ay[6] = {-Ez, T(0), Ex, Hz, T(0), -Hx};
        const T az[6] = {Ey, -Ex, T(0), -Hy, Hx, T(0)};
        const T nd[6] = {ndH * nx, ndH * ny, ndH * nz, ndE * nx, ndE * ny, ndE * nz};
#pragma unroll
        for (int m = 0; m < 6; ++m)
          fl[m] = T(0.5) * ax[m] * nx + T(0.5) * ay[m] * ny + T(0.5) * az[m] * nz +
                  T(0.5) * (cp * d[m]) - T(0.5) * (cu * nd[m]);
      }
      T* fo = sFlux + ((size_t)(le * 4 + f) * (L.stacks ? NCH : NF)) * Nfp + a;
#pragma unroll
      for (int ch = 0; ch < NCH; ++ch) fo[(size_t)ch * Nfp] = fl[ch];
    }

    // ---- 3a. volume term at degree N-1 (from the last warp on: the flux above started with the
    //          first, and a small tile keeps only some warps busy with each) ------------------
    for (int it = blockDim.x - 1 - threadIdx.x; it < ne * NpM1; it += blockDim.x) {
      const int le = by_npm1.div(it), b = it - le * NpM1;
      const uint32_t c = st.node3m1[b];
      const int i = c & 0xff, j = (c >> 8) & 0xff, k = c >> 16;
      const int idx[4] = {ijk3(N, i + 1, j, k), ijk3(N, i, j + 1, k), ijk3(N, i, j, k + 1),
                          ijk3(N, i, j, k)};
      // barycentric weights of d/dx, d/dy, d/dz (times J), staged per element; the fourth
      // weight is implied by the differences below
      const T* gx = sGh + le * 9;  // gx[a], then gy = gx + 3, gz = gx + 6
      const T* gy = gx + 3;
      const T* gz = gx + 6;
      const T* q0 = sQ + (size_t)le * Np;
      auto F = [&](int fld, int a) { return q0[(size_t)fld * epb * Np + idx[a]]; };
      T w[NW];
#pragma unroll
      for (int m = 0; m < NW; ++m) w[m] = T(0);
      // sum_a g_a x(beta+e_a) with sum_a g_a = 0, formed as sum_{a<3} g_a (x_a - x_3) so
      // that smooth data cancels in the differences (as the reference's Dr = (D0 - D3)/2)
      if constexpr (PHYS == BB_ADVECTION || PHYS == BB_ADVECTION3) {
        const T u3 = F(0, 3);
#pragma unroll
        for (int a = 0; a < 3; ++a) w[0] += gx[a] * (F(0, a) - u3);  // J du/dx
      } else if constexpr (PHYS == BB_WAVE) {
        const T p3 = F(0, 3), u3 = F(1, 3), v3 = F(2, 3), w3 = F(3, 3);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const T p = F(0, a) - p3, u = F(1, a) - u3, v = F(2, a) - v3, ww = F(3, a) - w3;
          if constexpr (sizeof(T) == 8) w[0] = fma(gz[a], ww, fma(gy[a], v, fma(gx[a], u, w[0])));
          else w[0] += gx[a] * u + gy[a] * v + gz[a] * ww;
          w[1] += gx[a] * p;
          w[2] += gy[a] * p;
          w[3] += gz[a] * p;
        }
      } else {
        const T Hx3 = F(0, 3), Hy3 = F(1, 3), Hz3 = F(2, 3);
        const T Ex3 = F(3, 3), Ey3 = F(4, 3), Ez3 = F(5, 3);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const T Hx = F(0, a) - Hx3, Hy = F(1, a) - Hy3, Hz = F(2, a) - Hz3;
          const T Ex = F(3, a) - Ex3, Ey = F(4, a) - Ey3, Ez = F(5, a) - Ez3;
          if constexpr (sizeof(T) == 8) {
            maxwell_curl<T>(w, gx[a], gy[a], gz[a], Hx, Hy, Hz, Ex, Ey, Ez);
            continue;
          }
          w[0] += -gy[a] * Ez + gz[a] * Ey;  // d/dt Hx = -dEz/dy + dEy/dz
          w[1] += gx[a] * Ez - gz[a] * Ex;   // d/dt Hy
          w[2] += -gx[a] * Ey + gy[a] * Ex;  // d/dt Hz
          w[3] += gy[a] * Hz - gz[a] * Hy;   // d/dt Ex
          w[4] += -gx[a] * Hz + gz[a] * Hx;  // d/dt Ey
          w[5] += gx[a] * Hy - gy[a] * Hx;   // d/dt Ez
        }
      }
#pragma unroll
      for (int m = 0; m < NW; ++m) sWork[((size_t)m * epb + le) * NpM1 + b] = w[m];
    }
    __syncthreads();
    if (L.stacks) {
      // ---- 3-5 with whole stacks: lift every face, then per coefficient the volume term, the
      // four faces (t=-1 first as src/BernsteinLift.jl:202-205), 1/J and the update -----------
      const int gs = Np | 1;
      T* sG = sbase + L.stack;
      lift_stacks<T>(N, ne * 4 * NCH, st.node2, sFlux, Nfp, sG, gs, sbase + L.out);
      // one thread per coefficient and group of FG fields: the wave's all (its faces' scalar chain
      // serves three), Maxwell's by twos, so that more warps share the pass (K = 2,058, N = 9:
      // 256 -> 252 us per stage; the wave by twos 131 -> 140 us at N = 7, K = 4,374)
      constexpr int FG = PHYS == BB_WAVE ? NF : PHYS == BB_MAXWELL ? 2 : 1;
      const uint4* gtab4 = reinterpret_cast<const uint4*>(P.gtab + P.tab.o_gather);
      const FastDiv by_gnp(NF / FG * Np);
      for (int it = threadIdx.x; it < ne * (NF / FG) * Np; it += blockDim.x) {
        const int le = by_gnp.div(it), rem = it - le * (NF / FG) * Np;
        const int fg = by_np.div(rem), n = rem - fg * Np, f0 = fg * FG;
        const uint4 ga = __ldg(gtab4 + n);
        const uint32_t c = st.node3[n];
        const int al[4] = {(int)(c & 0xff), (int)((c >> 8) & 0xff), (int)(c >> 16),
                           N - (int)(c & 0xff) - (int)((c >> 8) & 0xff) - (int)(c >> 16)};
        const int xb[4] = {(int)(ga.x & 0xffff), (int)(ga.x >> 16), (int)(ga.y & 0xffff),
                           (int)(ga.y >> 16)};
        const int pf[4] = {(int)(ga.z & 0xffff), (int)(ga.z >> 16), (int)(ga.w & 0xffff),
                           (int)(ga.w >> 16)};
        const size_t at = ((size_t)f0 * K + e0 + le) * Np + n, fs = (size_t)K * Np;
        T res[FG];  // the first stage of a step (rkA = 0) ignores what it holds
#pragma unroll
        for (int m = 0; m < FG; ++m) res[m] = use_res ? P.res[at + m * fs] : T(0);
        T acc[FG];
#pragma unroll
        for (int m = 0; m < FG; ++m) acc[m] = T(0);
        if (NW == NF || f0 < NW) {  // fields past NW have no volume term
          const T* wb = sWork + ((size_t)f0 * epb + le) * NpM1;
          const size_t ws = (size_t)epb * NpM1;
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            if (al[b] == 0) continue;
            const T v = small_int<T>(al[b]);
#pragma unroll
            for (int m = 0; m < FG; ++m) acc[m] = fma(v, wb[m * ws + xb[b]], acc[m]);
          }
          if (Phys<PHYS>::vol_sign < 0) {
#pragma unroll
            for (int m = 0; m < FG; ++m) acc[m] = -acc[m];
          }
        }
        // the faces, t=-1 first as src/BernsteinLift.jl:202-205
        const T* nc = sGeo + le * BB_GEO_STRIDE + 12;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int f = (q + 3) & 3;  // faces 3, 0, 1, 2
          const T* g = sG + (size_t)((le * 4 + f) * NCH) * gs + pf[f];
          if constexpr (PHYS == BB_WAVE) {
            // field 0 takes the pressure chain, velocity component m - 1 the scalar chain times
            // that component of the normal
            const T s = g[gs];
            acc[0] += g[0];
#pragma unroll
            for (int m = 1; m < NF; ++m) acc[m] = fma(nc[4 * (m - 1) + f], s, acc[m]);
          } else {
#pragma unroll
            for (int m = 0; m < FG; ++m) acc[m] += g[(size_t)(f0 + m) * gs];
          }
        }
        const T invJ = sGeo[le * BB_GEO_STRIDE + 9];
        if (P.mode == 0) {
#pragma unroll
          for (int m = 0; m < FG; ++m) P.rhs[at + m * fs] = acc[m] * invJ;
        } else {
          const T dtJ = P.dt * invJ;
#pragma unroll
          for (int m = 0; m < FG; ++m) {
            T* sq = sQ + ((size_t)(f0 + m) * epb + le) * Np + n;
            T r;
            if constexpr (sizeof(T) == 8) r = fma(dtJ, acc[m], P.rkA * res[m]);
            else r = fma(P.rkA, res[m], P.dt * (acc[m] * invJ));
            const T qn = fma(P.rkB, r, *sq);
            P.res[at + m * fs] = r;
            P.q[at + m * fs] = qn;
            *sq = qn;
          }
        }
      }
      if (P.mode != 0 && P.trace_out) {
        __syncthreads();
        write_traces<T, NF>(P, st, sQ, sConn, e0, ne);
      }
      return;
    }
    // ---- 3b. elevate back to degree N: out(alpha) = sign * sum_b alpha_b w(alpha - e_b) -
    for (int it = threadIdx.x; it < ne * Np; it += blockDim.x) {
      const int le = by_np.div(it), n = it - le * Np;
      const uint32_t c = st.node3[n];
      const int i = c & 0xff, j = (c >> 8) & 0xff, k = c >> 16, l = N - i - j - k;
      T acc[NW];
#pragma unroll
      for (int m = 0; m < NW; ++m) acc[m] = T(0);
      const T* wb = sWork + (size_t)le * NpM1;
      const size_t ws = (size_t)epb * NpM1;
      if (i > 0) {
        const int x = ijk3(N - 1, i - 1, j, k);
#pragma unroll
        for (int m = 0; m < NW; ++m) acc[m] += small_int<T>(i) * wb[m * ws + x];
      }
      if (j > 0) {
        const int x = ijk3(N - 1, i, j - 1, k);
#pragma unroll
        for (int m = 0; m < NW; ++m) acc[m] += small_int<T>(j) * wb[m * ws + x];
      }
      if (k > 0) {
        const int x = ijk3(N - 1, i, j, k - 1);
#pragma unroll
        for (int m = 0; m < NW; ++m) acc[m] += small_int<T>(k) * wb[m * ws + x];
      }
      if (l > 0) {
        const int x = ijk3(N - 1, i, j, k);
#pragma unroll
        for (int m = 0; m < NW; ++m) acc[m] += small_int<T>(l) * wb[m * ws + x];
      }
#pragma unroll
      for (int m = 0; m < NF; ++m) {
        const T v = m < NW ? acc[m < NW ? m : 0] : T(0);  // fields past NW: no volume term
        sOut[((size_t)m * epb + le) * Np + n] = Phys<PHYS>::vol_sign < 0 ? -v : v;
      }
    }
    __syncthreads();

    // ---- 4. lift of the face fluxes, face t=-1 first as src/BernsteinLift.jl:202-205 ----
    {
      const int S = np2(N + 1);
      T* bufA = sWork;
      T* bufB = sWork + (size_t)epb * NCH * S;
      for (int q = 0; q < 4; ++q) {
        const int f = (q + 3) & 3;  // faces 3, 0, 1, 2
        lift_face_accumulate<T, PHYS == BB_WAVE>(N, f, ne, NCH, st.node2,
                                                 sFlux + (size_t)f * NF * Nfp, 4 * NF * Nfp, Nfp,
                                                 sOut, Np, epb * Np, bufA, bufB, sGeo + 12 + f);
      }
    }

    // ---- 5. divide by J, RK update, write back -----------------------------------------
    if (P.mode == 0) {
      for (int fld = 0; fld < NF; ++fld) {
        T* dst = P.rhs + ((size_t)fld * K + e0) * Np;
        const T* src = sOut + (size_t)fld * epb * Np;
        for (int t = threadIdx.x; t < ne * Np; t += blockDim.x) {
          const int le = by_np.div(t);
          dst[t] = src[t] * sGeo[le * BB_GEO_STRIDE + 9];
        }
      }
    } else {
      for (int fld = 0; fld < NF; ++fld) {
        T* gq = P.q + ((size_t)fld * K + e0) * Np;
        T* gr = P.res + ((size_t)fld * K + e0) * Np;
        T* sq = sQ + (size_t)fld * epb * Np;
        const T* so = sOut + (size_t)fld * epb * Np;
        for (int t = threadIdx.x; t < ne * Np; t += blockDim.x) {
          const int le = by_np.div(t);
          const T rhs = so[t] * sGeo[le * BB_GEO_STRIDE + 9];
          const T r = P.rkA * (use_res ? gr[t] : T(0)) + P.dt * rhs;
          const T qn = sq[t] + P.rkB * r;
          gr[t] = r;
          gq[t] = qn;
          sq[t] = qn;
        }
      }
      if (P.trace_out) {
        __syncthreads();
        write_traces<T, NF>(P, st, sQ, sConn, e0, ne);
      }
    }
}

// ---- traces of a whole state ------------------------------------------------------------
// Writes the traces of the faces that leave their tile (of epb elements, from element 0 on) of
// elements [e_begin, e_end) of q into the trace buffer: the stage kernels read no others.
// An element's 4 NF Nfp trace entries are contiguous in the buffer; each block first decodes
// entry i into (field, volume node) once (shared table). Then each thread gathers four entries at
// a time from the element's field rows and stores them at once, over kExtractElems elements per
// turn, so that several gathers are in flight (wave N = 9, K = 196,608: one entry at a time, element
// after element, 300 us; four at a time 250; without the faces inside a tile, a third of them at
// four elements a tile, about 205. All faces' traffic at the HBM rate: 204).
constexpr int kExtractElems = 8;

template <class T, int NF>
__global__ void __launch_bounds__(256)
    extract_traces_kernel(DegTables tab, const uint32_t* __restrict__ gtab, int64_t K,
                          const int32_t* __restrict__ conn, int epb, const T* __restrict__ q,
                          T* __restrict__ tr, int64_t e_begin, int64_t e_end) {
  extern __shared__ __align__(16) uint32_t s_src[];  // entry i: face << 20 | field << 16 | volume node
  const int Np = tab.Np, Nfp = tab.Nfp, W = 4 * NF * Nfp;
  const uint16_t* fvol = reinterpret_cast<const uint16_t*>(gtab + tab.o_fvol);
  for (int i = threadIdx.x; i < W; i += blockDim.x) {
    const int f = i / (NF * Nfp), rem = i - f * NF * Nfp, fld = rem / Nfp, a = rem - fld * Nfp;
    s_src[i] = ((uint32_t)f << 20) | ((uint32_t)fld << 16) | fvol[f * Nfp + a];
  }
  __syncthreads();
  const size_t field = (size_t)K * Np;
  const int Q = NF * Nfp;  // groups of four entries per element
  const FastDiv by_q(Q);
  for (int64_t e0 = e_begin + (int64_t)blockIdx.x * kExtractElems; e0 < e_end;
       e0 += (int64_t)gridDim.x * kExtractElems) {
    const int ne = (int)min64(kExtractElems, e_end - e0);
    for (int it = threadIdx.x; it < ne * Q; it += blockDim.x) {
      const int le = by_q.div(it), g = it - le * Q;
      const uint4 v = reinterpret_cast<const uint4*>(s_src)[g];
      const int64_t e = e0 + le;
      auto leaves = [&](uint32_t f) {
        const int64_t nbr = (int64_t)((uint32_t)__ldg(conn + e * 4 + f) >> 5);
        const int64_t first = e - (uint32_t)e % (uint32_t)epb;  // e < 2^27
        return nbr < first || nbr >= first + epb;
      };
      if (!leaves(v.x >> 20) && (v.w >> 20 == v.x >> 20 || !leaves(v.w >> 20))) continue;
      const T* qe = q + (size_t)e * Np;
      auto at = [&](uint32_t x) { return __ldg(qe + ((x >> 16) & 15u) * field + (x & 0xffffu)); };
      T* te = tr + (size_t)(e0 + le) * W + 4 * g;
      if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(te) = make_float4(at(v.x), at(v.y), at(v.z), at(v.w));
      } else {
        reinterpret_cast<double2*>(te)[0] = make_double2(at(v.x), at(v.y));
        reinterpret_cast<double2*>(te)[1] = make_double2(at(v.z), at(v.w));
      }
    }
  }
}

// Launches it for elements [e0, e1) of an nf-field state; tr 16-byte aligned.
template <class T>
void extract_traces(const DegTables& t, int nf, int64_t K, const int32_t* conn, int epb,
                    const void* q, void* tr, int64_t e0, int64_t e1, int num_sms,
                    cudaStream_t st) {
  const int64_t turns = (e1 - e0 + kExtractElems - 1) / kExtractElems;
  const int grid = (int)min64(turns, (int64_t)num_sms * 8);
  const size_t smem = (size_t)4 * nf * t.Nfp * sizeof(uint32_t);
  auto go = [&](auto kern) {
    kern<<<grid, 256, smem, st>>>(t, t.d_words, K, conn, epb, (const T*)q, (T*)tr, e0, e1);
  };
  if (nf == 4) go(extract_traces_kernel<T, 4>);
  else if (nf == 1) go(extract_traces_kernel<T, 1>);
  else if (nf == 3) go(extract_traces_kernel<T, 3>);
  else go(extract_traces_kernel<T, 6>);
}
