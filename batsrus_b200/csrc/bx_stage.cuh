// bx_stage.cuh -- block geometry, gather and face states of the per-block
// kernels (bx_compat.cu) and of the stage kernel of 2D blocks (bx_stage_flat.cuh).
#pragma once
#include <cstdint>

#include "bx_device.h"
#include "bx_physics.cuh"

namespace bx {

template <int NI_, int NJ_, int NK_>
struct Shape {
  static constexpr int NI = NI_, NJ = NJ_, NK = NK_;
  static constexpr int NDIM = NK > 1 ? 3 : (NJ > 1 ? 2 : 1);
  static constexpr int GY = NJ > 1 ? 2 : 0, GZ = NK > 1 ? 2 : 0;
  static constexpr int TX = NI + 4, TY = NJ + 2 * GY, TZ = NK + 2 * GZ;
  static constexpr int NT = TX * TY * TZ;
  static constexpr int NC = NI * NJ * NK;
  static constexpr int NFX = (NI + 1) * NJ * NK;
  static constexpr int NFY = NDIM > 1 ? NI * (NJ + 1) * NK : 0;
  static constexpr int NFZ = NDIM > 2 ? NI * NJ * (NK + 1) : 0;
  static constexpr int NFMAX = NFX > NFY ? (NFX > NFZ ? NFX : NFZ) : (NFY > NFZ ? NFY : NFZ);
  static constexpr int NHX = 4 * NJ * NK;
  static constexpr int NHY = NDIM > 1 ? 4 * NI * NK : 0;
  static constexpr int NHZ = NDIM > 2 ? 4 * NI * NJ : 0;
  static constexpr int NLOAD = NC + NHX + NHY + NHZ;
  static constexpr int NTHREAD = NC >= 256 ? 256 : ((NFX + 31) / 32) * 32;
  static constexpr int CPT = (NC + NTHREAD - 1) / NTHREAD;  // cells per thread
  static constexpr int NSLOT = 11;  // 8 fluxes, Vdt, BnL, BnR
  __host__ __device__ static constexpr int t(int i, int j, int k) {
    return (i + 2) + TX * ((j + GY) + TY * (k + GZ));
  }
};

// ordered bits of a non-negative double: the unsigned integer order equals
// the numerical order, so atomicMin on the bits gives the minimum double
__device__ __forceinline__ unsigned long long dbits(double x) {
  return (unsigned long long)__double_as_longlong(x);
}

template <typename T> __device__ __forceinline__ T ldg_t(const T *p) { return __ldg(p); }

// ---------------------------------------------------------------------------
// gather (exchange_messages fused): fill the primitive tile of block b
template <class S, typename Real, typename InT>
__device__ __forceinline__ void gather_tile(const InT *__restrict__ in, const int *nb, int b,
                                            Real *tile) {
  for (int q = threadIdx.x; q < S::NLOAD; q += blockDim.x) {
    int ti, tj, tk;    // tile coordinates (0-based interior, may be -2..N+1)
    int src, si, sj, sk;  // source block and cell
    int r = q;
    if (r < S::NC) {
      ti = r % S::NI; tj = (r / S::NI) % S::NJ; tk = r / (S::NI * S::NJ);
      src = b; si = ti; sj = tj; sk = tk;
    } else if ((r -= S::NC) < S::NHX) {
      const int l = r & 1, jk = (r >> 1) % (S::NJ * S::NK), side = (r >> 1) / (S::NJ * S::NK);
      tj = jk % S::NJ; tk = jk / S::NJ; sj = tj; sk = tk;
      const int n = nb[side];
      ti = side == 0 ? l - 2 : S::NI + l;
      if (n >= 0) { src = n; si = side == 0 ? S::NI - 2 + l : l; }
      else { src = b; si = side == 0 ? 0 : S::NI - 1; }
    } else if ((r -= S::NHX) < S::NHY) {
      ti = r % S::NI; const int l = (r / S::NI) & 1;
      tk = (r / (2 * S::NI)) % S::NK; const int side = r / (2 * S::NI * S::NK);
      si = ti; sk = tk;
      const int n = nb[2 + side];
      tj = side == 0 ? l - 2 : S::NJ + l;
      if (n >= 0) { src = n; sj = side == 0 ? S::NJ - 2 + l : l; }
      else { src = b; sj = side == 0 ? 0 : S::NJ - 1; }
    } else {
      r -= S::NHY;
      ti = r % S::NI; tj = (r / S::NI) % S::NJ;
      const int l = (r / (S::NI * S::NJ)) & 1, side = r / (2 * S::NI * S::NJ);
      si = ti; sj = tj;
      const int n = nb[4 + side];
      tk = side == 0 ? l - 2 : S::NK + l;
      if (n >= 0) { src = n; sk = side == 0 ? S::NK - 2 + l : l; }
      else { src = b; sk = side == 0 ? 0 : S::NK - 1; }
    }
    const InT *p = in + (size_t)src * 8 * S::NC + si + S::NI * (sj + S::NJ * sk);
    Real u[8];
#pragma unroll
    for (int v = 0; v < 8; v++) u[v] = (Real)ldg_t(p + v * S::NC);
    // calc_primitives (src/ModFaceValue.f90:1530-1621): u = (1/rho) rhoU
    const Real rhoInv = Real(1) / u[kRho];
    u[kUx] = rhoInv * u[kUx]; u[kUy] = rhoInv * u[kUy]; u[kUz] = rhoInv * u[kUz];
    const int tt = S::t(ti, tj, tk);
#pragma unroll
    for (int v = 0; v < 8; v++) tile[v * S::NT + tt] = u[v];
  }
}

// face states of direction D at face (i,j,k) (face index along D is the
// index of the cell on its right) -- get_face{x,y,z}_first/second
template <class S, int D, typename Real>
__device__ __forceinline__ void face_states(const Real *tile, int i, int j, int k, int nOrder, int lim,
                                            Real beta, Real (&L)[8], Real (&R)[8]) {
  constexpr int st = D == 0 ? 1 : (D == 1 ? S::TX : S::TX * S::TY);
  const int c = S::t(i, j, k);
#pragma unroll
  for (int v = 0; v < 8; v++) {
    const Real *T = tile + v * S::NT + c;
    if (nOrder == 1) {
      L[v] = T[-st];
      R[v] = T[0];
    } else {
      limited_face(lim, beta, T[-2 * st], T[-st], T[0], T[st], L[v], R[v]);
    }
  }
}

template <class S, int D>
__device__ __forceinline__ void face_decode(int f, int &i, int &j, int &k) {
  if (D == 0) { i = f % (S::NI + 1); j = (f / (S::NI + 1)) % S::NJ; k = f / ((S::NI + 1) * S::NJ); }
  else if (D == 1) { i = f % S::NI; j = (f / S::NI) % (S::NJ + 1); k = f / (S::NI * (S::NJ + 1)); }
  else { i = f % S::NI; j = (f / S::NI) % S::NJ; k = f / (S::NI * S::NJ); }
}

template <class S, int D>
__device__ __forceinline__ int face_index(int i, int j, int k) {
  if (D == 0) return i + (S::NI + 1) * (j + S::NJ * k);
  if (D == 1) return i + S::NI * (j + (S::NJ + 1) * k);
  return i + S::NI * (j + S::NJ * k);
}

}  // namespace bx
