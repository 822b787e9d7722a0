// bx_stage_flat.cuh -- fused explicit stage kernel of 2D blocks (FP64): one CTA
// per block, one sweep per direction.
//
// The arithmetic is the reference's, operation by operation (numerical_flux,
// IEEE divisions and square roots, no contraction: compiled with
// --fmad=false).  Runs with the minmod limiter amplify the rounding of a step
// in 2D: the flux functions of the 3D kernel, with a thread per face and 20
// warps per SM, took 39 us per step at 384 x 384 where this kernel takes 78,
// but gave digits up to 2e-14 of the norm apart after 50 steps.  Kept of that
// is the end of the time step in the last CTA.  The gather loads through the
// read-only path, so the kernel does not start before the one that writes the
// state has ended.
//
// Five CTAs per SM (128 registers): Rusanov and HLLD fit; Roe spills 320 bytes
// and gains all the same (210 registers, three CTAs: 181 instead of 124 us per
// step at 384 x 384).  Linde needs 150 registers, for four; with the limit of 128
// it spills 104 bytes.  It takes five where that saves a wave of CTAs, else four
// (us per step with four / five: 90 blocks 20.9 / 22.5, 1024 41.4 / 43.5, 1600
// 59.8 / 61.6, 2304 78.6 / 80.6, but 1357 blocks 54 / 46, 3600 123 / 115).
#pragma once
#include "bx_stage.cuh"

namespace bx {

using Flat = Shape<8, 8, 1>;  // 96 threads: 72 faces per direction, 64 cells

// the cell's accumulators, held in registers across the two sweeps
struct CellAcc {
  double chg[8];    // flux divergence sum (rho, m, B, E)
  double divBint;   // DivBInternal_C
  double dbf[4];    // dB1nFace1..4
  double vdt;       // sum over dims of max(Vdt_left, Vdt_right)
};

template <int D, int FLUX>
__device__ __forceinline__ void sweep(const StageArgs &a, const BlockGeom &g, const double *tile, double *fbuf,
                                      CellAcc &acc, int &err) {
  using S = Flat;
  constexpr int NF = D == 0 ? S::NFX : S::NFY;
  for (int f = threadIdx.x; f < NF; f += blockDim.x) {
    int i, j, k;
    face_decode<S, D>(f, i, j, k);
    double L[8], R[8], F[8], vdt;
    face_states<S, D>(tile, i, j, k, a.nOrder, a.limiter, a.beta, L, R);
    if (FLUX == kFluxRoe) {
      // UseRS7 (src/ModFaceFlux.f90:600-625): each face state takes the
      // normal field of its cell before the div B slots are formed; the
      // Roe dissipation also uses the cells' normal velocities
      constexpr int st = D == 0 ? 1 : S::TX;
      const int c = S::t(i, j, k);
      const double cbL = tile[(kBx + D) * S::NT + c - st], cbR = tile[(kBx + D) * S::NT + c];
      const double cuL = tile[(kUx + D) * S::NT + c - st], cuR = tile[(kUx + D) * S::NT + c];
      const double dBnR = R[kBx + D] - cbR;
      R[kBx + D] = R[kBx + D] - dBnR;
      const double dBnL = L[kBx + D] - cbL;
      L[kBx + D] = L[kBx + D] - dBnL;
      fbuf[9 * S::NFMAX + f] = L[kBx + D];
      fbuf[10 * S::NFMAX + f] = R[kBx + D];
      vdt = roe_flux<D>(L, R, cuL, cuR, dBnL, dBnR, a.gamma, a.invGm1, g.area[D], F, 1);
    } else {
      fbuf[9 * S::NFMAX + f] = L[kBx + D];
      fbuf[10 * S::NFMAX + f] = R[kBx + D];
      if (!numerical_flux<D, FLUX>(L, R, a.gamma, a.invGm1, g.area[D], F, vdt)) err = 1;
    }
#pragma unroll
    for (int v = 0; v < 8; v++) fbuf[v * S::NFMAX + f] = F[v];
    fbuf[8 * S::NFMAX + f] = vdt;
  }
  __syncthreads();
  const int c = threadIdx.x;
  if (c < S::NC) {
    const double h = g.invHalf[D];  // DxInvHalf = 0.5/CellSize
    const int i = c % S::NI, j = c / S::NI;
    const int f0 = face_index<S, D>(i, j, 0), f1 = face_index<S, D>(i + (D == 0), j + (D == 1), 0);
#pragma unroll
    for (int v = 0; v < 8; v++) {
      const double F0 = fbuf[v * S::NFMAX + f0], F1 = fbuf[v * S::NFMAX + f1];
      acc.chg[v] = D == 0 ? F0 - F1 : acc.chg[v] + F0 - F1;
    }
    const double L0 = fbuf[9 * S::NFMAX + f0], R0 = fbuf[10 * S::NFMAX + f0];
    const double L1 = fbuf[9 * S::NFMAX + f1], R1 = fbuf[10 * S::NFMAX + f1];
    // calc_divb_source (src/ModCalcSource.f90:1694-1891)
    const double inner = 2 * h * (L1 - R0);
    acc.divBint = D == 0 ? inner : acc.divBint + inner;
    acc.dbf[2 * D] = h * (R0 - L0);
    acc.dbf[2 * D + 1] = h * (R1 - L1);
    const double vmax = fmax(fbuf[8 * S::NFMAX + f0], fbuf[8 * S::NFMAX + f1]);
    acc.vdt = D == 0 ? vmax : acc.vdt + vmax;
  }
  __syncthreads();
}

// CTAS: CTAs per SM that the register limit allows for
template <int FLUX, int CTAS>
__global__ void __launch_bounds__(Flat::NTHREAD, CTAS) stage_flat_kernel(const StageArgs a) {
  using S = Flat;
  __shared__ double tile[8 * S::NT], fbuf[S::NSLOT * S::NFMAX], wmin[S::NTHREAD / 32];
  __shared__ StepState step;

  const int b = a.order[blockIdx.x];
  int nb[6];
#pragma unroll
  for (int q = 0; q < 6; q++) nb[q] = a.nbr[6 * b + q];
  const BlockGeom g = a.geom[b];

  gather_tile<S, double>(reinterpret_cast<const double *>(a.in), nb, b, tile);
  load_step(a, step);
  __syncthreads();

  CellAcc acc;
  int err = 0;
  sweep<0, FLUX>(a, g, tile, fbuf, acc, err);
  sweep<1, FLUX>(a, g, tile, fbuf, acc, err);
  if (err) atomicOr(&a.ts->errFlag, kErrHlld);

  // ---- update (update_state_normal + update_explicit) --------------------
  double dtmin = 1e300;
  const int c = threadIdx.x;
  if (c < S::NC) {
    const double DtNoCfl = a.ts->DtNoCfl, V = g.volume;
    const double *__restrict__ old = a.old + (size_t)b * 8 * S::NC;
    double *__restrict__ out = reinterpret_cast<double *>(a.out) + (size_t)b * 8 * S::NC;
    double o[8];
#pragma unroll
    for (int v = 0; v < 8; v++) o[v] = old[v * S::NC + c];
    if (a.computeDt) dtmin = V / acc.vdt;
    if (DtNoCfl == 0.0) {  // IsTimeAccurate .and. Dt == 0: state unchanged, floored
      o[kP] = limit_pressure(o[kRho], o[kP], a.fl.pMin, a.fl.tMin, a.fl.massIon);
#pragma unroll
      for (int v = 0; v < 8; v++) out[v * S::NC + c] = o[v];
    } else {
      const double DtLocal = a.dtFactor * DtNoCfl;
      double src[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (a.useDivb) {
        const double divB = acc.divBint + acc.dbf[0] + acc.dbf[1] + acc.dbf[2] + acc.dbf[3];
        const int tt = S::t(c % S::NI, c / S::NI, 0);
        const double ux = tile[kUx * S::NT + tt], uy = tile[kUy * S::NT + tt], uz = tile[kUz * S::NT + tt];
        const double bx = tile[kBx * S::NT + tt], by = tile[kBy * S::NT + tt], bz = tile[kBz * S::NT + tt];
        src[kBx] = 0 - divB * ux; src[kBy] = 0 - divB * uy; src[kBz] = 0 - divB * uz;
        src[kE] = 0 - divB * (bx * ux + by * uy + bz * uz);
        src[kUx] = 0 + (0 - divB * bx); src[kUy] = 0 + (0 - divB * by); src[kUz] = 0 + (0 - divB * bz);
      }
      double s[8];
#pragma unroll
      for (int v = 0; v < 8; v++) s[v] = DtLocal * (src[v] + acc.chg[v] / V);
      // pressure_to_energy(StateOld) (src/ModEnergy.f90:47)
      double e = a.invGm1 * o[kP] + 0.5 * (o[kUx] * o[kUx] + o[kUy] * o[kUy] + o[kUz] * o[kUz]) / o[kRho];
      e = e + 0.5 * (o[kBx] * o[kBx] + o[kBy] * o[kBy] + o[kBz] * o[kBz]);
      double n[8];
#pragma unroll
      for (int v = 0; v < 7; v++) n[v] = o[v] + s[v];
      e = e + s[kE];
      if (a.fl.rhoMin > 0.0) n[kRho] = fmax(a.fl.rhoMin, n[kRho]);  // UseRhoMin
      // energy_to_pressure (src/ModEnergy.f90:243), then limit_pressure
      const double p = e - 0.5 * (n[kBx] * n[kBx] + n[kBy] * n[kBy] + n[kBz] * n[kBz]);
      n[kP] = (a.gamma - 1.0) * (p - 0.5 * (n[kUx] * n[kUx] + n[kUy] * n[kUy] + n[kUz] * n[kUz]) / n[kRho]);
      n[kP] = limit_pressure(n[kRho], n[kP], a.fl.pMin, a.fl.tMin, a.fl.massIon);
#pragma unroll
      for (int v = 0; v < 8; v++) out[v * S::NC + c] = n[v];
    }
  }

  if (a.computeDt) {
    // block minimum (calc_block_dt) then grid minimum (MPI_MIN of
    // set_global_timestep) via atomicMin on the ordered bits
    for (int off = 16; off > 0; off >>= 1) dtmin = fmin(dtmin, __shfl_xor_sync(0xffffffffu, dtmin, off));
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = dtmin;
    __syncthreads();
    if (threadIdx.x == 0) {
      double m = wmin[0];
      for (int w = 1; w < S::NTHREAD / 32; w++) m = fmin(m, wmin[w]);
      if (a.dtBlock) store_block_dt(a.dtBlock, b, m);
      atomicMin(&a.ts->DtMinBits, dbits(m));
    }
  }
  finish_stage(a, step);
}

}  // namespace bx
