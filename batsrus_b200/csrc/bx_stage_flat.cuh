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
// No limit on the registers: 128 (Rusanov), 148 (Linde), 122 (HLLD) and 212 (Roe)
// hold five, four, five and three CTAs per SM without spills; a limit of 128
// for five CTAs spilled 120 bytes of Linde's and 320 of Roe's: Linde 81.2 us
// per step at 384 x 384 instead of 78.3, 23.0 instead of 21.2 on 10 x 9 blocks.
#pragma once
#include "bx_stage.cuh"

namespace bx {

// per-cell accumulators held in registers across the three sweeps
struct CellAcc {
  double chg[8];    // flux divergence sum (rho, m, B, E)
  double divBint;   // DivBInternal_C
  double dbf[6];    // dB1nFace1..6
  double vdt;       // sum over dims of max(Vdt_left, Vdt_right)
};

template <class S, int D, int FLUX, typename Real>
__device__ __forceinline__ void sweep(const StageArgs &a, const BlockGeom &g, const Real *tile,
                                      Real *fbuf, CellAcc (&acc)[S::CPT], int &err) {
  constexpr int NF = D == 0 ? S::NFX : (D == 1 ? S::NFY : S::NFZ);
  const Real gamma = (Real)a.gamma, invGm1 = (Real)a.invGm1, beta = (Real)a.beta;
  const Real area = (Real)g.area[D];
  for (int f = threadIdx.x; f < NF; f += blockDim.x) {
    int i, j, k;
    face_decode<S, D>(f, i, j, k);
    Real L[8], R[8], F[8], vdt;
    face_states<S, D>(tile, i, j, k, a.nOrder, a.limiter, beta, L, R);
    if (FLUX == kFluxRoe) {
      // UseRS7 (src/ModFaceFlux.f90:600-625): each face state takes the
      // normal field of its cell before the div B slots are formed; the
      // Roe dissipation also uses the cells' normal velocities
      constexpr int st = D == 0 ? 1 : (D == 1 ? S::TX : S::TX * S::TY);
      const int c = S::t(i, j, k);
      const Real cbL = tile[(kBx + D) * S::NT + c - st], cbR = tile[(kBx + D) * S::NT + c];
      const Real cuL = tile[(kUx + D) * S::NT + c - st], cuR = tile[(kUx + D) * S::NT + c];
      const Real dBnR = R[kBx + D] - cbR;
      R[kBx + D] = R[kBx + D] - dBnR;
      const Real dBnL = L[kBx + D] - cbL;
      L[kBx + D] = L[kBx + D] - dBnL;
      fbuf[9 * S::NFMAX + f] = L[kBx + D];
      fbuf[10 * S::NFMAX + f] = R[kBx + D];
      vdt = roe_flux<D>(L, R, cuL, cuR, dBnL, dBnR, gamma, invGm1, area, F, 1);
    } else {
      fbuf[9 * S::NFMAX + f] = L[kBx + D];
      fbuf[10 * S::NFMAX + f] = R[kBx + D];
      if (!numerical_flux<D, FLUX>(L, R, gamma, invGm1, area, F, vdt)) err = 1;
    }
#pragma unroll
    for (int v = 0; v < 8; v++) fbuf[v * S::NFMAX + f] = F[v];
    fbuf[8 * S::NFMAX + f] = vdt;
  }
  __syncthreads();
  const double h = g.invHalf[D];  // DxInvHalf = 0.5/CellSize
#pragma unroll
  for (int m = 0; m < S::CPT; m++) {
    const int c = threadIdx.x + m * S::NTHREAD;
    if (c < S::NC) {
      const int i = c % S::NI, j = (c / S::NI) % S::NJ, k = c / (S::NI * S::NJ);
      const int f0 = face_index<S, D>(i, j, k);
      const int f1 = face_index<S, D>(i + (D == 0), j + (D == 1), k + (D == 2));
#pragma unroll
      for (int v = 0; v < 8; v++) {
        const double F0 = (double)fbuf[v * S::NFMAX + f0], F1 = (double)fbuf[v * S::NFMAX + f1];
        acc[m].chg[v] = D == 0 ? F0 - F1 : acc[m].chg[v] + F0 - F1;
      }
      const double L0 = (double)fbuf[9 * S::NFMAX + f0], R0 = (double)fbuf[10 * S::NFMAX + f0];
      const double L1 = (double)fbuf[9 * S::NFMAX + f1], R1 = (double)fbuf[10 * S::NFMAX + f1];
      // calc_divb_source (src/ModCalcSource.f90:1694-1891)
      const double inner = 2 * h * (L1 - R0);
      acc[m].divBint = D == 0 ? inner : acc[m].divBint + inner;
      acc[m].dbf[2 * D] = h * (R0 - L0);
      acc[m].dbf[2 * D + 1] = h * (R1 - L1);
      const double vmax = fmax((double)fbuf[8 * S::NFMAX + f0], (double)fbuf[8 * S::NFMAX + f1]);
      acc[m].vdt = D == 0 ? vmax : acc[m].vdt + vmax;
    }
  }
  __syncthreads();
}

template <class S, typename Real, typename InT, typename OutT, int FLUX>
__global__ void __launch_bounds__(S::NTHREAD) stage_flat_kernel(const StageArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Real *tile = reinterpret_cast<Real *>(smem_raw);
  Real *fbuf = tile + 8 * S::NT;
  __shared__ double wmin[32];

  const int b = a.order[blockIdx.x];
  int nb[6];
#pragma unroll
  for (int q = 0; q < 6; q++) nb[q] = a.nbr[6 * b + q];
  const BlockGeom g = a.geom[b];

  gather_tile<S, Real, InT>(reinterpret_cast<const InT *>(a.in), nb, b, tile);
  __syncthreads();

  CellAcc acc[S::CPT];
  int err = 0;
  sweep<S, 0, FLUX, Real>(a, g, tile, fbuf, acc, err);
  if (S::NDIM > 1) sweep<S, 1, FLUX, Real>(a, g, tile, fbuf, acc, err);
  if (S::NDIM > 2) sweep<S, 2, FLUX, Real>(a, g, tile, fbuf, acc, err);
  if (err) atomicOr(&a.ts->errFlag, kErrHlld);

  // ---- update (update_state_normal + update_explicit) --------------------
  const StepState &ts = *a.ts;
  const double DtNoCfl = ts.DtNoCfl;
  const double DtFactor = a.useHalfStep ? (a.cfl * a.iStage) / a.nStage : a.cfl;
  const double DtLocal = DtFactor * DtNoCfl;
  const double invGm1 = a.invGm1, gm1 = a.gamma - 1.0;
  const double V = g.volume;
  double dtmin = 1e300;
  const double *__restrict__ old = a.old + (size_t)b * 8 * S::NC;
  OutT *__restrict__ out = reinterpret_cast<OutT *>(a.out) + (size_t)b * 8 * S::NC;
#pragma unroll
  for (int m = 0; m < S::CPT; m++) {
    const int c = threadIdx.x + m * S::NTHREAD;
    if (c >= S::NC) continue;
    double o[8];
#pragma unroll
    for (int v = 0; v < 8; v++) o[v] = old[v * S::NC + c];
    if (a.computeDt) dtmin = fmin(dtmin, V / acc[m].vdt);
    if (DtNoCfl == 0.0) {  // IsTimeAccurate .and. Dt == 0: state unchanged, floored
      o[kP] = limit_pressure(o[kRho], o[kP], a.fl.pMin, a.fl.tMin, a.fl.massIon);
#pragma unroll
      for (int v = 0; v < 8; v++) out[v * S::NC + c] = (OutT)o[v];
      continue;
    }
    double src[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (a.useDivb) {
      double divB = acc[m].divBint + acc[m].dbf[0] + acc[m].dbf[1];
      if (S::NDIM > 1) divB = divB + acc[m].dbf[2] + acc[m].dbf[3];
      if (S::NDIM > 2) divB = divB + acc[m].dbf[4] + acc[m].dbf[5];
      const int i = c % S::NI, j = (c / S::NI) % S::NJ, k = c / (S::NI * S::NJ);
      const int tt = S::t(i, j, k);
      const double ux = tile[kUx * S::NT + tt], uy = tile[kUy * S::NT + tt], uz = tile[kUz * S::NT + tt];
      const double bx = tile[kBx * S::NT + tt], by = tile[kBy * S::NT + tt], bz = tile[kBz * S::NT + tt];
      src[kBx] = 0 - divB * ux; src[kBy] = 0 - divB * uy; src[kBz] = 0 - divB * uz;
      src[kE] = 0 - divB * (bx * ux + by * uy + bz * uz);
      src[kUx] = 0 + (0 - divB * bx); src[kUy] = 0 + (0 - divB * by); src[kUz] = 0 + (0 - divB * bz);
    }
    double s[8];
#pragma unroll
    for (int v = 0; v < 8; v++) s[v] = DtLocal * (src[v] + acc[m].chg[v] / V);
    // pressure_to_energy(StateOld) (src/ModEnergy.f90:47)
    double e = invGm1 * o[kP] + 0.5 * (o[kUx] * o[kUx] + o[kUy] * o[kUy] + o[kUz] * o[kUz]) / o[kRho];
    e = e + 0.5 * (o[kBx] * o[kBx] + o[kBy] * o[kBy] + o[kBz] * o[kBz]);
    double n[8];
#pragma unroll
    for (int v = 0; v < 7; v++) n[v] = o[v] + s[v];
    e = e + s[kE];
    if (a.fl.rhoMin > 0.0) n[kRho] = fmax(a.fl.rhoMin, n[kRho]);  // UseRhoMin
    // energy_to_pressure (src/ModEnergy.f90:243), then limit_pressure
    double p = e - 0.5 * (n[kBx] * n[kBx] + n[kBy] * n[kBy] + n[kBz] * n[kBz]);
    n[kP] = gm1 * (p - 0.5 * (n[kUx] * n[kUx] + n[kUy] * n[kUy] + n[kUz] * n[kUz]) / n[kRho]);
    n[kP] = limit_pressure(n[kRho], n[kP], a.fl.pMin, a.fl.tMin, a.fl.massIon);
#pragma unroll
    for (int v = 0; v < 8; v++) out[v * S::NC + c] = (OutT)n[v];
  }

  if (a.computeDt) {
    // block minimum (calc_block_dt) then grid minimum (MPI_MIN of
    // set_global_timestep) via atomicMin on the ordered bits
    for (int off = 16; off > 0; off >>= 1) dtmin = fmin(dtmin, __shfl_xor_sync(0xffffffffu, dtmin, off));
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = dtmin;
    __syncthreads();
    if (threadIdx.x == 0) {
      double m = wmin[0];
      for (int w = 1; w < (int)(blockDim.x >> 5); w++) m = fmin(m, wmin[w]);
      if (a.dtBlock) store_block_dt(a.dtBlock, b, m);
      atomicMin(&a.ts->DtMinBits, dbits(m));
    }
  }
  finish_stage(a);
}
}  // namespace bx
