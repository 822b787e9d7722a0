// bx_stage_line.cuh -- fused explicit stage kernel of 1D blocks (FP64).
//
// One CTA per block, one thread per face, launched as a programmatic
// dependent of the kernel before it; the last stage's last CTA ends the time
// step (finish_stage).  The arithmetic is the reference's, operation by
// operation (numerical_flux, IEEE divisions and square roots, no contraction:
// the file is compiled with --fmad=false): a shock tube of hundreds of steps
// at second order amplifies the rounding of a step a thousandfold, so
// another order of operations gives other digits (4e-13 of the norm), and a
// 1D step's time is the latency of its launches, not its arithmetic.
#pragma once
#include "bx_stage3d.cuh"

namespace bx {

template <int NI_>
struct Line {
  static constexpr int NI = NI_, PT = NI + 4, NF = NI + 1, NTHR = (PT + 31) / 32 * 32;  // tile cells -2 .. NI + 1
  static constexpr int MINB = NTHR > 32 ? 5 : 16;
};

template <class S, int FLUX, int LIM>
__global__ void __launch_bounds__(S::NTHR, S::MINB) stage_line_kernel(const StageArgs a) {
  constexpr int NI = S::NI, PT = S::PT, NF = S::NF;
  __shared__ double P[8 * PT], fb[11 * NF], wmin[S::NTHR / 32];
  __shared__ StepState step;
  const int t = threadIdx.x, b = blockIdx.x;  // the owned blocks come first
  const int nb0 = a.nbr[6 * b], nb1 = a.nbr[6 * b + 1];
  const BlockGeom g = a.geom[b];
  grid_go();
  grid_wait();  // the tables above are constant; the state and the time step are the previous kernel's
  const double DtNoCfl = a.ts->DtNoCfl;
  if (t < PT) {
    // the cell, or a ghost cell's source (float boundary: the boundary cell)
    int i = t - 2, src = b;
    if (i < 0) {
      if (nb0 >= 0) { src = nb0; i += NI; } else i = 0;
    } else if (i >= NI) {
      if (nb1 >= 0) { src = nb1; i -= NI; } else i = NI - 1;
    }
    const double *u = reinterpret_cast<const double *>(a.in) + (size_t)src * 8 * NI + i;
    double w[8];
#pragma unroll
    for (int v = 0; v < 8; v++) w[v] = u[v * NI];
    // calc_primitives (src/ModFaceValue.f90:1530-1621): u = (1/rho) rhoU
    const double rhoInv = 1.0 / w[kRho];
    w[kUx] = rhoInv * w[kUx]; w[kUy] = rhoInv * w[kUy]; w[kUz] = rhoInv * w[kUz];
#pragma unroll
    for (int v = 0; v < 8; v++) P[v * PT + t] = w[v];
  }
  double o[8];
  if (t < NI) {
#pragma unroll
    for (int v = 0; v < 8; v++) o[v] = a.old[(size_t)b * 8 * NI + v * NI + t];
  }
  load_step(a, step);
  __syncthreads();

  if (t < NF) {
    double L[8], R[8], F[8], vdt;
#pragma unroll
    for (int v = 0; v < 8; v++) {
      const double *q = P + v * PT + t;  // cells t - 2 .. t + 1
      if (a.nOrder == 1) { L[v] = q[1]; R[v] = q[2]; }
      else limited_face_t<LIM>(a.beta, q[0], q[1], q[2], q[3], L[v], R[v]);
    }
    if (FLUX == kFluxRoe) {
      // UseRS7 (src/ModFaceFlux.f90:600-625): each face state takes the
      // normal field of its cell before the div B slots are formed
      const double cbL = P[kBx * PT + t + 1], cbR = P[kBx * PT + t + 2];
      const double dBnR = R[kBx] - cbR;
      R[kBx] = R[kBx] - dBnR;
      const double dBnL = L[kBx] - cbL;
      L[kBx] = L[kBx] - dBnL;
      fb[9 * NF + t] = L[kBx];
      fb[10 * NF + t] = R[kBx];
      vdt = roe_flux<0>(L, R, P[kUx * PT + t + 1], P[kUx * PT + t + 2], dBnL, dBnR, a.gamma, a.invGm1, g.area[0], F, 1);
    } else {
      fb[9 * NF + t] = L[kBx];
      fb[10 * NF + t] = R[kBx];
      if (!numerical_flux<0, FLUX>(L, R, a.gamma, a.invGm1, g.area[0], F, vdt)) atomicOr(&a.ts->errFlag, kErrHlld);
    }
#pragma unroll
    for (int v = 0; v < 8; v++) fb[v * NF + t] = F[v];
    fb[8 * NF + t] = vdt;
  }
  __syncthreads();

  double dtmin = 1e300;
  if (t < NI) {
    const double V = g.volume;
    double *out = reinterpret_cast<double *>(a.out) + (size_t)b * 8 * NI + t;
    if (a.computeDt) dtmin = V / fmax(fb[8 * NF + t], fb[8 * NF + t + 1]);
    if (DtNoCfl == 0.0) {  // IsTimeAccurate .and. Dt == 0: state unchanged, floored
      o[kP] = limit_pressure(o[kRho], o[kP], a.fl.pMin, a.fl.tMin, a.fl.massIon);
#pragma unroll
      for (int v = 0; v < 8; v++) out[v * NI] = o[v];
    } else {
      const double DtLocal = a.dtFactor * DtNoCfl;
      double src[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      if (a.useDivb) {
        // calc_divb_source (src/ModCalcSource.f90:1694-1891)
        const double h = g.invHalf[0];
        const double L0 = fb[9 * NF + t], R0 = fb[10 * NF + t], L1 = fb[9 * NF + t + 1], R1 = fb[10 * NF + t + 1];
        const double divB = 2 * h * (L1 - R0) + h * (R0 - L0) + h * (R1 - L1);
        const double *q = P + t + 2;
        const double ux = q[kUx * PT], uy = q[kUy * PT], uz = q[kUz * PT];
        const double bx = q[kBx * PT], by = q[kBy * PT], bz = q[kBz * PT];
        src[kBx] = 0 - divB * ux; src[kBy] = 0 - divB * uy; src[kBz] = 0 - divB * uz;
        src[kE] = 0 - divB * (bx * ux + by * uy + bz * uz);
        src[kUx] = 0 + (0 - divB * bx); src[kUy] = 0 + (0 - divB * by); src[kUz] = 0 + (0 - divB * bz);
      }
      double s[8];
#pragma unroll
      for (int v = 0; v < 8; v++) s[v] = DtLocal * (src[v] + (fb[v * NF + t] - fb[v * NF + t + 1]) / V);
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
      for (int v = 0; v < 8; v++) out[v * NI] = n[v];
    }
  }
  if (a.computeDt) {
    // block minimum (calc_block_dt), then the grid minimum by atomicMin on
    // the ordered bits
    for (int off = 16; off > 0; off >>= 1) dtmin = fmin(dtmin, __shfl_xor_sync(0xffffffffu, dtmin, off));
    if ((t & 31) == 0) wmin[t >> 5] = dtmin;
    __syncthreads();
    if (t == 0) {
      double m = wmin[0];
      for (int w = 1; w < S::NTHR / 32; w++) m = fmin(m, wmin[w]);
      if (a.dtBlock) store_block_dt(a.dtBlock, b, m);
      atomicMin(&a.ts->DtMinBits, (unsigned long long)__double_as_longlong(m));
    }
  }
  finish_stage(a, step);
}

}  // namespace bx
