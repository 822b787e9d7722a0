// bx_stage_flat.cuh -- fused explicit stage kernel of 2D blocks (FP64).
//
// A CTA of one thread per face (five warps for the 144 faces of an 8 x 8
// block) works through blocks; per block:
//   1. gather: the block's cells and two ghost layers per side come straight
//      from the neighbours' interiors (float boundaries copy the boundary
//      cell), one cell per thread, loaded behind the faces of the block
//      before, into a primitive tile in shared memory;
//   2. faces: every face of both directions, one per thread, in the face's own
//      frame (flux_frame, hlld_frame; bx_physics.cuh), into the slot buffer;
//   3. cells: flux differences, Powell source, update and cell time step
//      (update_cell).
// Reference behaviour: update_state_fast (src/ModUpdateStateFast.f90:190)
// and the orig path calc_face_value -> calc_face_flux -> calc_source ->
// update_state (src/ModAdvanceExplicit.f90:140-226).
//
// What bounds it: the latency of the chain load - faces - update of a block
// with 20 warps per SM (96 registers).  384 x 384 Linde + Koren per step, two
// stages: 39.4 us; a CTA per block without the loads ahead 41.3; the kernel
// before (255 registers, two sweeps, IEEE divisions) 87.
#pragma once
#include "bx_stage_unit.cuh"

namespace bx {

template <int NI_, int NJ_>
struct Flat {
  static constexpr int NI = NI_, NJ = NJ_, NDIM = NJ > 1 ? 2 : 1, NC = NI * NJ;
  // primitive tile: interior, x ghosts [row][4], y ghosts [4][i]
  static constexpr int oX = NC, oY = oX + 4 * NJ, PT = oY + (NDIM > 1 ? 4 * NI : 0);
  // faces: x faces n < NI of all rows, then the n = NI ones; y faces
  static constexpr int F0 = (NI + 1) * NJ, F1 = NDIM > 1 ? NI * (NJ + 1) : 0, NF = F0 + F1;
  static constexpr int NTHR = (NF + 31) / 32 * 32;
  // CTAs per SM that the registers are limited for: 96 registers for a 2D block, but 128 for
  // the Roe flux (630 bytes of spills with 96)
  static constexpr int minb(int flux) { return NTHR > 96 ? (flux == kFluxRoe ? 3 : 4) : (NTHR > 32 ? 5 : 16); }
};

template <class S, int FLUX, int LIM>
__global__ void __launch_bounds__(S::NTHR, S::minb(FLUX)) stage_flat_kernel(const StageArgs a) {
  constexpr int NI = S::NI, NJ = S::NJ, NC = S::NC, PT = S::PT, NF = S::NF;
  __shared__ double P[8 * PT], fb[10 * NF], wmin[S::NTHR / 32];
  // the owned blocks come first, so a CTA's blocks need no look-up (nor does
  // the order matter: a 1D or 2D state lies in L2)
  static_assert(PT <= S::NTHR, "one cell of the tile per thread");
  const int t = threadIdx.x;
  const double *in = reinterpret_cast<const double *>(a.in);
  // the thread's cell of the tile, and the side it is a ghost cell of
  int ci = 0, cj = 0, side = -1;
  if (t < S::oX) {
    ci = t % NI; cj = t / NI;
  } else if (t < S::oY) {
    const int g = (t - S::oX) & 3;
    cj = (t - S::oX) >> 2;
    ci = g < 2 ? g - 2 : NI + g - 2;
    side = g < 2 ? 0 : 1;
  } else if (t < PT) {
    const int g = (t - S::oY) / NI;
    ci = (t - S::oY) % NI;
    cj = g < 2 ? g - 2 : NJ + g - 2;
    side = g < 2 ? 2 : 3;
  }
  // its source in the neighbour across the side, or (float boundary) the
  // boundary cell
  const int cw = min(max(ci, 0), NI - 1) + NI * min(max(cj, 0), NJ - 1);
  const int cn = (ci + NI) % NI + NI * ((cj + NJ) % NJ);
  auto neighbour = [&](int b) { return side >= 0 && b < a.nBlock ? a.nbr[6 * b + side] : b; };
  auto load = [&](int b, int nb, double (&w)[8]) {
    const double *u = in + (size_t)(nb >= 0 ? nb : b) * 8 * NC + (nb >= 0 ? cn : cw);
#pragma unroll
    for (int v = 0; v < 8; v++) w[v] = u[v * NC];
  };
  int nb = neighbour(blockIdx.x);
  grid_go();
  grid_wait();  // the neighbour table is constant; the state and the time step are the previous kernel's
  const double DtNoCfl = a.ts->DtNoCfl;
  double w[8];
  if (t < PT) load(blockIdx.x, nb, w);

  for (int b = blockIdx.x; b < a.nBlock; b += gridDim.x) {
    if (t < PT) {
      const double rhoInv = rcp_cell(w[kRho]);
      w[kUx] = rhoInv * w[kUx];
      w[kUy] = rhoInv * w[kUy];
      w[kUz] = rhoInv * w[kUz];
#pragma unroll
      for (int v = 0; v < 8; v++) P[t + v * PT] = w[v];
    }
    // the next block's neighbour now, its cells behind this block's faces
    const int bn1 = b + gridDim.x;
    nb = neighbour(bn1);
    const BlockGeom g = a.geom[b];
    __syncthreads();
    if (t < PT && bn1 < a.nBlock) load(bn1, nb, w);

    int err = 0;
    if (t < NF) {
      const int D = S::NDIM > 1 && t >= S::F0 ? 1 : 0;
      int n, in0, sIn, gh, sGh, extent;
      if (D == 0) {
        const int row = t < NI * NJ ? t / NI : t - NI * NJ;
        n = t < NI * NJ ? t % NI : NI;
        in0 = row * NI; sIn = 1;
        gh = S::oX + row * 4; sGh = 1;
        extent = NI;
      } else {
        const int f = t - S::F0;
        n = f / NI;
        in0 = f % NI; sIn = NI;
        gh = S::oY + in0; sGh = NI;
        extent = NJ;
      }
      int ad[4];
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const int c = n - 2 + m;
        ad[m] = (unsigned)c < (unsigned)extent ? in0 + c * sIn : gh + (c < 0 ? c + 2 : c - extent + 2) * sGh;
      }
      const int T1 = D + 1, T2 = D == 0 ? 2 : 0;
      const int var[8] = {0, 1 + D, 1 + T1, 1 + T2, 4 + D, 4 + T1, 4 + T2, 7};
      double L[8], R[8];
      if (a.nOrder == 1) {
#pragma unroll
        for (int v = 0; v < 8; v++) { L[v] = P[ad[1] + var[v] * PT]; R[v] = P[ad[2] + var[v] * PT]; }
      } else {
#pragma unroll
        for (int v = 0; v < 8; v++)
          limited_face_t<LIM>(a.beta, P[ad[0] + var[v] * PT], P[ad[1] + var[v] * PT], P[ad[2] + var[v] * PT],
                              P[ad[3] + var[v] * PT], L[v], R[v]);
      }
      double cbL = 0, cbR = 0, cuL = 0, cuR = 0, bn;
      if (FLUX == kFluxRoe) {
        cbL = P[ad[1] + var[4] * PT]; cbR = P[ad[2] + var[4] * PT];
        cuL = P[ad[1] + var[1] * PT]; cuR = P[ad[2] + var[1] * PT];
      }
      bool ok = true;
      const double vdt = unit_flux<FLUX, double>(D, L, R, a.gamma, a.invGm1, D == 0 ? g.area[0] : g.area[1], cbL, cbR, cuL, cuR, bn, ok,
                                                 [&](int q, double x) { fb[var[q] * NF + t] = x; });
      fb[8 * NF + t] = vdt;
      fb[9 * NF + t] = bn;
      if (!ok) err = 1;
    }
    if (err) atomicOr(&a.ts->errFlag, kErrHlld);
    __syncthreads();

    double dtmin = 1e300;
    if (t < NC) {
      double o[8];
#pragma unroll
      for (int v = 0; v < 8; v++) o[v] = a.old[(size_t)b * 8 * NC + v * NC + t];
      const int i = t % NI, j = t / NI;
      double chg[8], divB = 0.0, vsum = 0.0, ub[6];
#pragma unroll
      for (int D = 0; D < S::NDIM; D++) {
        const int f0 = D == 0 ? t : S::F0 + t, f1 = D == 0 ? (i + 1 < NI ? t + 1 : NC + j) : f0 + NI;
#pragma unroll
        for (int v = 0; v < 8; v++) {
          const double d = fb[v * NF + f0] - fb[v * NF + f1];
          chg[v] = D == 0 ? d : chg[v] + d;
        }
        const double e = mul_rn(g.invHalf[D], fb[9 * NF + f1] - fb[9 * NF + f0]);
        divB = D == 0 ? e : divB + e;
        const double x = fmax(fb[8 * NF + f0], fb[8 * NF + f1]);
        vsum = D == 0 ? x : vsum + x;
      }
#pragma unroll
      for (int q = 0; q < 6; q++) ub[q] = P[t + (kUx + q) * PT];
      if (a.computeDt) dtmin = g.volume / vsum;
      double *out = reinterpret_cast<double *>(a.out) + (size_t)b * 8 * NC + t;
      update_cell<double>(a, DtNoCfl, g.invVolume, chg, divB, ub, o, out, NC);
    }
    if (a.computeDt) {
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
    __syncthreads();  // P and the slots are read
  }
  finish_stage(a);
}

}  // namespace bx
