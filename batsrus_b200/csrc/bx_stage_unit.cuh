// bx_stage_unit.cuh -- fused explicit stage kernel of 3D blocks, in work units
// of 128 cells.
//
// Same arithmetic as stage3d_kernel (bx_stage3d.cuh): calc_primitives, the
// limited reconstruction (ModFaceValue), the face fluxes (ModFaceFlux), the
// Powell source (ModCalcSource), the conservative update with p <-> E and
// the floors (ModUpdateState, ModEnergy) and the cell time step
// (ModTimeStepControl).
//
// A unit is an 8 x 4 x 4 quarter of an 8^3 block or two 4^3 blocks; a CTA of
// five warps works through units, several CTAs per SM.  Per unit:
//  * the state lands in shared memory by TMA (the interior box and six
//    2-layer halo boxes of each tile; the halo of a quarter's inner side
//    comes from the same block), one unit ahead;
//  * the conversion pass writes the primitive tile P: the interior rows, then
//    the x, y and z ghost cells, each with unit stride along x, so that a
//    half warp's 16 FP64 cells (two rows of 8, four of 4) never share a bank;
//  * 15 groups of 32 faces, three per warp, compute the face fluxes into the
//    slot buffer R.  A group has one direction; the state is read in the
//    face's frame n, t1, t2 (flux_frame, flux_pair, hlld_frame);
//  * each thread updates one cell.
// The landing area of the next unit overlays R, behind P.
//
// What bounds it: instruction issue.  96^3 Linde + Koren under ncu: FP64 3150
// instructions per cell and stage, 1440 of them FP64 (two cycles each), issue
// 53 %, FP64 pipe 44 % of the cycles with 15 warps per SM; FP32-bulk 2220
// instructions, issue 65 %.  Against one CTA per SM and whole blocks
// (bx_stage3d_v2.cuh): 160^3 per step FP64 Linde 1694 -> 1238 us, HLLD (128^3)
// 943 -> 690 us, FP32-bulk Linde 789 -> 756 us; 16^3 (8 blocks, now 32 units)
// 41 -> 21 us; 96^3 cells / 8 in blocks of 4^3 125 -> 57 us.  With resolution
// changes: see stage3d_units (bx_stage3d.cu).
#pragma once
#include "bx_stage3d.cuh"

namespace bx {

template <int N_, typename TileT, typename Real, int MINB_>
struct Unit {
  static constexpr int N = N_, U = 4;                  // block size; tile N x 4 x 4
  static constexpr int TC = N * 16, NT = 128 / TC;     // cells per tile, tiles per unit
  static constexpr int PARTS = N == 8 ? 4 : 1;         // units per block
  static constexpr int NTHR = 160, NW = 5, MINB = MINB_;
  // primitive tile: interior, x ghosts [row][4], y ghosts [k][4][i], z ghosts [4][j][i]
  static constexpr int oX = TC, oY = oX + 64, oZ = oY + 16 * N, PT = oZ + 16 * N;
  static constexpr int PV = NT * PT;                   // cells per variable
  static constexpr int CCV = (PV + NTHR - 1) / NTHR;   // conversion cells per thread
  // faces per tile and direction, and in all; x faces n < N of all rows
  // first, then the n = N face of every row
  static constexpr int F0 = (N + 1) * 16, F1 = N * 20, F2 = N * 20;
  static constexpr int B1 = NT * F0, B2 = B1 + NT * F1, NF = B2 + NT * F2;
  static constexpr int GPD = 5;                        // groups of 32 faces per direction
  static_assert(NT * F0 <= 32 * GPD && NT * F1 <= 32 * GPD, "face groups");
  static constexpr int NSLOT = 10;                     // 8 fluxes, Vdt, BnL + BnR
  // landing area per tile
  static constexpr int HX = 16 / (int)sizeof(TileT);
  static constexpr int nIN = 8 * TC, nX = 8 * 16 * HX, nY = 8 * 4 * 2 * N, nZ = nY;
  static constexpr int oXL = nIN, oXH = oXL + nX, oYL = oXH + nX, oYH = oYL + nY, oZL = oYH + nY, oZH = oZL + nZ,
                       nAll = oZH + nZ;
  static constexpr size_t primBytes = sizeof(Real) * 8 * PV, fluxBytes = sizeof(Real) * NSLOT * NF,
                          stageBytes = sizeof(TileT) * (size_t)NT * nAll;
  static constexpr size_t smem_bytes = primBytes + (fluxBytes > stageBytes ? fluxBytes : stageBytes);
};

// what a tile needs before it is converted, loaded one unit ahead
struct UnitMeta {
  int b, part, j0, k0;      // block, and the tile's place in it
  int rcFine, rcCoarse;     // sides of the block next to a coarser / finer block
  int nb[6];                // neighbour of each side of the block
  int src[6];               // block that a side's halo comes from (the block itself at an inner side), or < 0
  int rcSlab[6];
  BlockGeom g;
};

template <class W>
__device__ __forceinline__ void load_unit_meta(const StageArgs &a, int unit, int p, UnitMeta &m) {
  const int q = W::N == 8 ? unit >> 2 : min(unit * W::NT + p, a.nBlock - 1);
  const int b = a.order[q], part = W::N == 8 ? unit & 3 : 0;
  m.b = b;
  m.part = part;
  m.j0 = 4 * (part & 1);
  m.k0 = 4 * (part >> 1);
  int fine = 0, coarse = 0;
#pragma unroll
  for (int s = 0; s < 6; s++) {
    const int nb = a.nbr[6 * b + s];
    const bool inner = (s == 2 && m.j0 > 0) || (s == 3 && m.j0 + 4 < W::N) || (s == 4 && m.k0 > 0) ||
                       (s == 5 && m.k0 + 4 < W::N);
    m.nb[s] = nb;
    m.src[s] = inner ? b : nb;
    int slab = 0;
    if (nb == kNbrResChange) {
      const int rt = a.rcType[6 * b + s];
      slab = a.rcSlab[6 * b + s];
      if (rt == 1) fine |= 1 << s;
      if (rt == -1) coarse |= 1 << s;
    }
    m.rcSlab[s] = slab;
  }
  m.rcFine = fine;
  m.rcCoarse = coarse;
  m.g = a.geom[b];
}

// TMA loads of the unit's tiles into buf.  Every box starts at an x that is a
// multiple of 16 bytes: 0, or N - HX
template <class W, typename TileT>
__device__ __forceinline__ void issue_unit(const TmaMaps &maps, TileT *buf, uint64_t *bar, const UnitMeta *m) {
  constexpr int N = W::N;
  uint32_t elems = 0;
#pragma unroll
  for (int p = 0; p < W::NT; p++) {
    elems += W::nIN;
#pragma unroll
    for (int s = 0; s < 6; s++)
      if (m[p].src[s] >= 0) elems += s < 2 ? W::nX : W::nY;
  }
  mbar_arrive_expect_tx(bar, elems * (uint32_t)sizeof(TileT));
#pragma unroll 1
  for (int p = 0; p < W::NT; p++) {
    const UnitMeta &q = m[p];
    TileT *d = buf + p * W::nAll;
    const int j = q.j0, k = q.k0;
    tma_load_5d(d, &maps.uin, bar, 0, j, k, 0, q.b);
    if (q.src[0] >= 0) tma_load_5d(d + W::oXL, &maps.uxh, bar, N - W::HX, j, k, 0, q.src[0]);
    if (q.src[1] >= 0) tma_load_5d(d + W::oXH, &maps.uxh, bar, 0, j, k, 0, q.src[1]);
    if (q.src[2] >= 0) tma_load_5d(d + W::oYL, &maps.uyh, bar, 0, (j + N - 2) % N, k, 0, q.src[2]);
    if (q.src[3] >= 0) tma_load_5d(d + W::oYH, &maps.uyh, bar, 0, (j + 4) % N, k, 0, q.src[3]);
    if (q.src[4] >= 0) tma_load_5d(d + W::oZL, &maps.uzh, bar, 0, j, (k + N - 2) % N, 0, q.src[4]);
    if (q.src[5] >= 0) tma_load_5d(d + W::oZH, &maps.uzh, bar, 0, j, (k + 4) % N, 0, q.src[5]);
  }
}

// cell c (0 .. PT - 1) of a primitive tile: tile coordinates and the side it
// is a ghost cell of (-1: interior)
template <class W>
__device__ __forceinline__ void unit_cell(int c, int &i, int &j, int &k, int &side) {
  constexpr int N = W::N;
  if (c < W::oX) {
    i = c % N; j = (c / N) & 3; k = c / (4 * N); side = -1;
  } else if (c < W::oY) {
    c -= W::oX;
    const int g = c & 3;
    i = g < 2 ? g - 2 : N + g - 2; j = (c >> 2) & 3; k = c >> 4; side = g < 2 ? 0 : 1;
  } else if (c < W::oZ) {
    c -= W::oY;
    const int g = (c / N) & 3;
    i = c % N; j = g < 2 ? g - 2 : g + 2; k = c / (4 * N); side = g < 2 ? 2 : 3;
  } else {
    c -= W::oZ;
    const int g = c / (4 * N);
    i = c % N; j = (c / N) & 3; k = g < 2 ? g - 2 : g + 2; side = g < 2 ? 4 : 5;
  }
}

// landing-area element of variable 0 of tile cell (i, j, k) and its variable
// stride (at most one coordinate outside the tile, by at most 2)
template <class W>
__device__ __forceinline__ int landing(int i, int j, int k, int &vs) {
  constexpr int N = W::N, HX = W::HX;
  if (i < 0) { vs = 16 * HX; return W::oXL + (4 * k + j) * HX + HX + i; }
  if (i >= N) { vs = 16 * HX; return W::oXH + (4 * k + j) * HX + i - N; }
  vs = 8 * N;
  if (j < 0) return W::oYL + (2 * k + j + 2) * N + i;
  if (j >= 4) return W::oYH + (2 * k + j - 4) * N + i;
  if (k < 0) return W::oZL + (4 * (k + 2) + j) * N + i;
  if (k >= 4) return W::oZH + (4 * (k - 4) + j) * N + i;
  vs = W::TC;
  return (4 * k + j) * N + i;
}

// primitive tile index of tile cell (i, j, k) (at most one outside)
template <class W>
__device__ __forceinline__ int prim_at(int i, int j, int k) {
  constexpr int N = W::N;
  if (i < 0) return W::oX + (4 * k + j) * 4 + i + 2;
  if (i >= N) return W::oX + (4 * k + j) * 4 + i - N + 2;
  if (j < 0) return W::oY + (4 * k + j + 2) * N + i;
  if (j >= 4) return W::oY + (4 * k + j - 2) * N + i;
  if (k < 0) return W::oZ + (4 * (k + 2) + j) * N + i;
  if (k >= 4) return W::oZ + (4 * (k - 2) + j) * N + i;
  return (4 * k + j) * N + i;
}

// the two face indices (slot buffer, within the tile's faces of direction D)
// of tile cell (i, row = j + 4 k)
template <class W>
__device__ __forceinline__ void cell_faces(int D, int i, int j, int k, int &f0, int &f1) {
  constexpr int N = W::N;
  if (D == 0) {
    const int row = j + 4 * k;
    f0 = row * N + i;
    f1 = i + 1 < N ? f0 + 1 : 16 * N + row;
  } else if (D == 1) {
    f0 = i + N * (j + 5 * k);
    f1 = f0 + N;
  } else {
    f0 = i + N * (j + 4 * k);
    f1 = f0 + 4 * N;
  }
}

// 1/rho of the conversion: branch-free in double; in float the IEEE quotient
__device__ __forceinline__ double rcp_cell(double x) { return rcp_nb(x); }
__device__ __forceinline__ float rcp_cell(float x) { return 1.0f / x; }

// a product that is not contracted into a sum: the three terms of div B
// cancel, and one rounded product less leaves a spurious remainder
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }

// the fluxes of one face from its states in the face's frame, through
// out(q, flux) (frame order); returns Vdt
template <int FLUX, typename Real, class Out>
__device__ __forceinline__ Real unit_flux(int D, Real (&L)[8], Real (&R)[8], Real gamma, Real invGm1, Real area,
                                          Real cbL, Real cbR, Real cuL, Real cuR, Real &bnSum, bool &ok,
                                          const Out &out) {
  if constexpr (FLUX == kFluxRoe) {
    // RS7 (src/ModFaceFlux.f90:600-625): see face_slots
    const Real dR = R[4] - cbR, dL = L[4] - cbL;
    R[4] = R[4] - dR;
    L[4] = L[4] - dL;
    bnSum = L[4] + R[4];
    // roe_flux keeps the axis order (its degenerate tangents depend on it)
    auto axes = [&](auto d) {
      constexpr int A = decltype(d)::value, T1 = (A + 1) % 3, T2 = (A + 2) % 3;
      Real l[8], r[8], F[8];
      constexpr int var[8] = {0, 1 + A, 1 + T1, 1 + T2, 4 + A, 4 + T1, 4 + T2, 7};
#pragma unroll
      for (int q = 0; q < 8; q++) { l[var[q]] = L[q]; r[var[q]] = R[q]; }
      const Real v = roe_flux<A>(l, r, cuL, cuR, dL, dR, gamma, invGm1, area, F, 1);
#pragma unroll
      for (int q = 0; q < 8; q++) out(q, F[var[q]]);
      return v;
    };
    if (D == 0) return axes(std::integral_constant<int, 0>{});
    if (D == 1) return axes(std::integral_constant<int, 1>{});
    return axes(std::integral_constant<int, 2>{});
  } else {
    bnSum = L[4] + R[4];
    if constexpr (FLUX == kFluxHlld) {
      Real v;
      ok = hlld_frame(L, R, gamma, invGm1, area, v, out);
      return v;
    } else {
      if constexpr (sizeof(Real) == sizeof(float)) {
        F2 X[8];
#pragma unroll
        for (int q = 0; q < 8; q++) X[q] = f2(L[q], R[q]);
        return flux_pair<FLUX>(X, gamma, invGm1, area, out);
      } else {
        return flux_frame<FLUX, Real>(L, R, gamma, invGm1, area, out);
      }
    }
  }
}

// update_state_normal / update_explicit of one cell: o the step's first
// state, chg the flux sums, ub velocity and field for the Powell source;
// writes out[v * stride]
template <typename OutT>
__device__ __forceinline__ void update_cell(const StageArgs &a, double DtNoCfl, double invV, const double (&chg)[8],
                                            double divB, const double (&ub)[6], double (&o)[8], OutT *out,
                                            int stride) {
  if (DtNoCfl == 0.0) {
    // update_state with Dt = 0: the state is unchanged, then
    // limit_pressure (src/ModUpdateState.f90:169, 241)
    o[kP] = limit_pressure(o[kRho], o[kP], a.fl.pMin, a.fl.tMin, a.fl.massIon);
#pragma unroll
    for (int v = 0; v < 8; v++) out[v * stride] = (OutT)o[v];
    return;
  }
  const double DtLocal = a.dtFactor * DtNoCfl;
  double src[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (a.useDivb) {
    const double ux = ub[0], uy = ub[1], uz = ub[2], bx = ub[3], by = ub[4], bz = ub[5];
    src[kBx] = -divB * ux; src[kBy] = -divB * uy; src[kBz] = -divB * uz;
    src[kE] = -divB * (bx * ux + by * uy + bz * uz);
    src[kUx] = -divB * bx; src[kUy] = -divB * by; src[kUz] = -divB * bz;
  }
  double e = a.invGm1 * o[kP] + div_nb(0.5 * (o[kUx] * o[kUx] + o[kUy] * o[kUy] + o[kUz] * o[kUz]), o[kRho]);
  e = e + 0.5 * (o[kBx] * o[kBx] + o[kBy] * o[kBy] + o[kBz] * o[kBz]);
  double n[8];
#pragma unroll
  for (int v = 0; v < 7; v++) n[v] = o[v] + DtLocal * (src[v] + chg[v] * invV);
  e = e + DtLocal * (src[kE] + chg[kE] * invV);
  if (a.fl.rhoMin > 0.0) n[kRho] = fmax(a.fl.rhoMin, n[kRho]);  // UseRhoMin
  const double pe = e - 0.5 * (n[kBx] * n[kBx] + n[kBy] * n[kBy] + n[kBz] * n[kBz]);
  n[kP] = (a.gamma - 1.0) * (pe - div_nb(0.5 * (n[kUx] * n[kUx] + n[kUy] * n[kUy] + n[kUz] * n[kUz]), n[kRho]));
  n[kP] = limit_pressure(n[kRho], n[kP], a.fl.pMin, a.fl.tMin, a.fl.massIon);
#pragma unroll
  for (int v = 0; v < 8; v++) out[v * stride] = (OutT)n[v];
}

// RC = false: the launch's grid has no resolution change and no sharper
// limiter at a float boundary (StageArgs::anySpecial = 0)
template <class W, typename TileT, typename Real, typename OutT, int FLUX, int LIM, bool RC>
__global__ void __launch_bounds__(W::NTHR, W::MINB)
    stage_unit_kernel(const __grid_constant__ TmaMaps maps, const StageArgs a) {
  constexpr int N = W::N, NT = W::NT, PV = W::PV, PT = W::PT;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Real *P = reinterpret_cast<Real *>(smem_raw);
  Real *fb = reinterpret_cast<Real *>(smem_raw + W::primBytes);
  TileT *stg = reinterpret_cast<TileT *>(smem_raw + W::primBytes);
  __shared__ uint64_t bar;
  __shared__ double wmin[4];
  __shared__ UnitMeta meta[2][NT];
  __shared__ int sTimeout;
  __shared__ StepState step;
  const int t = threadIdx.x, lane = t & 31, warp = __shfl_sync(0xffffffffu, t >> 5, 0);
  const int nUnit = N == 8 ? 4 * a.nBlock : (a.nBlock + NT - 1) / NT;
  const int nIter = nUnit > (int)blockIdx.x ? (nUnit - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  if (t == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    sTimeout = 0;
  }
  if (t < NT && nIter > 0) load_unit_meta<W>(a, blockIdx.x, t, meta[0][t]);
  __syncthreads();
  if (t == 0 && nIter > 0) issue_unit<W, TileT>(maps, stg, &bar, meta[0]);

  const double DtNoCfl = a.ts->DtNoCfl;
  load_step(a, step);
  const Real beta = (Real)a.beta, gammaR = (Real)a.gamma, invGm1R = (Real)a.invGm1;
  int err = 0;
  double dtRun = 1e300;  // thread 0: the smallest cell time step of this CTA's units

  for (int it = 0; it < nIter; it++) {
    const UnitMeta *M = meta[it & 1];
    if (!mbar_wait_bounded(&bar, (uint32_t)(it & 1))) sTimeout = 1;
    __syncthreads();  // (A) the unit's state has landed
    if (sTimeout) break;  // uniform: every thread read the flag after the barrier

    // ---- calc_primitives: landing area (conservative) -> P (primitive) ---
#pragma unroll
    for (int q = 0; q < W::CCV; q++) {
      const int cq = t + q * W::NTHR;
      if (cq >= PV) continue;
      const int p = NT > 1 ? cq / PT : 0;
      const UnitMeta &m = M[p];
      int i, j, k, side;
      unit_cell<W>(cq - p * PT, i, j, k, side);
      TileT w[8];
      const int src = side >= 0 ? m.src[side] : 0;
      if (RC && src == kNbrResChange) {
        // ghost layers of a resolution-change side: its slab
        // [var][layer][t1][t0] (injection / restriction, bx_amr.cu)
        const int d = side >> 1, hi = side & 1;
        const int bi = i, bj = j + m.j0, bk = k + m.k0;
        const int cd = d == 0 ? bi : (d == 1 ? bj : bk);
        const int l = hi ? cd - N : -1 - cd;
        const int t0 = d == 0 ? bj : bi, t1 = d == 2 ? bj : bk;
        const double *s = a.rcGhost + (size_t)m.rcSlab[side] * (16 * N * N) + (l * N + t1) * N + t0;
#pragma unroll
        for (int v = 0; v < 8; v++) w[v] = (TileT)s[v * 2 * N * N];
      } else {
        if (src < 0) {  // float boundary: copy of the boundary cell
          i = min(max(i, 0), N - 1);
          j = min(max(j, 0), 3);
          k = min(max(k, 0), 3);
        }
        int vs;
        const TileT *s = stg + p * W::nAll + landing<W>(i, j, k, vs);
#pragma unroll
        for (int v = 0; v < 8; v++) w[v] = s[v * vs];
      }
      const TileT rhoInv = rcp_cell(w[kRho]);
      w[kUx] = rhoInv * w[kUx];
      w[kUy] = rhoInv * w[kUy];
      w[kUz] = rhoInv * w[kUz];
#pragma unroll
      for (int v = 0; v < 8; v++) P[cq + v * PV] = (Real)w[v];
    }
    __syncthreads();  // (B) P is complete; the landing area becomes the slot buffer

    // the last warp loads the next unit's neighbours and geometry meanwhile
    if (t >= W::NTHR - NT && it + 1 < nIter)
      load_unit_meta<W>(a, blockIdx.x + (it + 1) * gridDim.x, t - (W::NTHR - NT), meta[(it + 1) & 1][t - (W::NTHR - NT)]);

    // ---- all faces of the unit: 15 groups of 32 ---------------------------
    auto face = [&](auto D, int gg) {
      const int ft = gg * 32 + lane;
      const int nfD = D == 0 ? W::F0 : W::F1;
      if (ft >= NT * nfD) return;
      const int p = NT > 1 ? ft / nfD : 0;
      const int f = ft - p * nfD;
      // the face's index n along D (its right cell) and transverse cell;
      // interior cells at in + m sIn, ghost cells of this direction at
      // gh + m sGh (m = 0..3, cells n - 2 .. n + 1)
      int n, u0, u1, in, sIn, gh, sGh, extent;
      if (D == 0) {
        const int row = f < 16 * N ? f / N : f - 16 * N;
        n = f < 16 * N ? f % N : N;
        u0 = row & 3; u1 = row >> 2;
        in = row * N; sIn = 1;
        gh = W::oX + row * 4; sGh = 1;
        extent = N;
      } else if (D == 1) {
        const int r = f / N;  // n + 5 k
        u0 = f % N; u1 = r / 5; n = r - 5 * u1;
        in = 4 * N * u1 + u0; sIn = N;
        gh = W::oY + in; sGh = N;
        extent = 4;
      } else {
        const int r = f / N;  // j + 4 n
        u0 = f % N; u1 = r & 3; n = r >> 2;
        in = N * u1 + u0; sIn = 4 * N;
        gh = W::oZ + in; sGh = 4 * N;
        extent = 4;
      }
      const int p0 = p * PT;  // the tile's cells in P
      int ad[4];
#pragma unroll
      for (int m = 0; m < 4; m++) {
        const int c = n - 2 + m;
        ad[m] = p0 + ((unsigned)c < (unsigned)extent ? in + c * sIn : gh + (c < 0 ? c + 2 : c - extent + 2) * sGh);
      }
      const UnitMeta &mt = M[p];
      const int nb0 = D == 0 ? n : n + (D == 1 ? mt.j0 : mt.k0);  // face index in the block
      const int side = nb0 == 0 ? 2 * D : (nb0 == N ? 2 * D + 1 : -1);
      const bool first = a.nOrder == 1 || (RC && !a.tvdRc && side >= 0 && ((mt.rcFine >> side) & 1));
      // the face states, the variables in the frame's order
      const int T1 = D == 2 ? 0 : D + 1, T2 = D == 0 ? 2 : D - 1;
      const int var[8] = {0, 1 + D, 1 + T1, 1 + T2, 4 + D, 4 + T1, 4 + T2, 7};
      Real L[8], R[8];
      if (first) {
#pragma unroll
        for (int v = 0; v < 8; v++) {
          L[v] = P[ad[1] + var[v] * PV];
          R[v] = P[ad[2] + var[v] * PV];
        }
      } else {
#pragma unroll
        for (int v = 0; v < 8; v++) {
          const Real *q = P + var[v] * PV;
          if constexpr (sizeof(Real) == sizeof(float))
            f2_get(limited_pair<LIM>(beta, q[ad[0]], q[ad[1]], q[ad[2]], q[ad[3]]), L[v], R[v]);
          else limited_face_t<LIM>(beta, q[ad[0]], q[ad[1]], q[ad[2]], q[ad[3]], L[v], R[v]);
        }
      }
      Real cbL = Real(0), cbR = Real(0), cuL = Real(0), cuR = Real(0);
      if (FLUX == kFluxRoe) {  // the cell values next to the face
        cbL = P[ad[1] + var[4] * PV]; cbR = P[ad[2] + var[4] * PV];
        cuL = P[ad[1] + var[1] * PV]; cuR = P[ad[2] + var[1] * PV];
      }
      if (RC) {
        const bool sharp = a.nOrder > 1 && a.betaRc < a.beta;
        const int lo = mt.nb[2 * D], hi = mt.nb[2 * D + 1];
        if ((sharp && (lo < 0 || hi < 0)) || (a.tvdRc && ((mt.rcFine >> (2 * D)) & 3))) {
          auto special = [&](auto d) {
            constexpr int A = decltype(d)::value;
            constexpr int vs[8] = {0, 1 + A, 1 + (A + 1) % 3, 1 + (A + 2) % 3,
                                   4 + A, 4 + (A + 1) % 3, 4 + (A + 2) % 3, 7};
            const int j0 = mt.j0, k0 = mt.k0;
            // transverse cells in block coordinates, lower dimension first
            const int t0 = A == 0 ? u0 + j0 : u0, t1 = A == 0 ? u1 + k0 : (A == 1 ? u1 + k0 : u1 + j0);
            reschange_face_states<N, A, LIM, Real>(a, nb0, t0, t1, lo, hi, mt.rcFine, first, L, R,
                                                   [&](int v, int ci, int cj, int ck) {
                                                     return P[vs[v] * PV + p0 + prim_at<W>(ci, cj - j0, ck - k0)];
                                                   });
          };
          if (D == 0) special(std::integral_constant<int, 0>{});
          else if (D == 1) special(std::integral_constant<int, 1>{});
          else special(std::integral_constant<int, 2>{});
        }
      }
      Real *o = fb + (D == 0 ? 0 : (D == 1 ? W::B1 : W::B2)) + ft;
      bool ok = true;
      Real bn;
      const Real vdt = unit_flux<FLUX, Real>(D, L, R, gammaR, invGm1R, (Real)mt.g.area[D], cbL, cbR, cuL, cuR, bn, ok,
                                             [&](int q, Real x) { o[var[q] * W::NF] = x; });
      o[8 * W::NF] = vdt;
      o[9 * W::NF] = bn;
      if (!ok) err = 1;
      if (RC && side >= 0 && ((mt.rcCoarse >> side) & 1)) {
        // apply_cons_flux: the summed fluxes of the finer faces
        const int t0 = D == 0 ? u0 + mt.j0 : u0, t1 = D == 2 ? u1 + mt.j0 : u1 + mt.k0;
        const double *cf = a.rcFlux + ((size_t)mt.rcSlab[side] * N * N + t0 + N * t1) * kRcSlots;
#pragma unroll
        for (int q = 0; q < kRcSlots; q++) o[q * W::NF] = (Real)cf[q];
      }
    };
#pragma unroll 1
    for (int gi = warp; gi < 3 * W::GPD; gi += W::NW) {
      // one copy of the short fluxes per direction (constant offsets: 1286
      // against 1320 us per step, 160^3 FP64 Linde); one for all three
      // directions of the long ones (320 against 351 us, 96^3 FP64 HLLD)
      if constexpr (FLUX != kFluxHlld) {
        if (gi < W::GPD) face(std::integral_constant<int, 0>{}, gi);
        else if (gi < 2 * W::GPD) face(std::integral_constant<int, 1>{}, gi - W::GPD);
        else face(std::integral_constant<int, 2>{}, gi - 2 * W::GPD);
      } else {
        const int d = gi / W::GPD;
        face(d, gi - d * W::GPD);
      }
    }
    __syncthreads();  // (C) every face slot is written

    // ---- flux differences of the thread's cell (and StateOld, loaded early)
    const int p = NT > 1 ? t / W::TC : 0, ct = t - p * W::TC;
    const int ci = ct % N, cj = (ct / N) & 3, ck = ct / (4 * N);
    const UnitMeta &m = M[NT > 1 ? min(p, NT - 1) : 0];
    const bool own = t < 128;
    double chg[8], divB = 0.0, vsum = 0.0, o[8], ub[6];
    size_t cell = 0;
    if (own) {
      cell = (size_t)m.b * 8 * (N * N * N) + ci + N * (cj + m.j0 + N * (ck + m.k0));
#pragma unroll
      for (int v = 0; v < 8; v++) o[v] = a.old[cell + v * (N * N * N)];
#pragma unroll
      for (int q = 0; q < 6; q++) ub[q] = P[p * PT + ct + (kUx + q) * PV];
      // FP32 fluxes: the three directions' differences are summed in FP32,
      // one conversion per variable
      Real cs[8], db = Real(0), vs = Real(0);
#pragma unroll
      for (int D = 0; D < 3; D++) {
        int f0, f1;
        cell_faces<W>(D, ci, cj, ck, f0, f1);
        const Real *F = fb + (D == 0 ? 0 : (D == 1 ? W::B1 : W::B2)) + p * (D == 0 ? W::F0 : W::F1);
#pragma unroll
        for (int v = 0; v < 8; v++) {
          const Real d = F[v * W::NF + f0] - F[v * W::NF + f1];
          cs[v] = D == 0 ? d : cs[v] + d;
        }
        const Real e = mul_rn((Real)m.g.invHalf[D], F[9 * W::NF + f1] - F[9 * W::NF + f0]);
        db = D == 0 ? e : db + e;
        if (a.computeDt) {
          const Real x = fmax(F[8 * W::NF + f0], F[8 * W::NF + f1]);
          vs = D == 0 ? x : vs + x;
        }
      }
#pragma unroll
      for (int v = 0; v < 8; v++) chg[v] = (double)cs[v];
      divB = (double)db;
      vsum = (double)vs;
    }
    __syncthreads();  // (D) the slots and P are read: the next unit's state streams in
    if (t == W::NTHR - 32 && it + 1 < nIter) {
      fence_proxy_async_smem();
      issue_unit<W, TileT>(maps, stg, &bar, meta[(it + 1) & 1]);
    }

    // ---- update_state_normal / update_explicit ---------------------------
    double dtmin = 1e300;
    if (own) {
      if (a.computeDt) dtmin = m.g.volume / vsum;
      update_cell<OutT>(a, DtNoCfl, m.g.invVolume, chg, divB, ub, o, reinterpret_cast<OutT *>(a.out) + cell,
                        N * N * N);
    }
    if (a.computeDt) {
      for (int off = 16; off > 0; off >>= 1) dtmin = fmin(dtmin, __shfl_xor_sync(0xffffffffu, dtmin, off));
      if (lane == 0 && warp < 4) wmin[warp] = dtmin;
      __syncthreads();  // (E) wmin is complete
      if (t < NT) {
        double w = fmin(wmin[4 / NT * t], wmin[4 / NT * t + 1]);
        if (NT == 1) w = fmin(w, fmin(wmin[2], wmin[3]));
        dtRun = fmin(dtRun, w);
        if (W::PARTS > 1) a.dtBlock[(size_t)kDtParts * M[t].b + M[t].part] = w;
        else store_block_dt(a.dtBlock, M[t].b, w);
      }
    }
  }
  if (a.computeDt && t < NT && nIter > 0)
    atomicMin(&a.ts->DtMinBits, (unsigned long long)__double_as_longlong(dtRun));
  if (err) atomicOr(&a.ts->errFlag, kErrHlld);
  if (t == 0 && sTimeout) {
    atomicOr(&a.ts->errFlag, kErrTimeout);
    // let loads already in flight land before the CTA exits (bounded)
    mbar_wait_bounded(&bar, 0);
    mbar_wait_bounded(&bar, 1);
  }
  finish_stage(a, step);
}

}  // namespace bx
