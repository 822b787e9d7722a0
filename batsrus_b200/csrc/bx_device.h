// bx_device.h -- structures shared by the host side of libbx200 and its
// kernels (plain C++ / CUDA, no torch types).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace bx {

enum { kErrHlld = 1, kErrNonPhysical = 2, kErrTimeout = 4 };

// SmallDouble of ModPartImplicit (src/ModPartImplicit.f90:34): a norm below
// it is replaced by 1 (Norm_V :465, the matvec's rms(x) :1192)
constexpr double kSmallDouble = 1.0e-30;

// Time-step bookkeeping kept in device memory so that whole steps can be
// captured in a CUDA graph (set_global_timestep, src/ModTimeStepControl.f90:
// 306-524, runs on the device).
struct StepState {
  double DtNoCfl;                 // DtMax_CB of every cell this step (Dt/Cfl)
  double Dt;                      // Cfl*DtNoCfl
  double tSimulation;
  unsigned long long DtMinBits;   // running min of cell time steps (bits)
  int nStep;
  int errFlag;
  unsigned nDone;                 // CTAs of the step's last stage that are through (finish_stage)
  int nLeft;                      // steps of the running bx_advance that are not through, and
  double tLimit;                  // its time limit (finish_stage)
};

// Floors of the updated state, each active where > 0: RhoMin_I (the
// UseRhoMin clamp, src/ModUpdateState.f90:901-908), pMin_I and TMin_I of
// limit_pressure (src/ModEnergy.f90:388-420) with NumDens = rho/MassIon
struct Floors {
  double rhoMin = 0.0, pMin = 0.0, tMin = 0.0, massIon = 1.0;
};

// per-block Cartesian geometry (BATL CellSize_DB, CellVolume_B,
// CellFace_DB = CellVolume_B/CellSize_DB)
struct BlockGeom {
  double cellSize[3];
  double volume;
  double area[3];
  double invHalf[3];  // 0.5/CellSize (DxInvHalf of calc_divb_source)
  double invVolume;   // 1/volume
};

// DtMax_B is kept in kDtParts parts per block (a unit of the 3D stage kernel
// covers one quarter of an 8^3 block); DtMax_B is the smallest of them
constexpr int kDtParts = 4;
__host__ __device__ inline void store_block_dt(double *dt, int b, double m) {
  for (int q = 0; q < kDtParts; q++) dt[(size_t)kDtParts * b + q] = m;
}

#ifdef __CUDACC__
// set_global_timestep (src/ModTimeStepControl.f90:306-524) on the device
__device__ inline void step_set_dt(StepState *ts, double tLimit, int useDtFixed, double dtFixed, double cfl) {
  ts->nStep = ts->nStep + 1;
  double dt;
  // BATS_advance always passes a positive limit (tSimulationMax or
  // huge(0.0)), so the first time-accurate step has Dt = 0
  if (useDtFixed) dt = dtFixed;
  else if (ts->nStep <= 1) dt = 0.0;
  else dt = __longlong_as_double((long long)ts->DtMinBits);
  if (tLimit > 0.0 && ts->tSimulation + cfl * dt > tLimit) dt = (tLimit - ts->tSimulation) / cfl;
  ts->DtNoCfl = dt;
  ts->Dt = cfl * dt;
  ts->DtMinBits = 0x7FF0000000000000ull;  // +inf
}

// end of BATS_advance: tSimulation += Dt/nStage per stage and the final
// adjustment to the time limit (src/ModBatsrusMethods.f90:606-640)
__device__ inline void step_end(StepState *ts, int nStage, double tLimit) {
  double t = ts->tSimulation;
  for (int s = 0; s < nStage; s++) t = t + ts->Dt / nStage;
  if (tLimit > 0.0 && t < tLimit && tLimit - t <= 1e-3 * ts->Dt) t = tLimit;
  ts->tSimulation = t;
}
#endif

struct StageArgs {
  const void *in;          // gather source (double* or float*)
  const double *old;       // StateOld: the step's initial state (own cells)
  void *out;               // stage result (double* or float*)
  const int *nbr;          // [nBlock][6] neighbour block or -1 (float BC)
  const int *order;        // processing order (Morton) of the blocks
  const BlockGeom *geom;   // [nBlock]
  StepState *ts;
  double *dtBlock;         // optional DtMax_B, kDtParts per block
  int nBlock;
  int iStage, nStage, nOrder, limiter, useDivb, useHalfStep, computeDt;
  double beta, gamma, invGm1, cfl;
  double dtFactor = 0.0;   // the stage's part of the time step: cfl, or cfl iStage/nStage (half step scheme)
  // the step's last stage: its last CTA ends the time step and, while steps
  // are left, sets the next one's time step (set_global_timestep)
  int finish = 0;
  int useDtFixed = 0;
  double dtFixed = 0.0;
  // residual mode of the 3D kernel (get_residual of the implicit scheme):
  // the input holds total energy in the pressure slot, the output is the
  // increment dtScale*DtMax_CB*(S + dF/V) of the implicit variables, with
  // DtMax_CB per cell (dtCellIn) or the global Dt/Cfl (dtCellIn == nullptr)
  int inputEnergy = 0, outputResidual = 0;
  const double *dtCellIn = nullptr;
  double *dtCellOut = nullptr;  // V/sum(Vdt) per cell when computeDt
  double dtScale = 0.5;
  // resolution changes (nbr == kNbrResChange): per block and side the level
  // difference (+1 coarser, -1 finer neighbour, else 0) and the slab holding
  // its two ghost layers ([slab][var][layer][t1][t0], FP64) and, on the
  // coarse side, the summed finer fluxes ([slab][t1][t0][10]: 8 fluxes, Vdt,
  // BnL + BnR)
  const int *rcType = nullptr;
  const int *rcSlab = nullptr;
  const double *rcGhost = nullptr;
  const double *rcFlux = nullptr;
  Floors fl;
  // #RESOLUTIONCHANGE: TVD faces next to a coarser block (tvd_reschange),
  // and BetaLimiterResChange for the nFaceRc cells next to a side with a
  // resolution change or an outer boundary when it is below beta
  int tvdRc = 0;
  double betaRc = 2.0;
  int nFaceRc = 2;
  // 0 when no block of the grid needs those resolution-change states (no
  // resolution change, and no sharper limiter next to a float boundary):
  // the stage kernel is then launched without that code
  int anySpecial = 1;
  int nRcBlock = 0;  // updated blocks with a side at a resolution change
  int isRank = 0;    // the blocks are one rank's part of a grid
};

#ifdef __CUDACC__
// The 1D stage kernel is launched as a programmatic dependent of the
// kernel before it (launch_dependent): its CTAs may start, and load what no
// kernel writes, while that kernel's last CTAs run; grid_wait returns when it
// has ended and its writes are visible.  grid_go lets the next kernel start
// so.  (The persistent 3D kernel gains nothing by it: 64^3 96.1 against 96.8
// us per step, 160^3 1265 against 1254.)
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_dependent(void (*k)(P...), int grid, int block, size_t smem, cudaStream_t st, const A &...args) {
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...);
}
#endif

#ifdef __CUDACC__
// The end of a stage kernel, called by every thread of the CTA after its last
// access to the time-step state: the last CTA through ends the time step and
// sets the next one's, in place of two launches of one thread each (5 us of
// a step's 23 on a grid of 16^3).  Every CTA has read DtNoCfl and added its
// minimum before it counts itself.  The steps left and the time limit stand in
// the state, so that the launches of all steps are alike.  What the last CTA
// needs but the minimum does not change during the stage: thread 0 of every
// CTA loads it early (load_step, into shared memory), since a load at the
// end queues behind the other CTAs' atomics on the same line (two of them
// cost 2 us of a step at 16^3).
__device__ __forceinline__ void load_step(const StageArgs &a, StepState &s) {
  if (!a.finish || threadIdx.x != 0) return;
  s.DtNoCfl = a.ts->DtNoCfl;
  s.Dt = a.ts->Dt;
  s.tSimulation = a.ts->tSimulation;
  s.nStep = a.ts->nStep;
  s.nLeft = a.ts->nLeft;
  s.tLimit = a.ts->tLimit;
}

__device__ __forceinline__ void finish_stage(const StageArgs &a, const StepState &loaded) {
  if (!a.finish) return;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&a.ts->nDone, 1u) == gridDim.x - 1) {
      __threadfence();
      StepState s = loaded;
      s.DtMinBits = atomicAdd(&a.ts->DtMinBits, 0ull);
      step_end(&s, a.nStage, s.tLimit);
      s.nLeft = s.nLeft - 1;
      if (s.nLeft > 0) step_set_dt(&s, s.tLimit, a.useDtFixed, a.dtFixed, a.cfl);
      a.ts->DtNoCfl = s.DtNoCfl;
      a.ts->Dt = s.Dt;
      a.ts->tSimulation = s.tSimulation;
      a.ts->nStep = s.nStep;
      a.ts->DtMinBits = s.DtMinBits;
      a.ts->nDone = 0;
      a.ts->nLeft = s.nLeft;
    }
  }
}
#endif

constexpr int kNbrFloat = -1, kNbrResChange = -2;
constexpr int kRcSlots = 10;

// per-block compatibility kernels (orig-path entry points, FP64)
struct CompatArgs {
  const double *state;     // current state (SoA, no ghosts)
  const double *old;       // StateOld buffer
  double *next;            // updated block output
  const int *nbr;
  const BlockGeom *geom;
  StepState *ts;
  double *left[3], *right[3], *flux[3];  // face scratch of one block
  double *source;          // Source_VC scratch (9 per cell)
  double *dtCell;          // DtMax_CB of the block (nCell)
  double *dtBlock;         // DtMax_B, kDtParts per block
  int iStage, nStage, nOrder, limiter, useDivb, useHalfStep;
  double beta, gamma, invGm1, cfl;
  Floors fl;
};

// shape ids of the supported block sizes
enum { kShape888 = 0, kShape444 = 1, kShape881 = 2, kShape811 = 3, kShape6411 = 4, kNumShape = 5 };

// launchers (explicitly instantiated in bx_stage_line.cu, bx_stage_flat.cu and
// bx_compat.cu): 1D blocks, 2D blocks
cudaError_t launch_stage_line(int shape, int flux, const StageArgs &a, cudaStream_t st);
cudaError_t launch_stage_flat(int flux, const StageArgs &a, int nSM, cudaStream_t st);
cudaError_t launch_compat(int shape, int flux, int phase, int iBlock, const CompatArgs &a,
                          cudaStream_t st);
// persistent TMA-staged kernel of 3D shapes (bx_stage3d.cu): tensor maps of
// the stage input for the interior box and the x, y, z ghost slabs of a
// block, and those of a tile of 4 x 4 rows (bx_stage_unit.cuh)
struct alignas(64) TmaMaps {
  CUtensorMap in, xh, yh, zh;
  CUtensorMap uin, uxh, uyh, uzh;
};
enum { kKindFp64 = 0, kKindFp32In64 = 1, kKindFp32In32 = 2 };
cudaError_t launch_stage3d(int shape, int flux, int kind, const TmaMaps &maps, const StageArgs &a, int nSM,
                           cudaStream_t st);
// whether an explicit stage runs in units (bx_stage_unit.cuh), which carry out
// StageArgs::finish
bool stage3d_units(int shape, int flux, int kind, const StageArgs &a, int nSM);
enum { kPhaseFaceValue = 0, kPhaseFaceFlux = 1, kPhaseSource = 2, kPhaseUpdate = 3, kPhaseTimestep = 4 };

}  // namespace bx
