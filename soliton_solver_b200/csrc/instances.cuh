// instances.cuh -- the kernels compiled in translation units of their own (coop.cu, batch.cu, plain.cu), so
// that the library's parts compile side by side.  SSB_INSTANCE is `extern` where they are only
// launched (abi.cu) and empty in the unit that holds them.
#pragma once

#include "batch.cuh"
#include "coop.cuh"

#define SSB_FOR_THEORIES(M) M(ChiralMagnet) M(BabySkyrme) M(GinzburgLandau) M(Anisotropic)

// every tile shape, with 16-byte and single-element staging; the third shape's buffers for six FP64
// components do not fit an SM
#define SSB_COOP(TH, R, TX, TY, NT, SPLIT, VW)                                          \
  SSB_INSTANCE template __global__ void coop_step_kernel<TH, R, TX, TY, NT, SPLIT, VW>( \
      const __grid_constant__ StepArgs<R>, const __grid_constant__ CoopArgs<R>);
#define SSB_COOP_SMALL(TH, R, VW) SSB_COOP(TH, R, 8, 32, 256, true, VW) SSB_COOP(TH, R, 16, 32, 128, false, VW)
#define SSB_COOP_LARGE(TH, R, VW) SSB_COOP(TH, R, 16, 64, 256, false, VW)
#define SSB_COOP_ALL(TH) \
  SSB_COOP_SMALL(TH, float, 1) SSB_COOP_SMALL(TH, float, 4) SSB_COOP_SMALL(TH, double, 1) SSB_COOP_SMALL(TH, double, 2)
#define SSB_COOP_INSTANCES                                                                          \
  SSB_FOR_THEORIES(SSB_COOP_ALL)                                                                    \
  SSB_COOP_LARGE(ChiralMagnet, float, 1) SSB_COOP_LARGE(ChiralMagnet, float, 4)                     \
  SSB_COOP_LARGE(BabySkyrme, float, 1) SSB_COOP_LARGE(BabySkyrme, float, 4)                         \
  SSB_COOP_LARGE(GinzburgLandau, float, 1) SSB_COOP_LARGE(GinzburgLandau, float, 4)                 \
  SSB_COOP_LARGE(Anisotropic, float, 1) SSB_COOP_LARGE(Anisotropic, float, 4)                       \
  SSB_COOP_LARGE(ChiralMagnet, double, 1) SSB_COOP_LARGE(ChiralMagnet, double, 2)                   \
  SSB_COOP_LARGE(BabySkyrme, double, 1) SSB_COOP_LARGE(BabySkyrme, double, 2)                       \
  SSB_COOP_LARGE(GinzburgLandau, double, 1) SSB_COOP_LARGE(GinzburgLandau, double, 2)

// phases A, B, E: TMA and plain staging, the small tiles for TMA-staged FP32
#define SSB_BATCH(TH, R, SMALL, TMA, PH)                                     \
  SSB_INSTANCE template __global__ void batch_step_kernel<TH, R, SMALL, TMA, PH>( \
      const BatchInst* __restrict__, const int* __restrict__, const __grid_constant__ BatchStep);
#define SSB_BATCH_PHASES(TH, R, SMALL, TMA) \
  SSB_BATCH(TH, R, SMALL, TMA, PH_A) SSB_BATCH(TH, R, SMALL, TMA, PH_B) SSB_BATCH(TH, R, SMALL, TMA, PH_E)
#define SSB_BATCH_ALL(TH)                                                                   \
  SSB_BATCH_PHASES(TH, float, false, true) SSB_BATCH_PHASES(TH, float, false, false)        \
  SSB_BATCH_PHASES(TH, float, true, true) SSB_BATCH_PHASES(TH, double, false, true)         \
  SSB_BATCH_PHASES(TH, double, false, false)
#define SSB_BATCH_INSTANCES SSB_FOR_THEORIES(SSB_BATCH_ALL)

// the FP32 step of plain rows
#define SSB_PLAIN(TH, PH)                                               \
  SSB_INSTANCE template __global__ void step_kernel<TH, float, false, PH>( \
      const __grid_constant__ StepMaps, const __grid_constant__ StepArgs<float>);
#define SSB_PLAIN_ALL(TH) SSB_PLAIN(TH, PH_A) SSB_PLAIN(TH, PH_B) SSB_PLAIN(TH, PH_E)
#define SSB_PLAIN_INSTANCES SSB_FOR_THEORIES(SSB_PLAIN_ALL)
