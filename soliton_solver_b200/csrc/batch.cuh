// batch.cuh -- many independent lattices of one theory advanced together.
//
// One launch per phase of the RK4 step (rk.cuh) covers the tiles of every lattice: block b
// works on tile b - tile0[i] of lattice i = tile_inst[b].  Each lattice keeps its own
// parameters, buffers, reduction partials and device step state (energy, arrest flag, err),
// so sizes, couplings and arrest histories are independent; the per-lattice last block
// (ticket counted per lattice) finalises that lattice's reductions.
#pragma once

#include "rk.cuh"

namespace ssb {

// a lattice's buffers (BatchInst::buf) and halo-box TMA maps (BatchInst::tm, the buffers
// BATCH_TM_BUF names: phi and V of both pairs in phase A's tile, then in phase B's, l1, l2)
enum { BB_FIELD = 0, BB_VEL = 1, BB_PHI2 = 2, BB_VEL2 = 3, BB_L1 = 4, BB_L2 = 5, BB_COUNT = 6 };
enum { BT_A = 0, BT_B = 4, BT_L = 8, BT_COUNT = 10 };
constexpr int BATCH_TM_BUF[BT_COUNT] = {BB_FIELD, BB_VEL, BB_PHI2, BB_VEL2, BB_FIELD,
                                        BB_VEL,   BB_PHI2, BB_VEL2, BB_L1,  BB_L2};

struct BatchInst {
  CUtensorMap tm[BT_COUNT];
  Grid G;
  Phys P;
  void* buf[BB_COUNT];
  StepState* st;
  double* partial;    // one slot per tile of this lattice
  double* E_traj;     // per-lattice trajectory rows
  double* err_traj;
  int tile0[2], ntiles[2];  // of phases A (and E) and B
};

struct BatchStep {
  int cur;   // the pair that holds phi and V: 0 the caller's, 1 the workspace's
  int copy;  // A: phi and V to the workspace's pair (first step of an odd count)
  int with_energy, arrest_update, init_state;
  int E_idx, err_idx;
  const double* prev_energy;  // device, one per lattice (NaN keeps E_last); read with init_state
  long long wait_cycles;
};

// Tile shapes of the batched phases: as the single lattice's, or (SMALL) 8 x 32 sites per
// 128-thread CTA.  Each CTA stages, computes and stores one tile, so the staging latency is
// hidden only by other resident CTAs.
template <class TH, typename R, int PH, bool SMALL>
struct BatchShape {
  using SH = StepShape<TH, R, PH>;
  // six FP64 components run phase A at one CTA per SM: 16 rows, so that fewer loads are waited for
  static constexpr bool TALL = PH != PH_B && sizeof(R) == 8 && TH::NF > 4;
  static constexpr int TX = SMALL ? 8 : TALL ? 16 : SH::TX, TY = SMALL ? 32 : SH::TY, NT = SMALL ? 128 : SH::NT;
  // (FP64 phase E stages one buffer and needs few registers: one CTA more, as with plain rows)
  static constexpr int CTAS = SMALL ? (TH::NF > 4 ? 4 : PH == PH_B ? 5 : 6)
                                    : SH::CTAS + (PH == PH_E && sizeof(R) == 8 ? 1 : 0);
};

template <class TH, typename R, bool SMALL, bool TMA, int PH>
__global__ void __launch_bounds__((BatchShape<TH, R, PH, SMALL>::NT), (BatchShape<TH, R, PH, SMALL>::CTAS))
    batch_step_kernel(const BatchInst* __restrict__ insts, const int* __restrict__ tile_inst,
                      const __grid_constant__ BatchStep B) {
  using SH = BatchShape<TH, R, PH, SMALL>;
  constexpr int TX = SH::TX, TY = SH::TY, NT = SH::NT, p = PH == PH_B ? 1 : 0;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ StageShared<NT> S;
  __shared__ StepArgs<R> A;
  const int inst = tile_inst[blockIdx.x];
  const BatchInst& I = insts[inst];
  const CUtensorMap* tm_phi = &I.tm[(PH == PH_B ? BT_B : BT_A) + 2 * B.cur];
  const CUtensorMap* tm_vel = tm_phi + 1;
  const CUtensorMap* tm_l1 = &I.tm[BT_L];
  const int tile = blockIdx.x - I.tile0[p];
  if constexpr (TMA) {
    // the tile's loads first, so the set-up below overlaps them
    if (threadIdx.x == 0) {
      const int tiles_y = (I.G.Y + TY - 1) / TY;
      mbar_init(&S.bar, 1);
      issue_step_tile<TH, R, TX, TY, NT, PH>(reinterpret_cast<R*>(smem_raw), tm_phi, tm_vel, tm_l1, tm_l1 + 1,
                                             (tile / tiles_y) * TX, (tile % tiles_y) * TY, &S.bar, I.st, 0u, 0);
    }
  }
  {  // the lattice's parameters into shared memory (word copy)
    const int* src = reinterpret_cast<const int*>(&I.G);
    int* dst = reinterpret_cast<int*>(&A.G);
    for (int i = threadIdx.x; i < (int)(sizeof(Grid) / 4); i += NT) dst[i] = src[i];
    src = reinterpret_cast<const int*>(&I.P);
    dst = reinterpret_cast<int*>(&A.P);
    for (int i = threadIdx.x; i < (int)(sizeof(Phys) / 4); i += NT) dst[i] = src[i];
  }
  if (threadIdx.x == 0) {
    const int in = 2 * B.cur, out = 2 - in;
    A.phi = (const R*)I.buf[in];
    A.vel = (const R*)I.buf[in + 1];
    A.l1 = A.out_l1 = (R*)I.buf[BB_L1];
    A.l2 = A.out_l2 = (R*)I.buf[BB_L2];
    A.phi_out = (R*)I.buf[out];
    A.vel_out = (R*)I.buf[out + 1];
    A.copy_phi = B.copy ? (R*)I.buf[BB_PHI2] : nullptr;
    A.copy_vel = B.copy ? (R*)I.buf[BB_VEL2] : nullptr;
    A.force = nullptr;
    A.partial = I.partial;
    A.st = I.st;
    A.E_traj = I.E_traj;
    A.err_traj = I.err_traj;
    A.E_idx = B.E_idx;
    A.err_idx = B.err_idx;
    A.with_energy = B.with_energy;
    A.arrest_update = B.arrest_update;
    A.init_state = B.init_state;
    A.predict = 0;
    A.prev_energy = B.prev_energy ? B.prev_energy[inst] : NAN;
    A.wait_cycles = B.wait_cycles;
    A.tx_extra = 0;
  }
  __syncthreads();
  step_tile<TH, R, TX, TY, NT, TMA, PH>(A, tm_phi, tm_vel, tm_l1, tm_l1 + 1, tile, I.ntiles[p], smem_raw, S, TMA);
}

// Apply each lattice's pending arrest (V = 0), left by the trailing energy pass, at the
// end of a call.  grid.y = lattice.
template <typename R, int NF>
__global__ void batch_finish_kernel(const BatchInst* __restrict__ insts) {
  const BatchInst& I = insts[blockIdx.y];
  if (!I.st->arrest) return;
  R* dv = (R*)I.buf[BB_VEL];
  const long long n = (long long)NF * I.G.N;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    dv[i] = (R)0;
}

}  // namespace ssb
