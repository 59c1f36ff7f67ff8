// rk.cuh -- the arrested-Newton-flow RK4 step in two phases.
//
// One RK4 step of the reference (core/integrator.py:217-348) is
//   k1 = dt V,            T1 = phi,           l1 = -dt G(T1)
//   k2 = dt (V + l1/2),   T2 = phi + k1/2,    l2 = -dt G(T2)
//   k3 = dt (V + l2/2),   T3 = phi + k2/2,    l3 = -dt G(T3)
//   k4 = dt (V + l3),     T4 = phi + k3,      l4 = -dt G(T4)
//   V' = V + (l1 + 2 l2 + 2 l3 + l4)/6,  phi' = phi + (k1 + 2 k2 + 2 k3 + k4)/6
// followed by the unit-norm re-projection, the energy of phi', the arrest test
// (E' > E -> V' = 0) and err = max G(T4).  T2 holds no l at all and T3, T4 hold l1 and l2
// only, so the four gradients form two independent pairs and a step is two kernels:
//   phase A  reads phi, V          writes l1, l2     (+ the energy of phi)
//   phase B  reads phi, V, l1, l2  writes phi', V'   (+ err)
// 10 words per site and step, two launches.  Phase B reads the neighbours of phi and V, so
// steps alternate between the caller's buffers and a pair in the workspace; an odd number of
// steps starts in that pair: the first phase A, which reads phi and V anyway, copies them there.
// The energy of a step's result is computed by the next step's phase A.  The arrest it
// decides (V = 0) is applied by phase B: V = 0 means T2 = T1, so l2 = l1 and phase B takes
// l1 for l2 (and loads neither V nor l2); phase A's l2, computed before the decision, is
// dropped.
// Saddle flows (the chiral magnet with demag: its psi is maximised, E rises) arrest nearly
// every step.  After two arrested steps in a row phase A expects the next: it reads phi alone
// and writes l1 alone, and should the energy fall after all, phase A2 (a launch that returns
// at once otherwise) supplies l2 before phase B: 6 words and three gradients per arrested step.
#pragma once

#include "flow.cuh"

namespace ssb {

enum StepPhase { PH_A = 0, PH_B = 1, PH_E = 2, PH_A2 = 3 };

// TMA maps of a phase's inputs: halo boxes of its tile shape
struct StepMaps {
  CUtensorMap phi, vel, l1, l2;
};
template <typename R>
struct StepArgs {
  const R* phi;
  const R* vel;
  const R* l1;  // B
  const R* l2;  // B
  R* out_l1;    // A
  R* out_l2;    // A
  R* phi_out;   // B: phi'
  R* vel_out;   // B: V'
  R* copy_phi;  // A (nullable): copies of phi and V for phase B to read
  R* copy_vel;
  const double* force;  // FP64 fields (nullable): added to the gradient rows in every stage
  double* partial;      // one energy partial per tile (A, E)
  StepState* st;
  double* E_traj;    // nullable
  double* err_traj;  // nullable
  int E_idx;         // slot of E_traj the energy goes to (< 0: none)
  int err_idx;       // slot of err_traj the error goes to (< 0: none)
  int with_energy;    // A, E: reduce the energy of phi
  int arrest_update;  // after the energy: arrest = killkinen && E > E_last; E_last = E
  int init_state;     // first phase A of a call: arrest = 0 and (unless NaN) E_last = prev_energy
  int predict;        // A: leave l2 out after two arrested steps in a row
  double prev_energy;
  long long wait_cycles;  // bound of every mbarrier wait (clock64 cycles)
  unsigned tx_extra;      // test hook: bytes the barrier expects beyond what is loaded (normally 0)
  Grid G;
  Phys P;
};

// Tile rows, threads and resident CTAs per SM of each phase (tiles are TX x 64 sites, a
// warp owns rows).  Registers follow from the CTAs: 64 for the chiral magnet's phase A, 80
// for the phase A of the other FP32 theories with up to four components and for the baby
// Skyrme phase B, else 128 (at most 52 bytes of spills; in the batched kernels up to 188, FP64 baby
// Skyrme's phase B); the s+id model's FP64 stencils take up to 255 and one CTA.
// Phase B stages four halo buffers by TMA: 16 rows where two CTAs' buffers fit an SM (FP32, up to
// four components), else 8.  Plain loads stage two (one in E), which fit at 16 rows in FP64 too, and fewer
// halo rows count there: every element is a load of its own.
template <class TH, typename R, int PH, bool TMA = true>
struct StepShape {
  static constexpr int TY = 64, NT = 256;
  static constexpr int BYTES = (int)sizeof(R) * TH::NF;  // per site
  static constexpr bool F32 = sizeof(R) == 4;
  static constexpr int TX = (!TMA && !F32) || BYTES <= (PH == PH_B ? 16 : 32) ? 16 : 8;
  static constexpr int PLAIN_E = PH == PH_E && !TMA ? 1 : 0;  // FP64: one buffer and few registers
  static constexpr int CTAS = TH::NF > 4                       ? (F32 ? 2 : 1 + PLAIN_E)
                              : !F32                           ? 2 + PLAIN_E
                              : PH == PH_B                     ? (TH::NF <= 3 ? 3 : 2)
                              : PH == PH_E || TH::S1_CTAS == 4 ? 4
                                                               : 3;
};
// halo buffers staged per phase (TMA: phi; V; l1, l2.  Plain loads combine on the way in: T1, T2 / T3, T4)
template <int PH, bool TMA>
__host__ __device__ constexpr int step_buffers() {
  return PH == PH_E ? 1 : (PH == PH_B && TMA) ? 4 : 2;  // A, A2: phi, V
}
template <class TH, typename R, int PH, bool TMA>
__host__ __device__ constexpr size_t step_smem() {
  using SH = StepShape<TH, R, PH, TMA>;
  return step_buffers<PH, TMA>() * tile_buf_bytes<R, TH::NF, SH::TX, SH::TY>();
}

// The flow's gradient rows of a site pair from the staged field T: jets, theory, forcing,
// halo zeroing and tangent projection.
template <class TH, typename V, typename R, int HY, int PLANE, bool FAST>
__device__ __forceinline__ void pair_gradient(const StepArgs<R>& A, const R* T, int toff, const PairCoef<V>& kc,
                                              const Masks& m0, const Masks& m1, int gx, int gy, long long sidx,
                                              bool v1, Jet<V, TH::NF>& J, V* g) {
  constexpr int NF = TH::NF;
  tile_jet<TH, V, R, HY, PLANE, FAST>(T, toff, kc, m0, m1, J);
  TH::gradient(J, A.P, g);
  if constexpr (sizeof(R) == 8) {
    if (A.force) {
      V fo[NF];
#pragma unroll
      for (int a = 0; a < NF; ++a) fo[a] = gload<V, double>(A.force + a * A.G.N + sidx, FAST, v1);
      TH::flow_rows(fo, A.P);
#pragma unroll
      for (int a = 0; a < NF; ++a) g[a] = g[a] + fo[a];
    }
  }
  flow_constraints<TH, V, FAST>(A.G, J, g, gx, gy);
}

// Flow energy (without dA) of a site pair from its jets: in the field's precision where the
// theory has energy_pair, else FP64 on the (converted) jets.
template <class TH, typename V, typename R>
__device__ __forceinline__ double pair_energy(const Jet<V, TH::NF>& J, const Phys& P, bool v1, V& chk) {
  if constexpr (TH::PAIR_ENERGY) {
    const V ep = TH::energy_pair(J, P);
    double e = (double)Lanes<V>::get(ep, 0);
    if (v1) e += (double)Lanes<V>::get(ep, 1);
    return e;
  } else if constexpr (sizeof(R) == 8) {
    Jet1<double, TH::NF> J0, J1;
#pragma unroll
    for (int a = 0; a < TH::NF; ++a) {
      J0.f[a] = J.f[a].x;
      J0.dx[a] = J.dx[a].x;
      J0.dy[a] = J.dy[a].x;
      J1.f[a] = J.f[a].y;
      J1.dx[a] = J.dx[a].y;
      J1.dy[a] = J.dy[a].y;
    }
    double e = TH::energy(J0, P, 1.0);
    if (v1) e += TH::energy(J1, P, 1.0);
    return e;
  } else {
    return jet_energy<TH, V, TH::NF>(J, P, 1.0, v1, chk);
  }
}

// Phase A (l1, l2 and the energy; skip: no l2), A2 (l2) or E (the energy) of a staged tile.
template <class TH, typename R, int TX, int TY, int NT, bool FAST, int PH>
__device__ __forceinline__ void first_half(const StepArgs<R>& A, const R* T1, const R* T2, int x0, int y0,
                                           bool skip, double* e_acc) {
  using TS = TileShape<TX, TY, NT>;
  using V = typename PairOf<R>::type;
  using S = typename ScalarOf<V>::type;
  constexpr int NF = TH::NF, PAIRS = TY / 2, RPP = NT / PAIRS;
  static_assert(NT % PAIRS == 0 && TX % RPP == 0, "pair mapping");
  const Grid& G = A.G;
  const long long N = G.N;
  const PairCoef<V> kc(G);
  const V mdt(grid_k<S>(G, GK_MDT));
  const int j = threadIdx.x % PAIRS;
  const int lxg = threadIdx.x / PAIRS;
  V chk(0.0);
  double e_sum = 0.0;
#pragma unroll(PH == PH_E && sizeof(R) == 4 ? 2 : 1)
  for (int pass = 0; pass < TX / RPP; ++pass) {
    const int lx = lxg * (TX / RPP) + pass;  // adjacent rows
    const int gx = x0 + lx, gy = y0 + 2 * j;
    bool v1 = true;
    Masks m0{true, true, true}, m1{true, true, true};
    if (!FAST) {
      if (gx >= G.X || gy >= G.Y) continue;
      v1 = gy + 1 < G.Y;
      m0 = site_masks(G, gx, gy);
      m1 = site_masks(G, gx, gy + 1);
      if (!v1) m1 = Masks{false, false, false};
    }
    const int toff = (lx + 2) * TS::HY + TS::YOFF + 2 * j;
    const long long sidx = (long long)gx * G.Y + gy;
    Jet<V, NF> J;
    if constexpr (PH == PH_E) {
      tile_jet<TH, V, R, TS::HY, TS::PLANE, FAST>(T1, toff, kc, m0, m1, J);
      e_sum += pair_energy<TH, V, R>(J, A.P, v1, chk);
    } else {
      V g[NF];
      if constexpr (PH == PH_A) {
        pair_gradient<TH, V, R, TS::HY, TS::PLANE, FAST>(A, T1, toff, kc, m0, m1, gx, gy, sidx, v1, J, g);
        if (e_acc) e_sum += pair_energy<TH, V, R>(J, A.P, v1, chk);
#pragma unroll
        for (int a = 0; a < NF; ++a) gstore<V, R>(A.out_l1 + a * N + sidx, mdt * g[a], FAST, v1);
        if (skip) continue;
      }
      pair_gradient<TH, V, R, TS::HY, TS::PLANE, FAST>(A, T2, toff, kc, m0, m1, gx, gy, sidx, v1, J, g);
#pragma unroll
      for (int a = 0; a < NF; ++a) gstore<V, R>(A.out_l2 + a * N + sidx, mdt * g[a], FAST, v1);
    }
  }
  if (e_acc) *e_acc = e_sum * G.dA + (double)(Lanes<V>::get(chk, 0) + Lanes<V>::get(chk, 1));
}

// The raw l1 and l2 of the thread's own pairs, read from the staged buffers before T3 and T4
// replace them there.
template <typename V, int NF, int PASSES>
struct CentreL {
  V l1[PASSES][NF], l2[PASSES][NF];
};

// Phase B of a staged tile: l3 from T3, l4 from T4, then phi' and V'.
//   TMA: phi and V are the staged raw buffers, C the centre l1 and l2
//   plain loads: phi, V, l1, l2 come from global memory
template <class TH, typename R, int TX, int TY, int NT, bool TMA, bool FAST, class CL>
__device__ __forceinline__ void second_half(const StepArgs<R>& A, const R* T3, const R* T4, const R* Bphi,
                                            const R* Bvel, const CL& C, int x0, int y0, bool arrest,
                                            double& err_max) {
  using TS = TileShape<TX, TY, NT>;
  using V = typename PairOf<R>::type;
  using S = typename ScalarOf<V>::type;
  constexpr int NF = TH::NF, PAIRS = TY / 2, RPP = NT / PAIRS;
  static_assert(NT % PAIRS == 0 && TX % RPP == 0, "pair mapping");
  const Grid& G = A.G;
  const long long N = G.N;
  const PairCoef<V> kc(G);
  const V mdt(grid_k<S>(G, GK_MDT)), sixth(grid_k<S>(G, GK_SIXTH)), two(2.0), dtv(grid_k<S>(G, GK_DT)),
      dt6(grid_k<S>(G, GK_DT6));
  const int j = threadIdx.x % PAIRS;
  const int lxg = threadIdx.x / PAIRS;
  S emax = -INFINITY;
#pragma unroll
  for (int pass = 0; pass < TX / RPP; ++pass) {
    const int lx = lxg * (TX / RPP) + pass;
    const int gx = x0 + lx, gy = y0 + 2 * j;
    bool v1 = true;
    Masks m0{true, true, true}, m1{true, true, true};
    if (!FAST) {
      if (gx >= G.X || gy >= G.Y) continue;
      v1 = gy + 1 < G.Y;
      m0 = site_masks(G, gx, gy);
      m1 = site_masks(G, gx, gy + 1);
      if (!v1) m1 = Masks{false, false, false};
    }
    const int toff = (lx + 2) * TS::HY + TS::YOFF + 2 * j;
    const long long sidx = (long long)gx * G.Y + gy;
    Jet<V, NF> J;
    V g[NF], Pn[NF], Vn[NF];
    pair_gradient<TH, V, R, TS::HY, TS::PLANE, FAST>(A, T3, toff, kc, m0, m1, gx, gy, sidx, v1, J, g);
    // phi' and V' but for l4 (core/integrator.py:151-189 with k1 = dt V, k2 = dt (V + l1/2),
    // k3 = dt (V + l2/2)), so that only these two stay live across the second stencil
#pragma unroll
    for (int a = 0; a < NF; ++a) {
      V p, v, l1, l2;
      if constexpr (TMA) {
        p = ld_pair(Bphi + a * TS::PLANE + toff);
        v = arrest ? V(0.0) : ld_pair(Bvel + a * TS::PLANE + toff);
        l1 = C.l1[pass][a];
        l2 = C.l2[pass][a];
      } else {
        p = gload<V, R>(A.phi + a * N + sidx, FAST, v1);
        v = arrest ? V(0.0) : gload<V, R>(A.vel + a * N + sidx, FAST, v1);
        l1 = gload<V, R>(A.l1 + a * N + sidx, FAST, v1);
        l2 = arrest ? l1 : gload<V, R>(A.l2 + a * N + sidx, FAST, v1);
      }
      const V l3 = mdt * g[a];
      Vn[a] = vfma(sixth, vfma(two, l3, vfma(two, l2, l1)), v);
      Pn[a] = vfma(dt6, (l1 + l2) + l3, vfma(dtv, v, p));
    }
    pair_gradient<TH, V, R, TS::HY, TS::PLANE, FAST>(A, T4, toff, kc, m0, m1, gx, gy, sidx, v1, J, g);
#pragma unroll
    for (int a = 0; a < NF; ++a) {
      Vn[a] = vfma(sixth, mdt * g[a], Vn[a]);
      emax = fmax(emax, Lanes<V>::get(g[a], 0));
      if (v1) emax = fmax(emax, Lanes<V>::get(g[a], 1));
    }
    // re-projected onto the sphere, V' onto the tangent space of phi'
    // (compute_norm_magnetization and project_orthogonal_magnetization,
    // chiral_magnet/kernels.py:48-122)
    if (TH::CONSTRAINED && G.unit_mag) {
      unit_project<TH::NMAG>(Pn);
      V lm = Vn[0] * Pn[0];
#pragma unroll
      for (int a = 1; a < TH::NMAG; ++a) lm = vfma(Vn[a], Pn[a], lm);
      const V mlm = -lm;
#pragma unroll
      for (int a = 0; a < TH::NMAG; ++a) Vn[a] = vfma(mlm, Pn[a], Vn[a]);
    }
#pragma unroll
    for (int a = 0; a < NF; ++a) {
      gstore<V, R>(A.phi_out + a * N + sidx, Pn[a], FAST, v1);
      gstore<V, R>(A.vel_out + a * N + sidx, Vn[a], FAST, v1);
    }
    asm volatile("" ::: "memory");  // one row at a time: the next row's loads would spill
  }
  err_max = fmax(err_max, (double)emax);
}

// Plain-load staging of a phase (row pitch not a multiple of 16 bytes): T1 = phi and T2 (A),
// T1 (E) or T3 and T4 (B; an arrested step takes V = 0 and l1 for l2) into D0 and D1.  Every
// thread issues the loads of one component plane before it combines them.  FUSED_T2: T2 rounded
// as in TMA-staged tiles.
template <int NF, typename R, int TX, int TY, int NT, int PH, bool FUSED_T2 = false>
__device__ inline void stage_step_plain(R* D0, R* D1, const StepArgs<R>& A, int x0, int y0, bool arrest) {
  using TS = TileShape<TX, TY, NT>;
  constexpr int KM = (TS::PLANE + NT - 1) / NT;
  const Grid& G = A.G;
  const R dt = (R)G.dt;
  long long off[KM];
  constexpr bool COPY = PH == PH_A && sizeof(R) == 8;  // FP64: phi and V to copy_phi and copy_vel on the way
  bool ok[KM], own[COPY ? KM : 1];
#pragma unroll
  for (int k = 0; k < KM; ++k) {
    const int i = threadIdx.x + k * NT;
    const int r = i / TS::HY, c = i - r * TS::HY;
    const int gx = x0 - 2 + r, gy = y0 - TS::YOFF + c;
    ok[k] = i < TS::PLANE && gx >= 0 && gx < G.X && gy >= 0 && gy < G.Y;
    off[k] = (long long)gx * G.Y + gy;
    if constexpr (COPY) own[k] = ok[k] && r >= 2 && r < TX + 2 && c >= TS::YOFF && c < TS::YOFF + TY;
  }
#pragma unroll 1
  for (int a = 0; a < NF; ++a) {
    const long long base = (long long)a * G.N;
    R p[KM], v[KM], w[KM], u[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) {
      p[k] = ok[k] ? A.phi[base + off[k]] : (R)0;
      if constexpr (PH != PH_E) v[k] = (ok[k] && !arrest) ? A.vel[base + off[k]] : (R)0;
      if constexpr (PH == PH_B) {
        w[k] = ok[k] ? A.l1[base + off[k]] : (R)0;
        u[k] = (ok[k] && !arrest) ? A.l2[base + off[k]] : (R)0;
      }
    }
#pragma unroll
    for (int k = 0; k < KM; ++k) {
      const int i = threadIdx.x + k * NT;
      if (i >= TS::PLANE) continue;
      if constexpr (PH == PH_B) {
        const R l2 = arrest ? w[k] : u[k];
        D0[a * TS::PLANE + i] = stage_t3<R>(p[k], v[k], w[k], dt);
        D1[a * TS::PLANE + i] = vfma(dt, vfma((R)0.5, l2, v[k]), p[k]);
      } else {
        D0[a * TS::PLANE + i] = p[k];
        if constexpr (COPY) {
          if (A.copy_phi && own[k]) {
            A.copy_phi[base + off[k]] = p[k];
            A.copy_vel[base + off[k]] = v[k];
          }
        }
        if constexpr (PH == PH_A)
          D1[a * TS::PLANE + i] = FUSED_T2 ? vfma(grid_k<R>(G, GK_HDT), v[k], p[k]) : stage_t2<R>(p[k], v[k], dt);
      }
    }
  }
}

// The tile's own phi and V from the staged raw buffers to copy_phi and copy_vel (TMA staging:
// rows, row pitch and buffers are 16-byte multiples, so no vector straddles the lattice's edge).
template <class TH, typename R, int TX, int TY, int NT>
__device__ __forceinline__ void copy_tile(const StepArgs<R>& A, const R* B0, int x0, int y0) {
  using TS = TileShape<TX, TY, NT>;
  constexpr int VW = 16 / (int)sizeof(R), CH = TY / VW;
  static_assert(TY % VW == 0 && TS::YOFF % VW == 0 && TS::HY % VW == 0 && TS::PLANE % VW == 0, "16-byte vectors");
  for (int i = threadIdx.x; i < TX * CH; i += NT) {
    const int lx = i / CH, c = (i % CH) * VW, gx = x0 + lx, gy = y0 + c;
    if (gx >= A.G.X || gy >= A.G.Y) continue;
    const R* t = B0 + (lx + 2) * TS::HY + TS::YOFF + c;
    const long long g = (long long)gx * A.G.Y + gy;
#pragma unroll
    for (int a = 0; a < TH::NF; ++a) {
      *reinterpret_cast<float4*>(A.copy_phi + a * A.G.N + g) = *reinterpret_cast<const float4*>(t + a * TS::PLANE);
      *reinterpret_cast<float4*>(A.copy_vel + a * A.G.N + g) =
          *reinterpret_cast<const float4*>(t + (TH::NF + a) * TS::PLANE);
    }
  }
}

// The same after plain staging in FP32: phi from the staged tile, V once more from global memory (copied on
// the way as in FP64, the staging loop of every step was 2% slower).
template <class TH, typename R, int TX, int TY, int NT>
__device__ __noinline__ void copy_tile_plain(const StepArgs<R>& A, const R* D0, int x0, int y0) {
  using TS = TileShape<TX, TY, NT>;
  for (int i = threadIdx.x; i < TX * TY; i += NT) {
    const int lx = i / TY, c = i % TY, gx = x0 + lx, gy = y0 + c;
    if (gx >= A.G.X || gy >= A.G.Y) continue;
    const long long g = (long long)gx * A.G.Y + gy;
#pragma unroll
    for (int a = 0; a < TH::NF; ++a) {
      A.copy_phi[a * A.G.N + g] = D0[a * TS::PLANE + (lx + 2) * TS::HY + TS::YOFF + c];
      A.copy_vel[a * A.G.N + g] = A.vel[a * A.G.N + g];
    }
  }
}

// Expect and issue the TMA loads of one tile (one thread, barrier initialised).  Phase B
// leaves V and l2 out of an arrested step, phase A leaves V out of a predicted one; phi and l1
// are issued before the flag is read.
template <class TH, typename R, int TX, int TY, int NT, int PH>
__device__ __forceinline__ void issue_step_tile(R* B0, const CUtensorMap* tm_phi, const CUtensorMap* tm_vel,
                                                const CUtensorMap* tm_l1, const CUtensorMap* tm_l2, int x0, int y0,
                                                uint64_t* bar, const StepState* st, unsigned tx_extra, int predict) {
  using TS = TileShape<TX, TY, NT>;
  constexpr int BUF = TH::NF * TS::PLANE;
  constexpr uint32_t bytes = (uint32_t)(sizeof(R) * BUF);
  const int c0 = y0 - TS::YOFF, c1 = x0 - 2;
  tma_load_3d(B0, tm_phi, c0, c1, 0, bar);
  if constexpr (PH == PH_E) {
    mbar_expect_tx(bar, bytes + tx_extra);
  } else if constexpr (PH == PH_A) {
    const bool skip = predict && __ldcg(&st->streak) >= 2;
    if (!skip) tma_load_3d(B0 + BUF, tm_vel, c0, c1, 0, bar);
    mbar_expect_tx(bar, (skip ? 1 : 2) * bytes + tx_extra);
  } else {
    tma_load_3d(B0 + 2 * BUF, tm_l1, c0, c1, 0, bar);
    const bool arrest = __ldcg(&st->arrest) != 0;
    if (!arrest) {
      tma_load_3d(B0 + BUF, tm_vel, c0, c1, 0, bar);
      tma_load_3d(B0 + 3 * BUF, tm_l2, c0, c1, 0, bar);
    }
    mbar_expect_tx(bar, (arrest ? 2 : 4) * bytes + tx_extra);
  }
}

// The reductions that close a phase: the tile's energy partial (A, E; stored by the caller's own
// loop over tiles where nblk CTAs walk more: ntiles) or err (B); the last CTA of the lattice sums
// the partials in a fixed order, updates the arrest state and writes the trajectory slots.
template <int NT, typename R, int PH>
__device__ __forceinline__ void step_reductions(const StepArgs<R>& A, StageShared<NT>& S, double e_acc, double err_max,
                                                int tile, int nblk, int ntiles = 0) {
  StepState* st = A.st;
  if (PH != PH_B && !A.with_energy) return;
  if constexpr (PH == PH_B) {
    const double bm = block_max<NT>(err_max, S.red);
    if (threadIdx.x == 0 && bm > -INFINITY) atomicMax(&st->err_enc, enc_max(bm));
  } else if (!ntiles) {
    const double bs = block_sum_fixed<NT>(e_acc, S.red);
    if (threadIdx.x == 0) A.partial[tile] = bs;
  }
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned t = atomicAdd(&st->ticket, 1u);
    S.am_last = (t == (unsigned)nblk - 1u);
  }
  __syncthreads();
  if (!S.am_last) return;
  __threadfence();
  if constexpr (PH == PH_B) {
    if (threadIdx.x == 0) {
      const double err = dec_max(atomicExch(&st->err_enc, 0ULL));
      if (A.err_traj && A.err_idx >= 0) A.err_traj[A.err_idx] = err;
    }
  } else {
    const double E = fixed_order_sum<NT>(A.partial, ntiles ? ntiles : nblk, S.sh_s, S.sh_c);
    if (threadIdx.x == 0) {
      st->scalar = E;
      if (!isfinite(E)) raise_status(st, ST_NONFINITE);
      if (A.E_traj && A.E_idx >= 0) A.E_traj[A.E_idx] = E;
      if (A.arrest_update) {
        const int arrest = (A.G.killkinen && E > st->E_last) ? 1 : 0;
        st->arrest = arrest;
        st->E_last = E;
        st->l2_missing = PH == PH_A && A.predict && st->streak >= 2 && !arrest;
        st->streak = arrest ? min(st->streak + 1, 2) : 0;
      }
    }
  }
  if (threadIdx.x == 0) st->ticket = 0u;
}

// T2 in place of V (A), or T3 in place of l1 and T4 in place of l2 (B: the raw l1 and l2 of
// the thread's own pairs go to C first), in a tile's TMA-staged buffers at B0.
template <class TH, typename R, int TX, int TY, int NT, int PH, class CL>
__device__ __forceinline__ void combine_tile(const Grid& G, R* B0, bool arrest, CL& C) {
  using TS = TileShape<TX, TY, NT>;
  using V = typename PairOf<R>::type;
  constexpr int NF = TH::NF, BUF = NF * TS::PLANE;
  constexpr int PAIRS = TY / 2, RPP = NT / PAIRS, PASSES = TX / RPP;
  R* B1 = B0 + BUF;
  const V half(0.5), hdt(grid_k<R>(G, GK_HDT)), dtv(grid_k<R>(G, GK_DT));
  if constexpr (PH == PH_A) {
    if (arrest) return;  // phase A: no l2 wanted
    for (int i = 4 * threadIdx.x; i < BUF; i += 4 * NT) {
      V p0, p1, v0, v1;
      ld_quad(B0 + i, p0, p1);
      ld_quad(B1 + i, v0, v1);
      st_quad(B1 + i, vfma(hdt, v0, p0), vfma(hdt, v1, p1));
    }
    __syncthreads();
  } else if constexpr (PH == PH_B) {
    R* B2 = B1 + BUF;
    R* B3 = B2 + BUF;
    const int j = threadIdx.x % PAIRS, lxg = threadIdx.x / PAIRS;
#pragma unroll
    for (int pass = 0; pass < PASSES; ++pass) {
      const int toff = (lxg * PASSES + pass + 2) * TS::HY + TS::YOFF + 2 * j;
#pragma unroll
      for (int a = 0; a < NF; ++a) {
        C.l1[pass][a] = ld_pair(B2 + a * TS::PLANE + toff);
        C.l2[pass][a] = arrest ? C.l1[pass][a] : ld_pair(B3 + a * TS::PLANE + toff);
      }
    }
    __syncthreads();
    if (arrest) {  // V = 0, l2 = l1
      for (int i = 4 * threadIdx.x; i < BUF; i += 4 * NT) {
        V p0, p1, w0, w1;
        ld_quad(B0 + i, p0, p1);
        ld_quad(B2 + i, w0, w1);
        w0 = vfma(half, w0, V(0.0));
        w1 = vfma(half, w1, V(0.0));
        st_quad(B2 + i, vfma(hdt, w0, p0), vfma(hdt, w1, p1));
        st_quad(B3 + i, vfma(dtv, w0, p0), vfma(dtv, w1, p1));
      }
    } else {
      for (int i = 4 * threadIdx.x; i < BUF; i += 4 * NT) {
        V p0, p1, v0, v1, w0, w1, u0, u1;
        ld_quad(B0 + i, p0, p1);
        ld_quad(B1 + i, v0, v1);
        ld_quad(B2 + i, w0, w1);
        ld_quad(B3 + i, u0, u1);
        st_quad(B2 + i, vfma(hdt, vfma(half, w0, v0), p0), vfma(hdt, vfma(half, w1, v1), p1));
        st_quad(B3 + i, vfma(dtv, vfma(half, u0, v0), p0), vfma(dtv, vfma(half, u1, v1), p1));
      }
    }
    __syncthreads();
  }
}

// The stencils of a staged (and combined) tile.  `arrest`: phase B's arrest, phase A's skip.
template <class TH, typename R, int TX, int TY, int NT, bool TMA, int PH, class CL>
__device__ __forceinline__ void compute_tile(const StepArgs<R>& A, const R* B0, const CL& C, int x0, int y0,
                                             bool arrest, double& e_acc, double& err_max) {
  constexpr int BUF = TH::NF * TileShape<TX, TY, NT>::PLANE;
  const Grid& G = A.G;
  const bool fast = G.pairs && x0 >= G.halo + 1 && x0 + TX - 1 <= G.X - G.halo - 2 && y0 >= G.halo + 1 &&
                    y0 + TY - 1 <= G.Y - G.halo - 2;
  if constexpr (PH == PH_B) {
    const R* T3 = TMA ? B0 + 2 * BUF : B0;
    if (fast)
      second_half<TH, R, TX, TY, NT, TMA, true>(A, T3, T3 + BUF, B0, B0 + BUF, C, x0, y0, arrest, err_max);
    else
      second_half<TH, R, TX, TY, NT, TMA, false>(A, T3, T3 + BUF, B0, B0 + BUF, C, x0, y0, arrest, err_max);
  } else {
    double* ep = A.with_energy ? &e_acc : nullptr;
    if (fast)
      first_half<TH, R, TX, TY, NT, true, PH>(A, B0, B0 + BUF, x0, y0, arrest, ep);
    else
      first_half<TH, R, TX, TY, NT, false, PH>(A, B0, B0 + BUF, x0, y0, arrest, ep);
  }
}

template <typename R>
__device__ __forceinline__ void step_init(const StepArgs<R>& A, int cta) {
  if (A.init_state && cta == 0 && threadIdx.x == 0) {
    A.st->arrest = 0;
    A.st->l2_missing = 0;
    if (!isnan(A.prev_energy)) A.st->E_last = A.prev_energy;
  }
}

// Stage, compute and reduce tile `tile` of a lattice of `nblk` tiles.  issued: thread 0 has
// already initialised S.bar and issued the tile's loads.
template <class TH, typename R, int TX, int TY, int NT, bool TMA, int PH>
__device__ __forceinline__ void step_tile(const StepArgs<R>& A, const CUtensorMap* tm_phi, const CUtensorMap* tm_vel,
                                          const CUtensorMap* tm_l1, const CUtensorMap* tm_l2, int tile, int nblk,
                                          unsigned char* smem_raw, StageShared<NT>& S, bool issued = false) {
  using V = typename PairOf<R>::type;
  constexpr int NF = TH::NF, BUF = NF * TileShape<TX, TY, NT>::PLANE;
  constexpr int PASSES = TX / (NT / (TY / 2));
  R* B0 = reinterpret_cast<R*>(smem_raw);
  const int tiles_y = (A.G.Y + TY - 1) / TY;
  const int x0 = (tile / tiles_y) * TX;
  const int y0 = (tile % tiles_y) * TY;
  bool arrest = false;
  CentreL<V, (PH == PH_B && TMA) ? NF : 1, (PH == PH_B && TMA) ? PASSES : 1> C;
  step_init(A, tile);
  if constexpr (TMA) {
    if (!issued) {
      if (threadIdx.x == 0) {
        mbar_init(&S.bar, 1);
        issue_step_tile<TH, R, TX, TY, NT, PH>(B0, tm_phi, tm_vel, tm_l1, tm_l2, x0, y0, &S.bar, A.st, A.tx_extra,
                                               A.predict);
      }
      __syncthreads();
    }
    if constexpr (PH == PH_B) arrest = __ldcg(&A.st->arrest) != 0;
    if constexpr (PH == PH_A) arrest = A.predict && __ldcg(&A.st->streak) >= 2;
    const bool ok = __syncthreads_and(mbar_wait_bounded(&S.bar, 0, A.wait_cycles));
    if (!ok) {
      if (threadIdx.x == 0) raise_status(A.st, ST_TIMEOUT);
      mbar_wait_bounded(&S.bar, 0, A.wait_cycles);
      return;
    }
    if constexpr (PH == PH_A) {
      if (A.copy_phi) {
        copy_tile<TH, R, TX, TY, NT>(A, B0, x0, y0);
        __syncthreads();  // V is combined in place next
      }
    }
    combine_tile<TH, R, TX, TY, NT, PH>(A.G, B0, arrest, C);
  } else {
    if constexpr (PH == PH_B) arrest = __ldcg(&A.st->arrest) != 0;
    stage_step_plain<NF, R, TX, TY, NT, PH>(B0, B0 + BUF, A, x0, y0, arrest);
    __syncthreads();
    if constexpr (PH == PH_A) {
      if constexpr (sizeof(R) == 4) {
        if (A.copy_phi) copy_tile_plain<TH, R, TX, TY, NT>(A, B0, x0, y0);
      }
      arrest = A.predict && __ldcg(&A.st->streak) >= 2;
    }
  }
  double e_acc = 0.0, err_max = -INFINITY;
  compute_tile<TH, R, TX, TY, NT, TMA, PH>(A, B0, C, x0, y0, arrest, e_acc, err_max);
  step_reductions<NT, R, PH>(A, S, e_acc, err_max, tile, nblk);
}

// Persistent phase B (TMA staging): the resident CTAs walk the tiles b, b + gridDim.x, ...
// through one staged tile each, so that a CTA's set-up is paid once and its SM's other CTAs
// compute while it waits for a tile.  us, one tile per CTA -> persistent: 4096^2 chiral magnet
// FP32 441 -> 361 (HBM floor 246; 46% issue, waits on loads at 16 warps per SM), 2048^2 baby Skyrme FP32 118 -> 95, 1024^2
// Abelian Higgs FP64 79 -> 66, 1024^2 s+id FP32 64 -> 53.  A ring of two tiles under one
// 512-thread CTA per SM took 391 us (chiral), 112 us (baby Skyrme).  Phase A gains nothing
// (four CTAs per SM already hide its waits: 241 against 244 us) and stays one tile per CTA.
template <class TH, typename R>
struct PipeShape : StepShape<TH, R, PH_B> {
  using SH = StepShape<TH, R, PH_B>;
  static constexpr size_t SMEM = 4 * tile_buf_bytes<R, TH::NF, SH::TX, SH::TY>();
};

template <class TH, typename R>
__global__ void __launch_bounds__((PipeShape<TH, R>::NT), (PipeShape<TH, R>::CTAS))
    step_kernel_pipe(const __grid_constant__ StepMaps M, const __grid_constant__ StepArgs<R> A) {
  using SH = PipeShape<TH, R>;
  using V = typename PairOf<R>::type;
  constexpr int TX = SH::TX, TY = SH::TY, NT = SH::NT, NF = TH::NF;
  using TS = TileShape<TX, TY, NT>;
  constexpr int BUF = NF * TS::PLANE;
  constexpr int PASSES = TX / (NT / (TY / 2));
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* B0 = reinterpret_cast<R*>(smem_raw);
  __shared__ StageShared<NT> S;
  const Grid& G = A.G;
  const int tiles_y = (G.Y + TY - 1) / TY;
  const int ntiles = ((G.X + TX - 1) / TX) * tiles_y;
  const bool arrest = __ldcg(&A.st->arrest) != 0;
  constexpr uint32_t bytes = (uint32_t)(sizeof(R) * BUF);
  const uint32_t tx = bytes * (arrest ? 2 : 4) + A.tx_extra;
  auto issue = [&](int tile) {
    const int c0 = (tile % tiles_y) * TY - TS::YOFF, c1 = (tile / tiles_y) * TX - 2;
    mbar_expect_tx(&S.bar, tx);
    tma_load_3d(B0, &M.phi, c0, c1, 0, &S.bar);
    tma_load_3d(B0 + 2 * BUF, &M.l1, c0, c1, 0, &S.bar);
    if (!arrest) {
      tma_load_3d(B0 + BUF, &M.vel, c0, c1, 0, &S.bar);
      tma_load_3d(B0 + 3 * BUF, &M.l2, c0, c1, 0, &S.bar);
    }
  };
  if (threadIdx.x == 0) {
    mbar_init(&S.bar, 1);
    if (blockIdx.x < ntiles) issue(blockIdx.x);
  }
  __syncthreads();
  double e_acc = 0.0, err_max = -INFINITY;
  const int dq = gridDim.x / tiles_y, dr = gridDim.x % tiles_y;
  int tx_i = blockIdx.x / tiles_y, ty_i = blockIdx.x % tiles_y;
  uint32_t parity = 0;
#pragma unroll 1
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const bool ok = __syncthreads_and(mbar_wait_bounded(&S.bar, parity, A.wait_cycles));
    if (!ok) {  // record, then wait (bounded) for the loads still in flight before leaving
      if (threadIdx.x == 0) raise_status(A.st, ST_TIMEOUT);
      mbar_wait_bounded(&S.bar, parity, A.wait_cycles);
      return;
    }
    CentreL<V, NF, PASSES> C;
    combine_tile<TH, R, TX, TY, NT, PH_B>(G, B0, arrest, C);
    compute_tile<TH, R, TX, TY, NT, true, PH_B>(A, B0, C, tx_i * TX, ty_i * TY, arrest, e_acc, err_max);
    // order this tile's in-place writes before the next bulk copies into its buffers
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // every thread is done with them
    if (threadIdx.x == 0 && t + (int)gridDim.x < ntiles) issue(t + gridDim.x);
    tx_i += dq;
    ty_i += dr;
    if (ty_i >= tiles_y) {
      ty_i -= tiles_y;
      ++tx_i;
    }
    parity ^= 1;
  }
  step_reductions<NT, R, PH_B>(A, S, e_acc, err_max, blockIdx.x, gridDim.x);
}

// Persistent phase E (TMA staging): the resident CTAs walk the tiles through a ring of staged
// tiles, the next ones' loads in flight behind the current one's stencil.  Tiles, their partials
// and the order of their sum are those of one tile per CTA: the same energy to the last bit.
template <class TH, typename R>
struct EnergyPipe : StepShape<TH, R, PH_E> {
  using SH = StepShape<TH, R, PH_E>;
  static constexpr size_t SLOT = tile_buf_bytes<R, TH::NF, SH::TX, SH::TY>();
  static constexpr int FIT = (int)(216 * 1024 / SH::CTAS / SLOT), SLOTS = FIT > 4 ? 4 : FIT;
  static_assert(SLOTS >= 2, "a load in flight behind the stencil");
};
template <class TH, typename R>
__global__ void __launch_bounds__((EnergyPipe<TH, R>::NT), (EnergyPipe<TH, R>::CTAS))
    step_energy_pipe(const __grid_constant__ CUtensorMap map, const __grid_constant__ StepArgs<R> A) {
  using SH = EnergyPipe<TH, R>;
  constexpr int TX = SH::TX, TY = SH::TY, NT = SH::NT, SLOTS = SH::SLOTS;
  using TS = TileShape<TX, TY, NT>;
  constexpr int BUF = TH::NF * TS::PLANE;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* ring = reinterpret_cast<R*>(smem_raw);
  __shared__ StageShared<NT> S;
  __shared__ __align__(8) uint64_t full[SLOTS];
  const Grid& G = A.G;
  const int tiles_y = (G.Y + TY - 1) / TY;
  const int ntiles = ((G.X + TX - 1) / TX) * tiles_y;
  auto issue = [&](int slot, int tile) {
    mbar_expect_tx(&full[slot], (uint32_t)(sizeof(R) * BUF) + A.tx_extra);
    tma_load_3d(ring + slot * BUF, &map, (tile % tiles_y) * TY - TS::YOFF, (tile / tiles_y) * TX - 2, 0, &full[slot]);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < SLOTS; ++s) mbar_init(&full[s], 1);
    for (int s = 0; s < SLOTS; ++s) {
      const int t = blockIdx.x + s * gridDim.x;
      if (t < ntiles) issue(s, t);
    }
  }
  __syncthreads();
  const int dq = gridDim.x / tiles_y, dr = gridDim.x % tiles_y;
  int tx_i = blockIdx.x / tiles_y, ty_i = blockIdx.x % tiles_y;
  int slot = 0;
  uint32_t parity = 0;
#pragma unroll 1
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const bool ok = __syncthreads_and(mbar_wait_bounded(&full[slot], parity, A.wait_cycles));
    if (!ok) {  // record, then wait (bounded) for every load still in flight before leaving
      if (threadIdx.x == 0) raise_status(A.st, ST_TIMEOUT);
      for (int s = 0; s < SLOTS && t + s * (int)gridDim.x < ntiles; ++s) {
        mbar_wait_bounded(&full[slot], parity, A.wait_cycles);
        if (++slot == SLOTS) {
          slot = 0;
          parity ^= 1;
        }
      }
      return;
    }
    double e_acc = 0.0, err_max = 0.0;
    CentreL<typename PairOf<R>::type, 1, 1> none;
    compute_tile<TH, R, TX, TY, NT, true, PH_E>(A, ring + slot * BUF, none, tx_i * TX, ty_i * TY, false, e_acc, err_max);
    const double bs = block_sum_fixed<NT>(e_acc, S.red);  // its barriers: every thread is done with this slot
    if (threadIdx.x == 0) {
      A.partial[t] = bs;
      const int nt = t + SLOTS * gridDim.x;
      if (nt < ntiles) issue(slot, nt);
    }
    tx_i += dq;
    ty_i += dr;
    if (ty_i >= tiles_y) {
      ty_i -= tiles_y;
      ++tx_i;
    }
    if (++slot == SLOTS) {
      slot = 0;
      parity ^= 1;
    }
  }
  step_reductions<NT, R, PH_E>(A, S, 0.0, 0.0, blockIdx.x, gridDim.x, ntiles);
}

template <class TH, typename R, bool TMA, int PH>
__global__ void __launch_bounds__((StepShape<TH, R, PH, TMA>::NT), (StepShape<TH, R, PH, TMA>::CTAS))
    step_kernel(const __grid_constant__ StepMaps M, const __grid_constant__ StepArgs<R> A) {
  using SH = StepShape<TH, R, PH, TMA>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ StageShared<SH::NT> S;
  step_tile<TH, R, SH::TX, SH::TY, SH::NT, TMA, PH>(A, &M.phi, &M.vel, &M.l1, &M.l2, blockIdx.x, gridDim.x,
                                                    smem_raw, S);
}

// Phase A2: l2 where phase A left it out on a prediction that did not hold, else nothing.  A
// resident grid walks the tiles with plain loads (it runs once in a while, and an idle launch
// must cost no more than its CTAs' start: 28 us with one CTA per tile at 4096^2).
template <class TH, typename R, bool FUSED_T2>
__global__ void __launch_bounds__((StepShape<TH, R, PH_A, false>::NT)) step_a2_kernel(const __grid_constant__ StepArgs<R> A) {
  using SH = StepShape<TH, R, PH_A, false>;
  constexpr int TX = SH::TX, TY = SH::TY, NT = SH::NT, NF = TH::NF;
  if (__ldcg(&A.st->l2_missing) == 0) return;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* D0 = reinterpret_cast<R*>(smem_raw);
  R* D1 = D0 + NF * TileShape<TX, TY, NT>::PLANE;
  const Grid& G = A.G;
  const int tiles_y = (G.Y + TY - 1) / TY, ntiles = ((G.X + TX - 1) / TX) * tiles_y;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int x0 = (t / tiles_y) * TX, y0 = (t % tiles_y) * TY;
    stage_step_plain<NF, R, TX, TY, NT, PH_A, FUSED_T2>(D0, D1, A, x0, y0, false);
    __syncthreads();
    first_half<TH, R, TX, TY, NT, false, PH_A2>(A, D0, D1, x0, y0, false, nullptr);
    __syncthreads();
  }
}

// End of a call: a pending arrest left by the trailing energy pass (V = 0) and the call's status
// to status_out (nullable; e.g. mapped host memory).
template <typename R>
__global__ void step_finish_kernel(R* vel, long long n, const StepState* st, int* status_out) {
  if (status_out && blockIdx.x == 0 && threadIdx.x == 0) *(volatile int*)status_out = st->status;
  if (!st->arrest) return;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    vel[i] = (R)0;
}

}  // namespace ssb
