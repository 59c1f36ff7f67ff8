// coop.cuh -- n flow steps of a small lattice in one cooperative launch.
//
// A lattice whose tiles are all resident at once (one tile per CTA) advances without leaving
// the kernel: the two phases of the step (rk.cuh) are separated by grid barriers instead of
// launches.  Each CTA stages its halo tile from L2 straight into the phase's two stencil
// fields, keeps its own sites' phi, V, l1, l2 in shared memory across phases and publishes
// l1, l2 (phase A) and phi', V' (phase B) for its neighbours.  Every CTA sums the energy
// partials itself, in the same order, so the arrest decision needs no further exchange.
// What bounds a step here is latency: two barriers, two L2 round trips for the halos and two
// stencils per thread, where separate launches paid two kernel boundaries with their drained
// tails and cold starts on a handful of CTAs.
#pragma once

#include "rk.cuh"

namespace ssb {

template <typename R>
struct CoopArgs {
  R* phi[2];  // the caller's buffers and the workspace's pair
  R* vel[2];
  R* l1;
  R* l2;
  int n;            // steps
  int* status_out;  // nullable, device-visible: the call's status
};

// Grid barrier of a cooperative launch: the count only grows within a launch (by at most 4096
// CTAs x 8193 barriers, below bit 31) and the last CTA to leave resets it.  Bounded: a CTA that
// has waited `limit` clock64 cycles sets bit 31 in place of a count still below the target.  No
// CTA can have passed that barrier then, so all of them see the mark and return false (in every
// thread), here or, in launches queued behind, at the first barrier, until the host has reported
// the timeout and put the state back (idle_counters).
constexpr unsigned COOP_EXPIRED = 0x80000000u;
__device__ __forceinline__ bool coop_barrier(StepState* st, unsigned target, long long limit) {
  __syncthreads();
  bool ok = true;
  if (threadIdx.x == 0) {
    // release: the CTA's writes (ordered before by the block barrier) before the arrival
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&st->bar) : "memory");
    const long long t0 = clock64();
    unsigned seen;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(&st->bar) : "memory");
      if (seen & COOP_EXPIRED) {
        ok = false;
        break;
      }
      if (seen >= target) break;
      if (clock64() - t0 > limit && atomicCAS(&st->bar, seen, seen | COOP_EXPIRED) == seen) {
        ok = false;
        break;
      }
    }
  }
  return __syncthreads_and(ok);
}

// VW consecutive elements of one plane as loaded from L2 (other CTAs wrote them in this launch).
template <typename R, int VW>
struct CoopVec {
  R x[VW];
};
template <typename R, int VW>
__device__ __forceinline__ CoopVec<R, VW> coop_load(const R* p, bool ok) {
  CoopVec<R, VW> r;
  if constexpr (VW == 1) {
    r.x[0] = ok ? __ldcg(p) : (R)0;
  } else if constexpr (sizeof(R) == 4) {
    const float4 t = ok ? __ldcg(reinterpret_cast<const float4*>(p)) : make_float4(0.f, 0.f, 0.f, 0.f);
    r.x[0] = t.x;
    r.x[1] = t.y;
    r.x[2] = t.z;
    r.x[3] = t.w;
  } else {
    const double2 t = ok ? __ldcg(reinterpret_cast<const double2*>(p)) : make_double2(0.0, 0.0);
    r.x[0] = t.x;
    r.x[1] = t.y;
  }
  return r;
}
template <typename R, int VW>
__device__ __forceinline__ void coop_put(R* p, const CoopVec<R, VW>& v) {
  if constexpr (VW == 1) {
    p[0] = v.x[0];
  } else if constexpr (sizeof(R) == 4) {
    *reinterpret_cast<float4*>(p) = make_float4(v.x[0], v.x[1], v.x[2], v.x[3]);
  } else {
    *reinterpret_cast<double2*>(p) = make_double2(v.x[0], v.x[1]);
  }
}

// Where a thread's k-th chunk of a halo tile lies: offset into the lattice's component planes,
// and whether it lies on the lattice.
template <int NF, typename R, int TX, int TY, int NT, int VW>
struct CoopChunks {
  using TS = TileShape<TX, TY, NT>;
  static constexpr int CH = TS::PLANE / VW, TOTAL = NF * CH;  // chunks per plane and in all
  static constexpr int ALL = (TOTAL + NT - 1) / NT;
  static constexpr bool KEEP = ALL <= 8;  // computed once per launch and kept in registers
  static_assert(TS::HY % VW == 0, "chunks stay within rows");
  long long off[KEEP ? ALL : 1];
  unsigned ok = 0;
  static __device__ __forceinline__ long long at(const Grid& G, int x0, int y0, int i, bool& in) {
    const int a = i / CH, q = i - a * CH, r = (q * VW) / TS::HY, c = q * VW - r * TS::HY;
    const int gx = x0 - 2 + r, gy = y0 - TS::YOFF + c;
    in = i < TOTAL && gx >= 0 && gx < G.X && gy >= 0 && gy < G.Y;
    return (long long)a * G.N + (long long)gx * G.Y + gy;
  }
  __device__ __forceinline__ void init(const Grid& G, int x0, int y0) {
    if constexpr (KEEP) {
#pragma unroll
      for (int k = 0; k < ALL; ++k) {
        bool in;
        off[k] = at(G, x0, y0, threadIdx.x + k * NT, in);
        if (in) ok |= 1u << k;
      }
    }
  }
};

// Halo tile -> the phase's stencil fields D0, D1 (A: phi, T2; B: T3, T4; E: phi).  `between`
// runs after the first group's loads are issued (phase B: the energy sum that decides the
// arrest, whose latency the loads hide) and returns the arrest flag.
template <int NF, typename R, int TX, int TY, int NT, int PH, int VW, class F>
__device__ __forceinline__ void coop_stage(R* D0, R* D1, const CoopChunks<NF, R, TX, TY, NT, VW>& K, const Grid& G,
                                           const R* phi, const R* vel, const R* l1, const R* l2, int x0, int y0,
                                           F&& between) {
  using KC = CoopChunks<NF, R, TX, TY, NT, VW>;
  constexpr int TOTAL = KC::TOTAL, ALL = KC::ALL;
  constexpr int CAP = PH == PH_B ? 16 / (VW * (int)sizeof(R) / 4) : 24 / (VW * (int)sizeof(R) / 4);
  // groups of equal size: a short last group pays a whole L2 round trip for a few chunks (500 x 333, us
  // per step, 16 + 3 chunks -> 10 + 9: baby Skyrme 20.3 -> 18.5; 16 + 9 -> 13 + 12: chiral magnet 20.1 -> 18.6)
  constexpr int GROUPS = (ALL + CAP - 1) / CAP, U = KC::KEEP ? ALL : (ALL + GROUPS - 1) / GROUPS;  // chunks in flight
  using C = CoopVec<R, VW>;
  const R dt = (R)G.dt, half = (R)0.5, hdt = grid_k<R>(G, GK_HDT);
  bool arrest = false;
#pragma unroll 1
  for (int base = 0; base < TOTAL; base += NT * U) {
    C p[U], v[PH == PH_E ? 1 : U], w[PH == PH_B ? U : 1], u[PH == PH_B ? U : 1];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      bool ok;
      long long o;
      if constexpr (KC::KEEP) {
        ok = (K.ok >> k) & 1u;
        o = K.off[k];
      } else {
        o = KC::at(G, x0, y0, base + threadIdx.x + k * NT, ok);
      }
      p[k] = coop_load<R, VW>(phi + o, ok);
      if constexpr (PH != PH_E) v[k] = coop_load<R, VW>(vel + o, ok);
      if constexpr (PH == PH_B) {
        w[k] = coop_load<R, VW>(l1 + o, ok);
        u[k] = coop_load<R, VW>(l2 + o, ok);
      }
    }
    if (base == 0) arrest = between();
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int i = base + threadIdx.x + k * NT;
      if (i >= TOTAL) continue;
      if constexpr (PH == PH_E) {
        coop_put<R, VW>(D0 + i * VW, p[k]);
      } else {
        C t0, t1;
#pragma unroll
        for (int e = 0; e < VW; ++e) {
          const R pe = p[k].x[e];
          if constexpr (PH == PH_A) {
            t0.x[e] = pe;
            t1.x[e] = VW == 1 ? stage_t2<R>(pe, v[k].x[e], dt) : vfma(hdt, v[k].x[e], pe);
          } else {
            const R ve = arrest ? (R)0 : v[k].x[e], we = w[k].x[e], ue = arrest ? we : u[k].x[e];
            t0.x[e] = VW == 1 ? stage_t3<R>(pe, ve, we, dt) : vfma(hdt, vfma(half, we, ve), pe);
            t1.x[e] = vfma(dt, vfma(half, ue, ve), pe);
          }
        }
        coop_put<R, VW>(D0 + i * VW, t0);
        coop_put<R, VW>(D1 + i * VW, t1);
      }
    }
  }
}

// A CTA's own sites across phases: [phi, V, l1, l2, l4][component][pair].  SPLIT: two threads
// per site pair, one per stencil field of the phase (l4 passes between them).
enum { CC_PHI = 0, CC_VEL = 1, CC_L1 = 2, CC_L2 = 3, CC_L4 = 4 };
template <class TH, typename R, int TX, int TY, int NT, bool SPLIT>
struct CoopTile {
  using V = typename PairOf<R>::type;
  static constexpr int NF = TH::NF, PT = SPLIT ? NT / 2 : NT;  // pair threads
  static constexpr int PAIRS = TY / 2, RPP = PT / PAIRS, PASSES = TX / RPP, SLOTS = PASSES * PT;
  static_assert(PT % PAIRS == 0 && TX % RPP == 0 && PT % 32 == 0, "pair mapping");
  static constexpr size_t BUF = tile_buf_bytes<R, NF, TX, TY>();
  static constexpr size_t SMEM = 2 * BUF + sizeof(V) * (SPLIT ? 5 : 4) * NF * SLOTS;
  // the two stencil fields first (16-byte aligned), then the own sites
  static __device__ __forceinline__ R* cell(unsigned char* smem, int arr, int a, int pass) {
    return reinterpret_cast<R*>(smem + 2 * BUF) + 2 * ((arr * NF + a) * SLOTS + pass * PT + threadIdx.x % PT);
  }
};

// phi' and V' of a pair from its own sites and l3, l4 (core/integrator.py:151-189), re-projected
// onto the sphere, V' onto the tangent space of phi' (compute_norm_magnetization and
// project_orthogonal_magnetization, chiral_magnet/kernels.py:48-122).
template <class TH, class CT, typename V, typename R>
__device__ __forceinline__ void coop_update(const Grid& G, unsigned char* smem, int pass, bool arrest, const V* l3,
                                            const V* l4, V* Pn, V* Vn) {
  using S = typename ScalarOf<V>::type;
  const V sixth(grid_k<S>(G, GK_SIXTH)), two(2.0), dtv(grid_k<S>(G, GK_DT)), dt6(grid_k<S>(G, GK_DT6));
#pragma unroll
  for (int a = 0; a < TH::NF; ++a) {
    const V p = ld_pair(CT::cell(smem, CC_PHI, a, pass)), l1 = ld_pair(CT::cell(smem, CC_L1, a, pass));
    const V v = arrest ? V(0.0) : ld_pair(CT::cell(smem, CC_VEL, a, pass));
    const V l2 = arrest ? l1 : ld_pair(CT::cell(smem, CC_L2, a, pass));
    Vn[a] = vfma(sixth, l4[a], vfma(sixth, vfma(two, l3[a], vfma(two, l2, l1)), v));
    Pn[a] = vfma(dt6, (l1 + l2) + l3[a], vfma(dtv, v, p));
  }
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
  for (int a = 0; a < TH::NF; ++a) {
    st_pair(CT::cell(smem, CC_PHI, a, pass), Pn[a]);
    st_pair(CT::cell(smem, CC_VEL, a, pass), Vn[a]);
  }
}

// The phase's stencils of the CTA's tile (as first_half and second_half, own sites in shared
// memory).
template <class TH, typename R, int TX, int TY, int NT, bool SPLIT, bool FAST, int PH>
__device__ __forceinline__ void coop_compute(const StepArgs<R>& A, unsigned char* smem, int x0, int y0, bool arrest,
                                             R* out0, R* out1, double& e_sum, double& err_max) {
  using TS = TileShape<TX, TY, NT>;
  using CT = CoopTile<TH, R, TX, TY, NT, SPLIT>;
  using V = typename PairOf<R>::type;
  using S = typename ScalarOf<V>::type;
  constexpr int NF = TH::NF;
  const R* D0 = reinterpret_cast<const R*>(smem);
  const R* D1 = reinterpret_cast<const R*>(smem + CT::BUF);
  const Grid& G = A.G;
  const long long N = G.N;
  const PairCoef<V> kc(G);
  const V mdt(grid_k<S>(G, GK_MDT));
  const int pt = threadIdx.x % CT::PT, half = SPLIT ? threadIdx.x / CT::PT : 0;
  const int j = pt % CT::PAIRS, lxg = pt / CT::PAIRS;
  V chk(0.0);
  S emax = -INFINITY;
#pragma unroll 1
  for (int pass = 0; pass < CT::PASSES; ++pass) {
    const int lx = lxg * CT::PASSES + pass;
    const int gx = x0 + lx, gy = y0 + 2 * j;
    const bool in = FAST || (gx < G.X && gy < G.Y);
    bool v1 = true;
    Masks m0{true, true, true}, m1{true, true, true};
    if (!FAST) {
      v1 = gy + 1 < G.Y;
      m0 = site_masks(G, gx, gy);
      m1 = site_masks(G, gx, gy + 1);
      if (!v1) m1 = Masks{false, false, false};
    }
    const int toff = (lx + 2) * TS::HY + TS::YOFF + 2 * j;
    const long long sidx = (long long)gx * G.Y + gy;
    Jet<V, NF> J;
    V g[NF];
    if constexpr (PH == PH_E) {
      if (in && half == 0) {
        tile_jet<TH, V, R, TS::HY, TS::PLANE, FAST>(D0, toff, kc, m0, m1, J);
        e_sum += pair_energy<TH, V, R>(J, A.P, v1, chk);
      }
    } else if constexpr (SPLIT) {
      // one stencil per thread: the field of the thread's half
      if (in) {
        pair_gradient<TH, V, R, TS::HY, TS::PLANE, FAST>(A, half ? D1 : D0, toff, kc, m0, m1, gx, gy, sidx, v1, J, g);
        if (PH == PH_A && half == 0) e_sum += pair_energy<TH, V, R>(J, A.P, v1, chk);
        R* const out = half ? out1 : out0;
#pragma unroll
        for (int a = 0; a < NF; ++a) {
          const V l = mdt * g[a];
          if constexpr (PH == PH_A) {
            st_pair(CT::cell(smem, half ? CC_L2 : CC_L1, a, pass), l);
            gstore<V, R>(out + a * N + sidx, l, FAST, v1);
          } else if (half) {
            st_pair(CT::cell(smem, CC_L4, a, pass), l);
            emax = fmax(emax, Lanes<V>::get(g[a], 0));
            if (v1) emax = fmax(emax, Lanes<V>::get(g[a], 1));
          } else {
            g[a] = l;  // l3
          }
        }
      }
      if constexpr (PH == PH_B) {
        __syncthreads();
        if (in && !half) {
          V l4[NF], Pn[NF], Vn[NF];
#pragma unroll
          for (int a = 0; a < NF; ++a) l4[a] = ld_pair(CT::cell(smem, CC_L4, a, pass));
          coop_update<TH, CT, V, R>(G, smem, pass, arrest, g, l4, Pn, Vn);
#pragma unroll
          for (int a = 0; a < NF; ++a) {
            gstore<V, R>(out0 + a * N + sidx, Pn[a], FAST, v1);
            gstore<V, R>(out1 + a * N + sidx, Vn[a], FAST, v1);
          }
        }
      }
    } else if (in) {
      V l0[NF];
      pair_gradient<TH, V, R, TS::HY, TS::PLANE, FAST>(A, D0, toff, kc, m0, m1, gx, gy, sidx, v1, J, g);
      if (PH == PH_A) e_sum += pair_energy<TH, V, R>(J, A.P, v1, chk);
#pragma unroll
      for (int a = 0; a < NF; ++a) {
        l0[a] = mdt * g[a];
        if constexpr (PH == PH_A) {
          st_pair(CT::cell(smem, CC_L1, a, pass), l0[a]);
          gstore<V, R>(out0 + a * N + sidx, l0[a], FAST, v1);
        }
      }
      pair_gradient<TH, V, R, TS::HY, TS::PLANE, FAST>(A, D1, toff, kc, m0, m1, gx, gy, sidx, v1, J, g);
      if constexpr (PH == PH_A) {
#pragma unroll
        for (int a = 0; a < NF; ++a) {
          const V l = mdt * g[a];
          st_pair(CT::cell(smem, CC_L2, a, pass), l);
          gstore<V, R>(out1 + a * N + sidx, l, FAST, v1);
        }
      } else {
        V Pn[NF], Vn[NF];
#pragma unroll
        for (int a = 0; a < NF; ++a) {
          emax = fmax(emax, Lanes<V>::get(g[a], 0));
          if (v1) emax = fmax(emax, Lanes<V>::get(g[a], 1));
          g[a] = mdt * g[a];
        }
        coop_update<TH, CT, V, R>(G, smem, pass, arrest, l0, g, Pn, Vn);
#pragma unroll
        for (int a = 0; a < NF; ++a) {
          gstore<V, R>(out0 + a * N + sidx, Pn[a], FAST, v1);
          gstore<V, R>(out1 + a * N + sidx, Vn[a], FAST, v1);
        }
      }
    }
  }
  if constexpr (PH == PH_B)
    err_max = fmax(err_max, (double)emax);
  else
    e_sum = e_sum * G.dA + (double)(Lanes<V>::get(chk, 0) + Lanes<V>::get(chk, 1));
}

// CTAs per SM the kernel is built for: 128 registers per thread, 80 with one FP32 stencil per
// thread, 255 for the s+id model's FP64 stencils; no more than fit an SM's shared memory (228 KB; each
// CTA's arrays and 1 KB), which leaves the larger tiles more registers: us per step, bounded by threads
// alone -> so, FP64 chiral magnet 333 x 400 22.2 -> 20.1, baby Skyrme 21.5 -> 21.0, FP32 Higgs
// 420 x 500 16.6 -> 15.5, chiral magnet 16.9 -> 16.1, s+id 333 x 400 20.8 -> 20.3.
template <class TH, typename R, int TX, int TY, int NT, bool SPLIT>
__host__ __device__ constexpr int coop_ctas() {
  const size_t per = CoopTile<TH, R, TX, TY, NT, SPLIT>::SMEM + sizeof(StageShared<NT>) + 128 + 1024;
  const int fit = (int)(228 * 1024 / per);
  const int want = (sizeof(R) == 8 && TH::NF > 4 ? 256 : SPLIT && sizeof(R) == 4 && TH::NF <= 4 ? 768 : 512) / NT;
  return fit < want ? fit : want;
}

template <class TH, typename R, int TX, int TY, int NT, bool SPLIT, int VW>
__global__ void __launch_bounds__(NT, (coop_ctas<TH, R, TX, TY, NT, SPLIT>())) coop_step_kernel(
    const __grid_constant__ StepArgs<R> A, const __grid_constant__ CoopArgs<R> C) {
  using CT = CoopTile<TH, R, TX, TY, NT, SPLIT>;
  using V = typename PairOf<R>::type;
  constexpr int NF = TH::NF;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ StageShared<NT> S;
  __shared__ double sh_E;
  R* D0 = reinterpret_cast<R*>(smem);
  R* D1 = reinterpret_cast<R*>(smem + CT::BUF);
  const Grid& G = A.G;
  StepState* st = A.st;
  const int tiles_y = (G.Y + TY - 1) / TY;
  const int x0 = (blockIdx.x / tiles_y) * TX, y0 = (blockIdx.x % tiles_y) * TY;
  const bool fast = G.pairs && x0 >= G.halo + 1 && x0 + TX - 1 <= G.X - G.halo - 2 && y0 >= G.halo + 1 &&
                    y0 + TY - 1 <= G.Y - G.halo - 2;
  const int j = threadIdx.x % CT::PAIRS, lxg = (threadIdx.x % CT::PT) / CT::PAIRS;
  CoopChunks<NF, R, TX, TY, NT, VW> K;
  K.init(G, x0, y0);
  // own sites
  auto own = [&](auto&& f) {
    if (threadIdx.x >= CT::PT) return;
#pragma unroll 1
    for (int pass = 0; pass < CT::PASSES; ++pass) {
      const int gx = x0 + lxg * CT::PASSES + pass, gy = y0 + 2 * j;
      if (gx >= G.X || gy >= G.Y) continue;
      f(pass, (long long)gx * G.Y + gy, gy + 1 < G.Y);
    }
  };
  own([&](int pass, long long i, bool v1) {
#pragma unroll
    for (int a = 0; a < NF; ++a) {
      st_pair(CT::cell(smem, CC_PHI, a, pass), gload<V, R>(C.phi[0] + a * G.N + i, fast, v1));
      st_pair(CT::cell(smem, CC_VEL, a, pass), gload<V, R>(C.vel[0] + a * G.N + i, fast, v1));
    }
  });
  double E_last = isnan(A.prev_energy) ? __ldcg(&st->E_last) : A.prev_energy;
  unsigned bar = 0;
  int cur = 0;
  bool arrest = false, failed = false;
  auto sync_grid = [&]() {
    bar += gridDim.x;
    if (!coop_barrier(st, bar + A.tx_extra, A.wait_cycles)) {
      if (threadIdx.x == 0) {
        raise_status(st, ST_TIMEOUT);
        if (C.status_out) *(volatile int*)C.status_out = (int)ST_TIMEOUT;
      }
      failed = true;
    }
    return !failed;
  };
  // every CTA: the sum of all partials in the same order, the trajectory slot, the arrest test
  auto take_energy = [&](int slot) {
    const double E = fixed_order_sum<NT>(A.partial, gridDim.x, S.sh_s, S.sh_c);
    if (threadIdx.x == 0) sh_E = E;
    __syncthreads();
    const double En = sh_E;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      if (!isfinite(En)) raise_status(st, ST_NONFINITE);
      if (A.E_traj) A.E_traj[slot] = En;
      st->scalar = En;
    }
    const bool ar = G.killkinen && En > E_last;
    E_last = En;
    return ar;
  };
  // err of step s: its B phase's maximum, complete after the barrier that follows
  auto take_err = [&](int s) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      const double err = dec_max(atomicExch(&st->err2[s & 1], 0ULL));
      if (A.err_traj) A.err_traj[s] = err;
    }
  };
#pragma unroll 1
  for (int s = 0; s < C.n; ++s) {
    double e_sum = 0.0, err_max = -INFINITY;
    // ---- phase A
    coop_stage<NF, R, TX, TY, NT, PH_A, VW>(D0, D1, K, G, C.phi[cur], C.vel[cur], C.l1, C.l2, x0, y0, [&]() { return false; });
    __syncthreads();
    if (fast)
      coop_compute<TH, R, TX, TY, NT, SPLIT, true, PH_A>(A, smem, x0, y0, false, C.l1, C.l2, e_sum, err_max);
    else
      coop_compute<TH, R, TX, TY, NT, SPLIT, false, PH_A>(A, smem, x0, y0, false, C.l1, C.l2, e_sum, err_max);
    if (s > 0) {
      const double bs = block_sum_fixed<NT>(e_sum, S.red);
      if (threadIdx.x == 0) A.partial[blockIdx.x] = bs;
    }
    if (!sync_grid()) return;
    if (s > 0) take_err(s - 1);
    // ---- phase B
    coop_stage<NF, R, TX, TY, NT, PH_B, VW>(D0, D1, K, G, C.phi[cur], C.vel[cur], C.l1, C.l2, x0, y0, [&]() {
      arrest = s > 0 ? take_energy(s - 1) : false;
      return arrest;
    });
    __syncthreads();
    if (fast)
      coop_compute<TH, R, TX, TY, NT, SPLIT, true, PH_B>(A, smem, x0, y0, arrest, C.phi[cur ^ 1], C.vel[cur ^ 1], e_sum, err_max);
    else
      coop_compute<TH, R, TX, TY, NT, SPLIT, false, PH_B>(A, smem, x0, y0, arrest, C.phi[cur ^ 1], C.vel[cur ^ 1], e_sum, err_max);
    const double bm = block_max<NT>(err_max, S.red);
    if (threadIdx.x == 0 && bm > -INFINITY) atomicMax(&st->err2[s & 1], enc_max(bm));
    cur ^= 1;
    if (!sync_grid()) return;
  }
  // ---- energy of the final field, its arrest test, and the caller's buffers
  take_err(C.n - 1);
  {
    double e_sum = 0.0, err_max = 0.0;
    coop_stage<NF, R, TX, TY, NT, PH_E, VW>(D0, D1, K, G, C.phi[cur], C.vel[cur], C.l1, C.l2, x0, y0, [&]() { return false; });
    __syncthreads();
    if (fast)
      coop_compute<TH, R, TX, TY, NT, SPLIT, true, PH_E>(A, smem, x0, y0, false, nullptr, nullptr, e_sum, err_max);
    else
      coop_compute<TH, R, TX, TY, NT, SPLIT, false, PH_E>(A, smem, x0, y0, false, nullptr, nullptr, e_sum, err_max);
    const double bs = block_sum_fixed<NT>(e_sum, S.red);
    if (threadIdx.x == 0) A.partial[blockIdx.x] = bs;
  }
  if (!sync_grid()) return;
  arrest = take_energy(C.n - 1);
  if (cur || arrest)
    own([&](int pass, long long i, bool v1) {
#pragma unroll
      for (int a = 0; a < NF; ++a) {
        if (cur) gstore<V, R>(C.phi[0] + a * G.N + i, ld_pair(CT::cell(smem, CC_PHI, a, pass)), fast, v1);
        gstore<V, R>(C.vel[0] + a * G.N + i, arrest ? V(0.0) : ld_pair(CT::cell(smem, CC_VEL, a, pass)), fast, v1);
      }
    });
  if (threadIdx.x == 0) {
    if (blockIdx.x == 0) {
      st->E_last = E_last;
      st->arrest = 0;  // applied above
      __threadfence();
      if (C.status_out) *(volatile int*)C.status_out = __ldcg(&st->status);
    }
    // the last CTA to leave resets the barrier for the next launch
    if (atomicAdd(&st->leave, 1u) == gridDim.x - 1) {
      st->leave = 0u;
      st->bar = 0u;
    }
  }
}

}  // namespace ssb
