// flow.cuh -- tiles, stencils and single-pass kernels over a lattice: the gradient hook, the
// exact FP64 energy of the stored values, densities, charges and coupling partials, and the
// reference's RK4 building blocks.  The flow's own step is in rk.cuh, on the same tiles.
#pragma once

#include <cuda.h>

#include "common.cuh"
#include "pair.cuh"
#include "theories.cuh"

namespace ssb {

// Indices of the staging variants: M_GRAD the gradient hook, M_S1, M_S2 the step's phase A,
// M_S3, M_S4 its phase B; M_ENERGY and M_S23 are kept for the pinning interface.
enum FlowMode { M_GRAD = 0, M_S1 = 1, M_S2 = 2, M_S3 = 3, M_S4 = 4, M_ENERGY = 5, M_S23 = 6 };
constexpr int N_FLOW_MODES = 7;
enum { ST_NONFINITE = 3, ST_TIMEOUT = 6 };

// Default bound of a device-side wait on an mbarrier (~1 s at 1.9 GHz).  On expiry
// the kernel records ST_TIMEOUT, waits the same bound again for its copies in
// flight and returns without computing.
constexpr long long WAIT_CYCLES = 2000000000LL;

template <typename R>
struct FlowArgs {
  CUtensorMap tm_phi;  // TMA map of the field (used when the kernel is instantiated with TMA)
  const R* phi;        // the staged field
  R* out_l;            // M_GRAD: l_out (nullable)
  R* out_eg;           // M_GRAD: energy gradient (nullable)
  StepState* st;
  const double* scale;    // grad_raw: rows times *scale * dA, rounded to R (nullable: unscaled)
  int grad_raw;           // M_GRAD: unprojected, not halo-zeroed dE/dphi with true saddle rows
  long long wait_cycles;  // bound of every mbarrier wait (clock64 cycles)
  unsigned tx_extra;      // test hook: bytes the barrier expects beyond what is loaded (normally 0)
  Grid G;
  Phys P;
};

// Tile of TX x TY sites.  Staged planes hold rows x0-2 .. x0+TX+1 and columns
// y0-4 .. y0+TY+3: the y start is rounded down to a 16-byte boundary so the same
// geometry serves TMA boxes and plain loads; the stencil uses columns 2 .. TY+5.
template <int TX, int TY, int NT>
struct TileShape {
  static constexpr int HX = TX + 4, HY = TY + 8, YOFF = 4;
  static constexpr int PLANE = HX * HY;
  static constexpr int ROWS_PER_PASS = NT / TY;
  static constexpr int SITES_PER_THREAD = TX / ROWS_PER_PASS;
  static_assert(NT % TY == 0 && TX % (NT / TY) == 0, "tile/thread mismatch");
  static_assert(TY % 4 == 0, "TY must keep the y start 16-byte aligned");
};

template <typename R, int NF, int TX, int TY>
__host__ __device__ constexpr size_t tile_buf_bytes() {
  return sizeof(R) * NF * (TX + 4) * (TY + 8);
}

// ---------------------------------------------------------------------------
// TMA / mbarrier helpers (inline PTX, sm_90+ instructions, used on sm_100a)
// ---------------------------------------------------------------------------
__device__ inline uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ inline void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ inline void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// try_wait with a suspend-time hint: the thread sleeps until the phase completes or
// ~1 ms passes instead of spinning, so waiting warps take no issue slots from the
// warps that compute.
__device__ inline bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity), "r"(1000000u)
      : "memory");
  return ok != 0;
}
// 3-D tiled bulk tensor load global -> shared (no multicast), completion on `bar`.
__device__ inline void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
      ::"r"(smem_u32(dst)), "l"((uint64_t)map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}
// Bounded wait; returns false when `limit` clock64 cycles elapsed first.
__device__ inline bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, long long limit) {
  const long long t0 = clock64();
  while (!mbar_try_wait(bar, parity)) {
    if (clock64() - t0 > limit) return false;
  }
  return true;
}

// T2 = phi + k1/2 and T3 = phi + k2/2 of one element, rounded as the reference's k / Temp
// algebra (core/integrator.py:51-96 and :323-334): used by plain-load staging
template <typename R>
__device__ inline R stage_t2(R p, R v, R dt) {
  return p + (R)0.5 * (dt * v);
}
template <typename R>
__device__ inline R stage_t3(R p, R v, R l1, R dt) {
  const R half = (R)0.5;
  return p + half * (dt * (v + half * l1));
}

// Plain-load staging of one field's halo buffer (all components), used when a TMA map cannot
// describe the buffer (row pitch not a multiple of 16 bytes).  Every thread first issues all
// loads of one component plane, then stores, so each plane costs one memory round trip.
template <int NF, typename R, int TX, int TY, int NT>
__device__ inline void stage_plain(R* T, const Grid& G, const R* src, int x0, int y0) {
  using TS = TileShape<TX, TY, NT>;
  constexpr int KM = (TS::PLANE + NT - 1) / NT;
  const long long N = G.N;
  long long off[KM];
  bool ok[KM];
#pragma unroll
  for (int k = 0; k < KM; ++k) {
    const int i = threadIdx.x + k * NT;
    const int r = i / TS::HY, c = i - r * TS::HY;
    const int gx = x0 - 2 + r, gy = y0 - TS::YOFF + c;
    ok[k] = i < TS::PLANE && gx >= 0 && gx < G.X && gy >= 0 && gy < G.Y;
    off[k] = (long long)gx * G.Y + gy;
  }
#pragma unroll
  for (int a = 0; a < NF; ++a) {
    R p[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) p[k] = ok[k] ? src[(long long)a * N + off[k]] : (R)0;
#pragma unroll
    for (int k = 0; k < KM; ++k) {
      const int i = threadIdx.x + k * NT;
      if (i < TS::PLANE) T[a * TS::PLANE + i] = p[k];
    }
  }
}

// The unit-norm re-projection of a site pair's magnetisation components
// (compute_norm_magnetization, chiral_magnet/kernels.py:48-84): m / |m| where |m| > 0.
template <int NMAG, typename V>
__device__ __forceinline__ void unit_project(V* m) {
  using S = typename ScalarOf<V>::type;
  V s2 = m[0] * m[0];
#pragma unroll
  for (int a = 1; a < NMAG; ++a) s2 = vfma(m[a], m[a], s2);
  V inv(1.0);
#pragma unroll
  for (int l = 0; l < 2; ++l) {
    const S s = sqrt(Lanes<V>::get(s2, l));
    if (s != (S)0) Lanes<V>::set(inv, l, (S)1 / s);
  }
#pragma unroll
  for (int a = 0; a < NMAG; ++a) m[a] = m[a] * inv;
}

// Stencil weights pre-scaled by the lattice spacings, as broadcast pairs.
template <typename V>
struct PairCoef {
  using S = typename ScalarOf<V>::type;
  V c23hx, mc12hx, c43hx2, mc12hx2, c23hy, mc12hy, c43hy2, mc12hy2, c43hd, mc12hd;
  __device__ explicit PairCoef(const Grid& G)
      : c23hx(grid_k<S>(G, GK_C23HX)), mc12hx(grid_k<S>(G, GK_MC12HX)), c43hx2(grid_k<S>(G, GK_C43HX2)),
        mc12hx2(grid_k<S>(G, GK_MC12HX2)), c23hy(grid_k<S>(G, GK_C23HY)), mc12hy(grid_k<S>(G, GK_MC12HY)),
        c43hy2(grid_k<S>(G, GK_C43HY2)), mc12hy2(grid_k<S>(G, GK_MC12HY2)), c43hd(grid_k<S>(G, GK_C43HD)),
        mc12hd(grid_k<S>(G, GK_MC12HD)) {}
};

// Unmasked jet of one component for the site pair (x, y), (x, y+1) whose centre
// pair starts at `row` in the staged tile (rows HY apart).  Difference form as in
// d1_stencil / d2_stencil; Dx1 = f(x+1)-f(x-1), Dx2 = f(x+2)-f(x-2) and the y
// analogues are returned for the FP64 energy.
template <typename V, typename R, int HY, bool XY>
__device__ __forceinline__ void pair_jet(const R* row, const PairCoef<V>& k, V& f, V& dx, V& dy, V& dxx, V& dyy,
                                         V& dxy, V& Dx1, V& Dx2, V& Dy1, V& Dy2) {
  const V A = ld_pair(row - 2), B = ld_pair(row), C = ld_pair(row + 2);
  const V xm1 = ld_pair(row - HY), xp1 = ld_pair(row + HY);
  const V xm2 = ld_pair(row - 2 * HY), xp2 = ld_pair(row + 2 * HY);
  const V ym1 = shift1(A, B), yp1 = shift1(B, C);
  f = B;
  Dx1 = xp1 - xm1;
  Dx2 = xp2 - xm2;
  Dy1 = yp1 - ym1;
  Dy2 = C - A;
  dx = vfma(Dx1, k.c23hx, Dx2 * k.mc12hx);
  dy = vfma(Dy1, k.c23hy, Dy2 * k.mc12hy);
  dxx = vfma((xp1 - B) + (xm1 - B), k.c43hx2, ((xp2 - B) + (xm2 - B)) * k.mc12hx2);
  dyy = vfma((yp1 - B) + (ym1 - B), k.c43hy2, ((C - B) + (A - B)) * k.mc12hy2);
  if constexpr (XY) {
    // main diagonal (x+k, y+k), soliton_solver/core/derivatives.py:105-112
    const V dp1 = shift1(xp1, ld_pair(row + HY + 2));
    const V dp2 = ld_pair(row + 2 * HY + 2);
    const V dm1 = shift1(ld_pair(row - HY - 2), xm1);
    const V dm2 = ld_pair(row - 2 * HY - 2);
    const V diag = vfma((dp1 - B) + (dm1 - B), k.c43hd, ((dp2 - B) + (dm2 - B)) * k.mc12hd);
    dxy = vfma(dxx, V(-0.5), vfma(dyy, V(-0.5), diag));
  } else {
    dxy = V(0.0);
  }
}

template <typename V>
__device__ __forceinline__ V mask_lanes(V v, bool m0, bool m1) {
  using S = typename ScalarOf<V>::type;
  if (!m0) Lanes<V>::set(v, 0, (S)0);
  if (!m1) Lanes<V>::set(v, 1, (S)0);
  return v;
}

// global pair load / store; `fast` pairs are aligned and both in range
template <typename V, typename R>
__device__ __forceinline__ V gload(const R* p, bool fast, bool v1) {
  using S = typename ScalarOf<V>::type;
  if (fast) return ld_pair(p);
  V r(0.0);
  Lanes<V>::set(r, 0, (S)p[0]);
  if (v1) Lanes<V>::set(r, 1, (S)p[1]);
  return r;
}
template <typename V, typename R>
__device__ __forceinline__ void gstore(R* p, V v, bool fast, bool v1) {
  if (fast) {
    st_pair(p, v);
    return;
  }
  p[0] = Lanes<V>::get(v, 0);
  if (v1) p[1] = Lanes<V>::get(v, 1);
}

// Stored value -> FP64 for the energy stencil.  For FP32 the float's bits are placed
// in a double without re-biasing the exponent (two ALU ops and a shift instead of an
// F2F conversion, which issues on the narrow XU pipe): the result is x * 2^-896
// exactly for zero, normal and subnormal x (2^-126 * 2^-896 = 2^-1022, the smallest
// normal double).  Derivative coefficients carry the factor 2^896 back and centre
// values are multiplied by it, both exact, so every derivative and density is
// bitwise what an F2F conversion gives.  Inf/NaN map to finite values here; the
// caller folds v * 0 of every centre value into a sentinel instead.
template <typename E>
struct ScaledValue {
  static constexpr double SCALE = 1.0;
  __device__ static __forceinline__ double get(E x) { return (double)x; }
};
template <>
struct ScaledValue<float> {
  static constexpr double SCALE = 0x1p896;
  __device__ static __forceinline__ double get(float x) {
    const int u = __float_as_int(x);
    return __hiloint2double((u >> 3) & (int)0x8fffffff, u << 29);
  }
};

// FP64 energy of an FP32 site pair from the jets the gradient stencil already built
// (f, dx, dy after masking): the theory's energy point evaluated in FP64 on the
// converted jets, so phase A pays no second stencil for its energy.  The jets
// carry FP32 rounding (~1e-7 relative per site), the precision the flow's gradient
// has.  `chk` folds v * 0 of every jet value (Inf/NaN -> NaN, see ScaledValue).
template <class TH, typename V, int NF>
__device__ __forceinline__ double jet_energy(const Jet<V, NF>& J, const Phys& P, double dA, bool v1, V& chk) {
  using SV = ScaledValue<float>;
  Jet1<double, NF> J0, J1;
#pragma unroll
  for (int a = 0; a < NF; ++a) {
    chk = vfma(J.f[a], V(0.0f), chk);
    chk = vfma(J.dx[a], V(0.0f), chk);
    chk = vfma(J.dy[a], V(0.0f), chk);
    J0.f[a] = SV::get(Lanes<V>::get(J.f[a], 0)) * SV::SCALE;
    J1.f[a] = SV::get(Lanes<V>::get(J.f[a], 1)) * SV::SCALE;
    J0.dx[a] = SV::get(Lanes<V>::get(J.dx[a], 0)) * SV::SCALE;
    J1.dx[a] = SV::get(Lanes<V>::get(J.dx[a], 1)) * SV::SCALE;
    J0.dy[a] = SV::get(Lanes<V>::get(J.dy[a], 0)) * SV::SCALE;
    J1.dy[a] = SV::get(Lanes<V>::get(J.dy[a], 1)) * SV::SCALE;
  }
  double e = TH::energy(J0, P, dA);
  if (v1) e += TH::energy(J1, P, dA);
  return e;
}

// Jet of every component of the site pair whose centre starts at `toff` in the staged
// halo buffer T (NF planes of PLANE values), with the derivative masks applied.
template <class TH, typename V, typename R, int HY, int PLANE, bool FAST>
__device__ __forceinline__ void tile_jet(const R* T, int toff, const PairCoef<V>& kc, const Masks& m0, const Masks& m1,
                                         Jet<V, TH::NF>& J) {
#pragma unroll
  for (int a = 0; a < TH::NF; ++a) {
    V Dx1, Dx2, Dy1, Dy2;
    pair_jet<V, R, HY, TH::NEED_XY>(T + a * PLANE + toff, kc, J.f[a], J.dx[a], J.dy[a], J.dxx[a], J.dyy[a], J.dxy[a],
                                    Dx1, Dx2, Dy1, Dy2);
    if (!FAST) {
      J.dx[a] = mask_lanes(J.dx[a], m0.x, m1.x);
      J.dy[a] = mask_lanes(J.dy[a], m0.y, m1.y);
      J.dxx[a] = mask_lanes(J.dxx[a], m0.x, m1.x);
      J.dyy[a] = mask_lanes(J.dyy[a], m0.y, m1.y);
      J.dxy[a] = mask_lanes(J.dxy[a], m0.xy, m1.xy);
    }
  }
}

// The flow's constraints on a site pair's gradient rows: zero on the frozen ring
// (theories with HALO_ZERO) and the tangent projection g - (g . m) m
// (project_orthogonal_magnetization, chiral_magnet/kernels.py:86-122).
template <class TH, typename V, bool FAST>
__device__ __forceinline__ void flow_constraints(const Grid& G, const Jet<V, TH::NF>& J, V* g, int gx, int gy) {
  if (TH::HALO_ZERO && !FAST) {
    const bool e0 = gx < G.halo || gx > G.X - G.halo - 1 || gy < G.halo || gy > G.Y - G.halo - 1;
    const bool e1 = gx < G.halo || gx > G.X - G.halo - 1 || gy + 1 < G.halo || gy + 1 > G.Y - G.halo - 1;
#pragma unroll
    for (int a = 0; a < TH::NF; ++a) g[a] = mask_lanes(g[a], !e0, !e1);
  }
  if (TH::CONSTRAINED) {
    V lm = g[0] * J.f[0];
#pragma unroll
    for (int a = 1; a < TH::NMAG; ++a) lm = vfma(g[a], J.f[a], lm);
    const V mlm = -lm;
#pragma unroll
    for (int a = 0; a < TH::NMAG; ++a) g[a] = vfma(mlm, J.f[a], g[a]);
  }
}

// The gradient hook on one staged tile.  Each thread owns y-adjacent site pairs; FAST: the
// tile is interior (every derivative mask true, no halo site) and the output buffers hold
// aligned pairs (Grid::pairs), which need no lane masks.
template <class TH, typename R, int TX, int TY, int NT, bool FAST>
__device__ __forceinline__ void grad_tile(const FlowArgs<R>& A, const R* T, int x0, int y0) {
  using TS = TileShape<TX, TY, NT>;
  using V = typename PairOf<R>::type;
  using S = typename ScalarOf<V>::type;
  constexpr int NF = TH::NF, PAIRS = TY / 2, RPP = NT / PAIRS;
  static_assert(NT % PAIRS == 0 && TX % RPP == 0, "pair mapping");
  const Grid& G = A.G;
  const long long N = G.N;
  const PairCoef<V> kc(G);
  const V mdt(grid_k<S>(G, GK_MDT));
  const V scale(A.scale ? (S)*A.scale * (S)G.dA : (S)1);
  const int j = threadIdx.x % PAIRS;
  const int lxg = threadIdx.x / PAIRS;
#pragma unroll 1
  for (int pass = 0; pass < TX / RPP; ++pass) {
    const int lx = lxg + pass * RPP;
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
    tile_jet<TH, V, R, TS::HY, TS::PLANE, FAST>(T, toff, kc, m0, m1, J);
    V g[NF];
    TH::gradient(J, A.P, g);
    if (A.grad_raw) {
      // functional derivative of the energy: no halo zeroing, no projection, and rows the
      // flow stores scaled (saddle fields) converted to dE/dphi
      TH::true_rows(g, A.P);
      if (A.scale) {
#pragma unroll
        for (int a = 0; a < NF; ++a) g[a] = g[a] * scale;
      }
#pragma unroll
      for (int a = 0; a < NF; ++a) {
        if (A.out_eg) gstore<V, R>(A.out_eg + a * N + sidx, g[a], FAST, v1);
      }
      continue;
    }
    flow_constraints<TH, V, FAST>(G, J, g, gx, gy);
#pragma unroll
    for (int a = 0; a < NF; ++a) {
      if (A.out_eg) gstore<V, R>(A.out_eg + a * N + sidx, g[a], FAST, v1);
      if (A.out_l) gstore<V, R>(A.out_l + a * N + sidx, mdt * g[a], FAST, v1);
    }
  }
}

// Shared scratch of the tile kernels besides the staged tile.
template <int NT>
struct StageShared {
  double red[NT / 32];
  double sh_s[NT / 32], sh_c[NT / 32];
  uint64_t bar;
  int am_last;
};

template <class TH, typename R, int TX, int TY, int NT>
__device__ __forceinline__ void grad_any_tile(const FlowArgs<R>& A, const R* T, int x0, int y0) {
  const Grid& G = A.G;
  if (G.pairs && x0 >= G.halo + 1 && x0 + TX - 1 <= G.X - G.halo - 2 && y0 >= G.halo + 1 &&
      y0 + TY - 1 <= G.Y - G.halo - 2)
    grad_tile<TH, R, TX, TY, NT, true>(A, T, x0, y0);
  else
    grad_tile<TH, R, TX, TY, NT, false>(A, T, x0, y0);
}

// One halo tile of `map` (all components) into T by the CTA: TMA load, bounded wait.  Returns
// false in every thread, with the status recorded, when the wait ran out.
template <int NF, typename R, int TX, int TY, int NT>
__device__ __forceinline__ bool stage_tma(R* T, const CUtensorMap* map, uint64_t* bar, int x0, int y0, unsigned tx_extra,
                                          long long limit, StepState* st) {
  using TS = TileShape<TX, TY, NT>;
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    mbar_expect_tx(bar, (uint32_t)(sizeof(R) * NF * TS::PLANE) + tx_extra);
    tma_load_3d(T, map, y0 - TS::YOFF, x0 - 2, 0, bar);
  }
  __syncthreads();
  const bool ok = __syncthreads_and(mbar_wait_bounded(bar, 0, limit));
  if (!ok) {
    if (threadIdx.x == 0) raise_status(st, ST_TIMEOUT);
    mbar_wait_bounded(bar, 0, limit);
  }
  return ok;
}

// CTAs per SM of the gradient hook, one tile per CTA: its tiles' load latency is hidden by the other
// CTAs only.  us at 2048^2 (plain rows 1501 x 999), registers unbounded -> bounded for the CTAs below:
// FP64 chiral magnet 65 -> 56 (33 -> 31), Abelian Higgs 68 -> 56 (33 -> 29), baby Skyrme 66 -> 66 (41 ->
// 31; three CTAs 35), s+id 176 -> 115 (74 -> 64; three CTAs spill: 236); s+id FP32 69 -> 62 (37 -> 33).
// FP32 stencils of up to four components take 56 to 66 registers unbounded: four CTAs.
template <class TH, typename R>
__host__ __device__ constexpr int grad_ctas() {
  if (sizeof(R) == 4) return TH::NF > 4 ? 3 : 4;
  return TH::NF == 4 ? 3 : 2;
}

// The gradient hook, one tile per CTA.
template <class TH, typename R, int TX, int TY, int NT, bool TMA>
__global__ void __launch_bounds__(NT, (grad_ctas<TH, R>())) flow_kernel(const __grid_constant__ FlowArgs<R> A) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ uint64_t bar;
  R* T = reinterpret_cast<R*>(smem_raw);
  const int tiles_y = (A.G.Y + TY - 1) / TY;
  const int x0 = (blockIdx.x / tiles_y) * TX, y0 = (blockIdx.x % tiles_y) * TY;
  if constexpr (TMA) {
    if (!stage_tma<TH::NF, R, TX, TY, NT>(T, &A.tm_phi, &bar, x0, y0, A.tx_extra, A.wait_cycles, A.st)) return;
  } else {
    stage_plain<TH::NF, R, TX, TY, NT>(T, A.G, A.phi, x0, y0);
    __syncthreads();
  }
  grad_any_tile<TH, R, TX, TY, NT>(A, T, x0, y0);
}

// Persistent, TMA-pipelined form of flow_kernel (FP32 fields): one 512-thread CTA per SM
// walks the tiles blockIdx.x, blockIdx.x + gridDim.x, ... through a ring of STAGES
// shared-memory slots, so the bulk tensor loads of the next tiles are in flight while the
// current tile is computed.
template <class TH, typename R, int TX, int TY, int NT, int STAGES>
__global__ void __launch_bounds__(NT, 1) flow_kernel_pipe(const __grid_constant__ FlowArgs<R> A) {
  using TS = TileShape<TX, TY, NT>;
  constexpr int SLOT = TH::NF * TS::PLANE;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* ring = reinterpret_cast<R*>(smem_raw);
  __shared__ __align__(8) uint64_t full[STAGES];
  const Grid& G = A.G;
  const int tiles_y = (G.Y + TY - 1) / TY;
  const int ntiles = ((G.X + TX - 1) / TX) * tiles_y;
  constexpr uint32_t bytes = (uint32_t)(sizeof(R) * SLOT);
  auto issue = [&](int slot, int tile) {
    mbar_expect_tx(&full[slot], bytes + A.tx_extra);
    tma_load_3d(ring + slot * SLOT, &A.tm_phi, (tile % tiles_y) * TY - TS::YOFF, (tile / tiles_y) * TX - 2, 0,
                &full[slot]);
  };
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) mbar_init(&full[s], 1);
    for (int s = 0; s < STAGES; ++s) {
      const int t = blockIdx.x + s * gridDim.x;
      if (t < ntiles) issue(s, t);
    }
  }
  __syncthreads();
  int k = 0;
  // tile coordinates advanced without a division per tile
  const int dq = gridDim.x / tiles_y, dr = gridDim.x % tiles_y;
  int tx = blockIdx.x / tiles_y, ty = blockIdx.x % tiles_y;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++k) {
    const int slot = k % STAGES;
    const uint32_t parity = (uint32_t)((k / STAGES) & 1);
    const bool ok = __syncthreads_and(mbar_wait_bounded(&full[slot], parity, A.wait_cycles));
    if (!ok) {
      // record, then wait (bounded) for every load still in flight before leaving
      if (threadIdx.x == 0) raise_status(A.st, ST_TIMEOUT);
      for (int s = 0; s < STAGES; ++s) {
        const int kk = k + s;
        if (blockIdx.x + kk * gridDim.x < ntiles)
          mbar_wait_bounded(&full[kk % STAGES], (uint32_t)((kk / STAGES) & 1), A.wait_cycles);
      }
      return;
    }
    grad_any_tile<TH, R, TX, TY, NT>(A, ring + slot * SLOT, tx * TX, ty * TY);
    tx += dq;
    ty += dr;
    if (ty >= tiles_y) {
      ty -= tiles_y;
      ++tx;
    }
    __syncthreads();  // every thread is done with this slot
    if (threadIdx.x == 0) {
      const int nt = t + STAGES * gridDim.x;
      if (nt < ntiles) issue(slot, nt);
    }
  }
}

// ---------------------------------------------------------------------------
// observables: energy, charges and coupling partials, as sums and as densities
// ---------------------------------------------------------------------------
enum DensityKind { D_ENERGY = 0, D_CHARGE = 1, D_COUPLING = 2 };
constexpr int OBS_MAX = 4;  // quantities per pass
struct ObsList {
  int n;
  int kind[OBS_MAX], which[OBS_MAX];
  unsigned comps;  // components whose jets any of them reads
};

// n quantities of the stored field in one pass: FP64 jets (values and masked first
// derivatives) of the components they need, the theory's points on them, one fixed-order
// compensated sum each (partial: n * gridDim.x slots, nullable) and, for n = 1, the density.
// A thread owns four adjacent rows of one column and takes them two at a time, so that the
// two rows' x neighbours are read and converted once (six FP64 components would spill: one).
// Bound for FP32 fields by the conversions (XU pipe: 16 per clock and SM), FP64 arithmetic and,
// with one tile per CTA, the tiles' load latency.  NQ: 1, or OBS_MAX for several quantities.  One
// quantity needs registers for its own sum only, and a CTA more per SM hides more of the loads; us,
// OBS_MAX at three CTAs -> 1 at four: energy 4096^2 chiral 228 -> 189, baby Skyrme 205 -> 166, density
// 1501 x 999 (plain loads) chiral 26.8 -> 22.7.  A ring of staged tiles under resident CTAs gave the
// same (189, 160) and slower densities (174 against 187).
template <class TH, typename R, int NQ>
struct ObserveShape {
  static constexpr bool WIDE = TH::NF > 4;
  static constexpr int PER = NQ == 1 && WIDE && sizeof(R) == 8 ? 1 : 2;
  static constexpr int CTAS = (WIDE ? 2 : 3) + (NQ == 1 ? 1 : 0);
};
template <class TH, typename R, int TX, int TY, int NT, bool TMA, int NQ>
__global__ void __launch_bounds__(NT, (ObserveShape<TH, R, NQ>::CTAS))
    observe_kernel(const __grid_constant__ CUtensorMap map, const R* __restrict__ phi, double* density, double* partial,
                   StepState* st, const __grid_constant__ ObsList L, const __grid_constant__ Grid G,
                   const __grid_constant__ Phys P, long long wait_cycles, unsigned tx_extra) {
  using TS = TileShape<TX, TY, NT>;
  constexpr int NF = TH::NF, ROWS = TX / (NT / TY), PER = ObserveShape<TH, R, NQ>::PER;
  static_assert(NT % TY == 0 && ROWS % PER == 0, "column mapping");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  R* tile = reinterpret_cast<R*>(smem_raw);
  __shared__ StageShared<NT> S;
  const int tiles_y = (G.Y + TY - 1) / TY;
  const int x0 = (blockIdx.x / tiles_y) * TX;
  const int y0 = (blockIdx.x % tiles_y) * TY;
  if constexpr (TMA) {
    if (!stage_tma<NF, R, TX, TY, NT>(tile, &map, &S.bar, x0, y0, tx_extra, wait_cycles, st)) return;
  } else {
    stage_plain<NF, R, TX, TY, NT>(tile, G, phi, x0, y0);
    __syncthreads();
  }
  const double ihx = G.ihx, ihy = G.ihy;
  const int ly = threadIdx.x % TY, gy = y0 + ly;
  double acc[NQ] = {};
#pragma unroll 1
  for (int s = 0; s < ROWS; s += PER) {
    const int lx = (threadIdx.x / TY) * ROWS + s;
    if (x0 + lx >= G.X || gy >= G.Y) break;
    const R* base = tile + (lx + 2) * TS::HY + (ly + TS::YOFF);
    Jet1<double, NF> J[PER];
#pragma unroll
    for (int a = 0; a < NF; ++a) {
      if (!((L.comps >> a) & 1u)) {
#pragma unroll
        for (int p = 0; p < PER; ++p) J[p].f[a] = J[p].dx[a] = J[p].dy[a] = 0.0;
        continue;
      }
      const R* pa = base + a * TS::PLANE;
      double x[PER + 4];
#pragma unroll
      for (int k = 0; k < PER + 4; ++k) x[k] = (double)pa[(k - 2) * TS::HY];
#pragma unroll
      for (int p = 0; p < PER; ++p) {
        const R* pr = pa + p * TS::HY;
        const Masks mk = site_masks(G, x0 + lx + p, gy);
        const double dx = d1_stencil<double>(x[p], x[p + 1], x[p + 3], x[p + 4], ihx);
        const double dy = d1_stencil<double>((double)pr[-2], (double)pr[-1], (double)pr[1], (double)pr[2], ihy);
        J[p].f[a] = x[p + 2];
        J[p].dx[a] = mk.x ? dx : 0.0;
        J[p].dy[a] = mk.y ? dy : 0.0;
      }
    }
#pragma unroll
    for (int p = 0; p < PER; ++p) {
      const int gx = x0 + lx + p;
      if (gx >= G.X) break;
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        if (NQ > 1 && q >= L.n) break;
        const double v = L.kind[q] == D_ENERGY   ? TH::energy(J[p], P, G.dA)
                         : L.kind[q] == D_CHARGE ? TH::charge(J[p], P, L.which[q], G.dA)
                                                 : TH::coupling(J[p], P, L.which[q], G.dA);
        if (q == 0 && density) density[(long long)gx * G.Y + gy] = v;
        acc[q] = __dadd_rn(acc[q], v);  // no contraction: both NQ round alike
      }
    }
  }
  if (!partial) return;
  for (int q = 0; q < L.n; ++q) {
    double a = acc[0];
    if constexpr (NQ > 1) a = q == 0 ? a : q == 1 ? acc[1] : q == 2 ? acc[2] : acc[3];
    const double bs = block_sum_fixed<NT>(a, S.red);
    if (threadIdx.x == 0) partial[(long long)q * gridDim.x + blockIdx.x] = bs;
  }
  if (threadIdx.x == 0) {
    __threadfence();
    const unsigned t = atomicAdd(&st->ticket, 1u);
    S.am_last = (t == gridDim.x - 1);
  }
  __syncthreads();
  if (!S.am_last) return;
  __threadfence();
  for (int q = 0; q < L.n; ++q) {
    const double E = fixed_order_sum<NT>(partial + (long long)q * gridDim.x, gridDim.x, S.sh_s, S.sh_c);
    if (threadIdx.x == 0) {
      st->scalars[q] = E;
      if (q == 0) st->scalar = E;
      if (!isfinite(E)) raise_status(st, ST_NONFINITE);
    }
  }
  if (threadIdx.x == 0) st->ticket = 0u;
}

// do_rk4_step_kernel (core/integrator.py:51-96)
template <typename R>
__global__ void rk4_stage_kernel(R* k_out, const R* vel, const R* l_in, R* temp, const R* phi, const R* k_prev,
                                 R factor, R dt, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const R k = dt * (vel[i] + factor * l_in[i]);
    const R t = phi[i] + factor * k_prev[i];
    k_out[i] = k;
    temp[i] = t;
  }
}

// do_rk4_kernel / do_rk4_kernel_no_constraint (core/integrator.py:99-189)
template <typename R, int NF, int NMAG>
__global__ void rk4_finalize_kernel(R* vel, R* phi, const R* k1, const R* k2, const R* k3, const R* k4, const R* l1,
                                    const R* l2, const R* l3, const R* l4, long long N, int normalize) {
  const R sixth = (R)(1.0 / 6.0), two = (R)2;
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N; s += (long long)gridDim.x * blockDim.x) {
    R P[NF], V[NF];
#pragma unroll
    for (int a = 0; a < NF; ++a) {
      const long long i = a * N + s;
      V[a] = vel[i] + sixth * (l1[i] + two * l2[i] + two * l3[i] + l4[i]);
      P[a] = phi[i] + sixth * (k1[i] + two * k2[i] + two * k3[i] + k4[i]);
    }
    if (NMAG > 0 && normalize) {
      R s2 = (R)0;
#pragma unroll
      for (int a = 0; a < NMAG; ++a) s2 += P[a] * P[a];
      const R nrm = sqrt(s2);
      if (nrm != (R)0) {
#pragma unroll
        for (int a = 0; a < NMAG; ++a) P[a] /= nrm;
      }
      R lm = (R)0;
#pragma unroll
      for (int a = 0; a < NMAG; ++a) lm += V[a] * P[a];
#pragma unroll
      for (int a = 0; a < NMAG; ++a) V[a] -= lm * P[a];
    }
#pragma unroll
    for (int a = 0; a < NF; ++a) {
      vel[a * N + s] = V[a];
      phi[a * N + s] = P[a];
    }
  }
}

// Copy of a field in another element type (S -> D), optionally with each site's
// unit-vector components divided by their FP64 norm (the projection the flow applies
// after every step).  A stored FP32 unit vector cannot hold m3 = 1 - |m_perp|^2/2 once
// |m_perp| < 2.4e-4: it rounds to 1 and |m|^2 - 1 = |m_perp|^2 > 0 there; an FP64
// projected copy restores the constraint to FP64 rounding.  Each site's components are
// read and normalised in FP64, then rounded once to D.
template <typename S, typename D, int NF, int NMAG>
__global__ void convert_kernel(const S* src, D* dst, long long N, int normalize) {
  for (long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x; s < N; s += (long long)gridDim.x * blockDim.x) {
    double P[NF];
#pragma unroll
    for (int a = 0; a < NF; ++a) P[a] = (double)src[a * N + s];
    if (NMAG > 0 && normalize) {
      double s2 = 0.0;
#pragma unroll
      for (int a = 0; a < NMAG; ++a) s2 += P[a] * P[a];
      if (s2 > 0.0) {
        const double nrm = sqrt(s2);
#pragma unroll
        for (int a = 0; a < NMAG; ++a) P[a] /= nrm;
      }
    }
#pragma unroll
    for (int a = 0; a < NF; ++a) dst[a * N + s] = (D)P[a];
  }
}

}  // namespace ssb
