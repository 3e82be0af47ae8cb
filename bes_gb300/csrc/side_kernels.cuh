// Residual kernels of the explicit iteration.
//
// GB300 issues one FP64 warp instruction per 16 to 19 cycles and SM (measured with chains of
// DFMA, DADD, DMUL and DSETP: 64 cycles per sub-partition, whatever the number of active
// lanes), against four 32-bit warp instructions per cycle, so these kernels are bound by the
// NUMBER of FP64 instructions and everything else is traded for it:
//   * Green-Gauss, the scaling by 1/V and the products with the centroid-to-face vectors are one
//     4x4 matrix per cell (hmat, built once per mesh): with D_j the difference to neighbour j
//     (sum_j S_j = 0 removes the cell's own value), h_k = G . r_k = sum_j (r_k . S_j (1-w_j)/V) D_j;
//   * the limiter needs only the largest positive and the most negative h_k, because for one
//     variable and one sign of h every face has the same D1 and the limiter function
//     (t + h D)/(t + h(h + D)/2), t = D^2 + eps^2, is >= 1 for |h| <= |D| and falls with |h|
//     beyond; the extremes and all comparisons are integer comparisons of the bit patterns;
//   * the MUSCL state is u + phi h_k;
//   * the thermodynamic side state (reciprocal density, velocity, pressure, enthalpy, sound
//     speed) is computed once per reconstructed state instead of once per face side;
//   * the Roe flux takes |A| dU = l2 dU + ((l1-l2) a1 + (l5-l2) a5) (1, u, H)
//     + ((l5-l2) a5 - (l1-l2) a1) c (0, n, vn), which follows from dU = sum of all waves, and
//     the Roe-averaged c^2 = a cL^2 + b cR^2 + (gamma-1)/2 a b |du|^2;
//   * reciprocals and square roots from the hardware's 2^-20 seeds with one third-order step
//     (Halley for 1/x, Householder for 1/sqrt(x)): at most 1 and 2 ulp measured over 2^-60..2^60.
// FP64 instructions per cell and stage (Nf/Nc = 2): about 570 + 420 + 30 before, 180 + 155 + 27.
//
// Implicit steps keep the kernels of explicit_kernels.cuh, and with them the bits of their results:
// the linear solves of the FP32 and 16-bit systems amplify a rounding difference of the right-hand
// side (1e-15 becomes 5e-9 and 5e-7 of the state after one step, well inside the solves' own
// tolerance).  The residual is 7 to 8 % of a step on 2.16M cells in 16-bit storage.
#pragma once
#include "explicit_kernels.cuh"

namespace bes {

constexpr int kSideW = 8;    // doubles per side state
constexpr int kReconCells = 32;  // cells of a cell-sweep block (one warp per variable)

// A side state holds half-scaled values, so that the flux's 1/2 costs no instruction:
// rho/2, sqrt(rho/2), u, v | w, p/2, H, c^2.
struct SideState {
  double rho, s, u[3], p, H, c2;
};

// x in [2^-1000, 2^1000]: the range in which the fast reciprocals need no special case
__device__ __forceinline__ bool mid_range(double x) {
  return (unsigned)(__double2hiint(x) - 0x01700000) < 0x7d000000u;
}
// 1/x: hardware seed, one Halley step (e = 1 - x r; r (1 + e + e^2))
__device__ __forceinline__ double fast_rcp(double x) {
  if (!mid_range(x)) return 1.0 / x;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  double e = fma(-x, r, 1.0);
  e = fma(e, e, e);
  return fma(r, e, r);
}
// 1/sqrt(x): hardware seed, one third-order Householder step (y (1 + e/2 + 3 e^2/8))
__device__ __forceinline__ double fast_rsqrt(double x) {
  if (!mid_range(x)) return 1.0 / sqrt(x);
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}
// sqrt(x) as a product s y, so that adding to it is one fma: x times 1/sqrt(x), or sqrt(x) times 1
// outside of the range (0 times 1/sqrt(0) is a NaN, and a cell without pressure is a valid state)
struct RootFactors {
  double s, y;
};
__device__ __forceinline__ RootFactors fast_sqrt(double x) {
  return mid_range(x) ? RootFactors{x, fast_rsqrt(x)} : RootFactors{sqrt(x), 1.0};
}
__device__ __forceinline__ long long dbits(double x) { return __double_as_longlong(x); }
// a <= b for a, b >= 0 (or a NaN, which compares greater than every number)
__device__ __forceinline__ bool le_nonneg(double a, double b) { return dbits(a) <= dbits(b); }
__device__ __forceinline__ bool is_nan_bits(double x) {
  return (dbits(x) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}

// hmat[(k*2 + j/2)*nc + c] (pairs j, j+1): r_k . S_j / V times 1 - w_j for an interior face j,
// 1 for a slip wall (its difference is that of the tangential momentum), 0 otherwise.
static __global__ void __launch_bounds__(128) face_matrix_kernel(DevMesh m, double2* __restrict__ H) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int nc = m.nc;
  if (c >= nc) return;
  const double iv = m.inv_vol[c];
  const int flags = m.cflags[c];
  double S[4][3];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const bool interior = m.adj[j * nc + c] >= 0;
    const double k = interior ? (1.0 - m.w[j * nc + c]) * iv : ((flags >> j) & 1 ? iv : 0.0);
#pragma unroll
    for (int d = 0; d < 3; ++d) S[j][d] = m.Sc[(j * 3 + d) * nc + c] * k;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    double r[3], h[4];
#pragma unroll
    for (int d = 0; d < 3; ++d) r[d] = m.r[(k * 3 + d) * nc + c];
#pragma unroll
    for (int j = 0; j < 4; ++j) h[j] = r[0] * S[j][0] + r[1] * S[j][1] + r[2] * S[j][2];
    H[(int64_t)(k * 2) * nc + c] = make_double2(h[0], h[1]);
    H[(int64_t)(k * 2 + 1) * nc + c] = make_double2(h[2], h[3]);
  }
}

// Side state of the reconstructed conserved variables x.
__device__ __forceinline__ void store_side(const Params& g, const double* x, double* __restrict__ dst) {
  SideState q;
  q.rho = 0.5 * x[0];
  double ir;
  if (mid_range(q.rho)) {
    const double y = fast_rsqrt(q.rho);
    q.s = q.rho * y;
    ir = 0.5 * (y * y);
  } else {
    // a density extrapolated below 0 at a wall face has a pressure all the same, which is all
    // that the wall's flux takes; only the Roe flux takes its root (a NaN)
    q.s = sqrt(q.rho);
    ir = 1.0 / x[0];
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) q.u[d] = x[1 + d] * ir;
  const double k = fma(x[1], q.u[0], fma(x[2], q.u[1], x[3] * q.u[2]));
  q.p = g.half_gm1 * fma(-0.5, k, x[4]);
  q.H = fma(2.0, q.p, x[4]) * ir;
  q.c2 = g.two_gamma * q.p * ir;
  double2* o = reinterpret_cast<double2*>(dst);
  o[0] = make_double2(q.rho, q.s);
  o[1] = make_double2(q.u[0], q.u[1]);
  o[2] = make_double2(q.u[2], q.p);
  o[3] = make_double2(q.H, q.c2);
}
__device__ __forceinline__ SideState load_side(const double* __restrict__ src) {
  const double2* o = reinterpret_cast<const double2*>(src);
  const double2 a = o[0], b = o[1], c = o[2], d = o[3];
  return SideState{a.x, a.y, {b.x, b.y, c.x}, c.y, d.x, d.y};
}

// Local time step CFL V / sum_d (c~ + |u_d|) L_d with c~ = sqrt(gamma) c (quirk Q3) at the
// cell's own state u.
__device__ __forceinline__ double local_time_step(const DevMesh& m, const Params& g, int c,
                                                  const double* u, double cfl) {
  const double ir = fast_rcp(u[0]);
  double w[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) w[d] = u[1 + d] * ir;
  const double k = fma(u[1], w[0], fma(u[2], w[1], u[3] * w[2]));
  const double cs2 = g.gamma2_gm1 * fma(-0.5, k, u[4]) * ir;
  const RootFactors cs = fast_sqrt(cs2);
  double spec = 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d)
    spec = fma(fma(cs.s, cs.y, fabs(w[d])), m.plen[(int64_t)d * m.nc + c], spec);
  return cfl * m.vol[c] * fast_rcp(spec);
}

// Cell sweep: 32 cells per block, warp v reconstructs variable v of the 32 cells (a fifth of a
// cell's FP64 chain per thread: a mesh with fewer cells than the chip has sub-partitions x 32
// runs in the time of one chain), then the side states are built from shared memory by warps
// 0..NS (slot NS: the extra state of quirk Q13) while warp 4 computes the time step.
// U is [5][nc], side states [ld][8] at index slot*nc + cell, extras after them.
template <bool STAGE0, int NS>
__global__ void __launch_bounds__(kReconCells * 5) side_recon_kernel(
    DevMesh m, Params prm, const double* __restrict__ U, double* __restrict__ RS, int64_t ldr,
    double* __restrict__ dt, double cfl, int local_dt, unsigned long long* __restrict__ dtmin,
    unsigned long long* stamp) {
  __shared__ double sx[NS + 1][5][kReconCells];
  const int nc = m.nc;
  const int v = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * kReconCells + lane;
  stamp_start(stamp);
  if (condition_frozen(prm)) return;
  {
    const int64_t b = blockIdx.y;
    U += b * 5 * nc;
    RS += b * kSideW * ldr;
    dt += b * nc;
    dtmin += b;
  }
  int flags = 0;
  if (c < nc) {
    const double* Uv = U + (int64_t)v * nc;
    const double u = Uv[c];
    int a[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) a[k] = m.adj[k * nc + c];
    double2 h2[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) h2[q] = m.hmat[(int64_t)q * nc + c];
    const double eps2 = m.eps2[c];
    flags = m.cflags[c];
    double D[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) D[k] = Uv[a[k] >= 0 ? a[k] : c];
    long long hi = 0;                             // largest difference, >= +0
    unsigned long long lo = 0x8000000000000000ull;  // most negative difference, <= -0
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      D[k] = D[k] - u;  // +0 on a boundary face
      const long long q = dbits(D[k]);
      hi = q > hi ? q : hi;
      lo = (unsigned long long)q > lo ? (unsigned long long)q : lo;
    }
    if ((flags & 15) && v >= 1 && v <= 3) {
      // slip wall: the momentum's tangential part at the face (GradientGreenGauss.cpp:83-121)
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (flags & (1 << k)) {
          const int f = m.cface[k * nc + c];
          double vn = 0.0;
#pragma unroll
          for (int d = 0; d < 3; ++d) vn = fma(U[(int64_t)(1 + d) * nc + c], m.fn[(int64_t)d * m.nf + f], vn);
          D[k] = -vn * m.fn[(int64_t)(v - 1) * m.nf + f];
        }
    }
    double h[4];
    long long hp = 0;
    unsigned long long hn = 0x8000000000000000ull;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      h[k] = fma(h2[2 * k].x, D[0], fma(h2[2 * k].y, D[1], fma(h2[2 * k + 1].x, D[2], h2[2 * k + 1].y * D[3])));
      const long long q = a[k] >= 0 ? dbits(h[k]) : 0ll;  // boundary faces do not limit
      hp = q > hp ? q : hp;
      hn = (unsigned long long)q > hn ? (unsigned long long)q : hn;
    }
    double phi = 1.0;
    const bool up = hp > hi, down = hn > lo;
    if (up || down) {
      double hh = __longlong_as_double(up ? hp : (long long)hn);
      double dd = __longlong_as_double(up ? hi : (long long)lo);
      double t = fma(dd, dd, eps2);
      double num = fma(hh, dd, t), den = fma(0.5 * hh, hh + dd, t);
      if (up && down) {  // both signs limit: the smaller ratio
        hh = __longlong_as_double((long long)hn);
        dd = __longlong_as_double((long long)lo);
        t = fma(dd, dd, eps2);
        const double num2 = fma(hh, dd, t), den2 = fma(0.5 * hh, hh + dd, t);
        if (num2 * den < num * den2) {
          num = num2;
          den = den2;
        }
      }
      if (dbits(num) < dbits(den)) phi = num * fast_rcp(den);
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) sx[s][v][lane] = fma(phi, h[s], u);
    if (flags & 0x10) {
      for (int k = 0; k < m.n_extra; ++k)
        if (m.extra_cell[k] == c) {
          const int s = m.extra_m[k];
          sx[NS][v][lane] = fma(phi, s == 0 ? h[0] : (s == 1 ? h[1] : (s == 2 ? h[2] : h[3])), u);
        }
    }
  }
  __syncthreads();
  double dt_c = 1e300;
  if (c < nc) {
    // NS 1: warp 0 the main state, warp 1 the extra one; NS 4: warps 0..3 their slots
    if (v < NS) {
      double x[5];
#pragma unroll
      for (int q = 0; q < 5; ++q) x[q] = sx[v][q][lane];
      store_side(prm, x, RS + ((int64_t)v * nc + c) * kSideW);
    } else if (NS == 1 && v == 1 && (flags & 0x10)) {
      double x[5];
#pragma unroll
      for (int q = 0; q < 5; ++q) x[q] = sx[NS][q][lane];
      for (int k = 0; k < m.n_extra; ++k)
        if (m.extra_cell[k] == c) store_side(prm, x, RS + ((int64_t)nc * NS + k) * kSideW);
    }
    if (STAGE0 && v == 4) {
      double u[5];
#pragma unroll
      for (int q = 0; q < 5; ++q) u[q] = U[(int64_t)q * nc + c];
      dt_c = local_time_step(m, prm, c, u, cfl);
      dt[c] = dt_c;
    }
  }
  if (STAGE0 && !local_dt && v == 4) {
    // positive doubles order like their bit patterns
    unsigned long long x = (unsigned long long)dbits(dt_c);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long y = __shfl_xor_sync(0xffffffffu, x, o);
      x = y < x ? y : x;
    }
    if (lane == 0) atomicMin(dtmin, x);
  }
}

// Characteristic freestream boundary (FluxFreestream.tpp:35-190) from a side state, per unit area.
__device__ __forceinline__ void side_freestream_flux(const GasConst& g, const SideState& L,
                                                     const double* __restrict__ Pinf,
                                                     const double* n, double* F) {
  const double rho = 2.0 * L.rho, p = 2.0 * L.p, c2 = L.c2;
  const double cL = sqrt(c2);
  const double vn = L.u[0] * n[0] + L.u[1] * n[1] + L.u[2] * n[2];
  double B[6];
  const bool super = fabs(vn) >= cL;
  if (super && vn <= 0.0) {
#pragma unroll
    for (int i = 0; i < 6; ++i) B[i] = Pinf[i];
  } else if (super) {
    B[0] = rho;
#pragma unroll
    for (int d = 0; d < 3; ++d) B[1 + d] = L.u[d];
    B[4] = p;
    B[5] = p / (g.R * rho);
  } else {
    const double c1 = rho * cL;
    if (vn <= 0.0) {  // subsonic inlet (:49-126)
      const double t = n[0] * (Pinf[1] - L.u[0]) + n[1] * (Pinf[2] - L.u[1]) + n[2] * (Pinf[3] - L.u[2]);
      B[4] = 0.5 * (Pinf[4] + p - c1 * t);
      const double k = (Pinf[4] - B[4]) / c1;
      B[0] = Pinf[0] + (B[4] - Pinf[4]) / c2;
#pragma unroll
      for (int d = 0; d < 3; ++d) B[1 + d] = Pinf[1 + d] - k * n[d];
    } else {  // subsonic outlet (:129-190)
      B[4] = Pinf[4];
      const double k = (p - B[4]) / c1;
      B[0] = rho + (B[4] - p) / c2;
#pragma unroll
      for (int d = 0; d < 3; ++d) B[1 + d] = L.u[d] + k * n[d];
    }
    B[5] = B[4] / (g.R * B[0]);
  }
  prim_flux(g, B, n, F);
}

// Roe flux with Harten's fix times area (FluxRoe.tpp:110-333) of two side states; 77 FP64
// instructions.
__device__ __forceinline__ void side_roe_flux(const Params& g, const SideState& L,
                                              const SideState& R, const double* n, double A,
                                              double* F) {
  const double iden = fast_rcp(L.s + R.s);
  const double a = L.s * iden, b = R.s * iden;
  double du[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) du[d] = R.u[d] - L.u[d];
  const double dd = fma(du[0], du[0], fma(du[1], du[1], du[2] * du[2]));
  const double vL = fma(L.u[0], n[0], fma(L.u[1], n[1], L.u[2] * n[2]));
  const double dv = fma(du[0], n[0], fma(du[1], n[1], du[2] * n[2]));
  const double vR = vL + dv;
  const double vn = fma(b, dv, vL);
  const double c2 = fma(a, L.c2, fma(b, R.c2, (g.half_gm1 * (a * b)) * dd));
  const double y = fast_rsqrt(c2);  // 1/c
  const double c = c2 * y;
  const double delta = fabs(g.gas.harten * c);
  double l1 = fabs(vn - c), l2 = fabs(vn), l5 = fabs(vn + c);
  if (le_nonneg(l1, delta) || le_nonneg(l2, delta) || le_nonneg(l5, delta)) {
    const double ih = 0.5 * fast_rcp(delta), d2 = delta * delta;
    if (le_nonneg(l1, delta)) l1 = fma(l1, l1, d2) * ih;
    if (le_nonneg(l2, delta)) l2 = fma(l2, l2, d2) * ih;
    if (le_nonneg(l5, delta)) l5 = fma(l5, l5, d2) * ih;
  }
  const double dp = R.p - L.p;              // half the pressure difference
  const double x = (L.s * R.s) * c * dv;    // half of rho c dvn
  const double b1 = (l1 - l2) * (dp - x), b5 = (l5 - l2) * (dp + x);
  const double hy = 0.5 * y;
  const double A1 = (b1 + b5) * (hy * y), A2 = (b5 - b1) * hy;
  const double PL = fma(-A1, a, L.rho * (vL + l2)) * A;
  const double PR = fma(-A1, b, R.rho * (vR - l2)) * A;
  const double cn = (L.p + R.p - A2) * A;
  const double e = fma(l2, dp, -A2 * vn) * A;
  F[0] = PL + PR;
#pragma unroll
  for (int d = 0; d < 3; ++d) F[1 + d] = fma(PL, L.u[d], fma(PR, R.u[d], cn * n[d]));
  F[4] = fma(PL, L.H, fma(PR, R.H, e));
}

// Per face: flux times area, FA [nf][kFaW].
static __global__ void __launch_bounds__(128) side_flux_kernel(
    DevMesh m, Params prm, const double* __restrict__ RS, int64_t ldr, double* __restrict__ FA,
    int* __restrict__ nan_flag, unsigned long long* stamp) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  const int nf = m.nf;
  stamp_start(stamp);
  if (f >= nf || condition_frozen(prm)) return;
  const int64_t cond = blockIdx.y;
  RS += cond * kSideW * ldr;
  FA += cond * kFaW * nf;
  const SideState L = load_side(RS + (int64_t)m.fsrc_own[f] * kSideW);
  double n[3], F[5];
#pragma unroll
  for (int d = 0; d < 3; ++d) n[d] = m.fn[(int64_t)d * nf + f];
  const double A = m.farea[f];
  if (f < m.nf_int) {
    const SideState R = load_side(RS + (int64_t)m.fsrc_nb[f] * kSideW);
    side_roe_flux(prm, L, R, n, A, F);
  } else if (f < m.nf_int + m.nf_slip) {
    const double pA = 2.0 * L.p * A;
    F[0] = F[4] = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) F[1 + d] = pA * n[d];
  } else {
    side_freestream_flux(prm.gas, L, prm.pinf_dev + 6 * cond, n, F);
#pragma unroll
    for (int v = 0; v < 5; ++v) F[v] *= A;
  }
  bool bad = false;
#pragma unroll
  for (int v = 0; v < 5; ++v) bad |= is_nan_bits(F[v]);
  store_fa(FA, f, F);
  if (bad) atomicCAS(nan_flag, 0, f + 1);
}

// Face-side states and fluxes of every condition at U (stage0: with the time step).  stamps
// (may be null): [2] start times of the two kernels.
inline void launch_side_residual(bes_ctx* c, cudaStream_t s, const double* U, bool stage0,
                                 double cfl, const Params& prm, unsigned long long* stamps) {
  const DevMesh& m = c->dm;
  const dim3 gc((unsigned)((m.nc + kReconCells - 1) / kReconCells), c->nb);
  const dim3 gf((unsigned)((m.nf + 127) / 128), c->nb);
  const int local = c->opt.local_time_step;
#define BES_RECON(ST, NS)                                                                    \
  side_recon_kernel<ST, NS><<<gc, kReconCells * 5, 0, s>>>(m, prm, U, c->RS, c->rs_ld, c->dt, \
                                                           cfl, local, c->dtmin, stamps)
  if (m.nslots == 1) {
    if (stage0) BES_RECON(true, 1);
    else BES_RECON(false, 1);
  } else {
    if (stage0) BES_RECON(true, 4);
    else BES_RECON(false, 4);
  }
#undef BES_RECON
  side_flux_kernel<<<gf, 128, 0, s>>>(m, prm, c->RS, c->rs_ld, c->FA, c->nan_flag,
                                      stamps ? stamps + 1 : nullptr);
}

}  // namespace bes
