// Kernels of the implicit (backward-Euler) path: first-order flux Jacobians, assembly of
// the 5x5-block system, the block-ILU(0) factorisation and the 16-bit
// block-scaled copies of the system (the Krylov side is in krylov_kernels.cuh).  T is the
// precision of the matrix, preconditioner and Krylov vectors (double for the plain method,
// float for the defect correction); residuals, right-hand sides and the state stay FP64.
//
// Slots of a row: 0 the diagonal block, 1 + m the block coupling to the neighbour across local face
// m (zero where there is none).
// The Krylov-side vectors (right-hand side b, iterates, basis, preconditioner output) are
// cell-major: component v of cell i is x[i*5 + v], so a neighbour's five values are one
// 20-byte gather (SoA would touch five 32-byte sectors) while streams stay coalesced; the
// FP64 state and residual keep the solver's [5][nc] layout.
#pragma once
#include <cuda_fp16.h>

#include <type_traits>

#include "explicit_kernels.cuh"
#include "flux_jacobian.cuh"

namespace bes {

constexpr int kRedBlocks = 1024;  // fixed grid of the reduction kernels (deterministic sums)

// ---- storage of the 5x5 blocks (matrix, factors, inverse diagonal) in the system's type ----------
// Groups of 32 rows; within a group slot after slot (the matrix: 0 the diagonal, 1..4 the local
// faces); of a slot first entries 0..W-1 of the 32 rows' row-major blocks, W the entries in 16
// bytes, then entries W..2W-1 and so on, and last the entries 24.  A warp reads a block with 16-byte
// loads (seven instead of 25 in FP32, thirteen in FP64), all from one contiguous piece per group,
// before the products.  With one array per entry, every product waiting for its own load, a
// preconditioner application took 169 us on 540,000 cells in FP32 and 160 us on 129,600 in FP64,
// now 66 and 83; a factorisation on 2.16M cells 3.0 ms, now 1.8.
template <class T>
struct Vec16 {
  static constexpr int W = 16 / sizeof(T);
};
constexpr int kGroupVals = 32 * 25;
inline int64_t block_values(int64_t nc, int nslots) { return (nc + 31) / 32 * nslots * kGroupVals; }
// entry q of slot s of row i
template <class T>
__host__ __device__ __forceinline__ int64_t block_at(int nslots, int s, int q, int64_t i) {
  constexpr int W = Vec16<T>::W;
  return ((i >> 5) * nslots + s) * kGroupVals +
         (q < 24 ? (q / W) * (32 * W) + (i & 31) * W + q % W : 768 + (i & 31));
}
template <class T>
__device__ __forceinline__ void load_block(const T* A, int nslots, int s, int i, T* a) {
  constexpr int W = Vec16<T>::W;
  const T* p = A + block_at<T>(nslots, s, 0, i);
#pragma unroll
  for (int k = 0; k < 24 / W; ++k) {
    const uint4 u = *reinterpret_cast<const uint4*>(p + k * 32 * W);
    const T* v = reinterpret_cast<const T*>(&u);
#pragma unroll
    for (int e = 0; e < W; ++e) a[k * W + e] = v[e];
  }
  a[24] = A[block_at<T>(nslots, s, 24, i)];
}
template <class T>
__device__ __forceinline__ void store_block(T* A, int nslots, int s, int i, const T* a) {
  constexpr int W = Vec16<T>::W;
  T* p = A + block_at<T>(nslots, s, 0, i);
#pragma unroll
  for (int k = 0; k < 24 / W; ++k) {
    uint4 u;
    T* v = reinterpret_cast<T*>(&u);
#pragma unroll
    for (int e = 0; e < W; ++e) v[e] = a[k * W + e];
    *reinterpret_cast<uint4*>(p + k * 32 * W) = u;
  }
  A[block_at<T>(nslots, s, 24, i)] = a[24];
}

// ---- 16-bit block-scaled storage of the FP32 system (precision 2)
// Entry q of a 5x5 block = scale * half q.  The scale is the smallest power of two >= the block's
// largest |entry|, so the rescaling is exact and every stored entry lies in [-1, 1] with FP16's
// 11-bit significand; entries below 2^-14 of the scale become FP16 subnormals (absolute error at
// most 2^-25 of the scale).  A block is 13 words: words 0..11 the halves 0..23, word 12 the
// half 24 and, in its upper 16 bits, the upper 16 bits of the FP32 scale (a power of two has no
// others).  52 bytes instead of 100.
// Layout: groups of 32 rows; within a group slot after slot; of a slot first words 0..3 of the 32
// rows, then words 4..7, words 8..11 (16 bytes per row each) and words 12.  A warp reads a block
// with three 16-byte loads and one of 4 bytes per lane, and its group's slots are one contiguous
// piece.  With one 4-byte array per word and a separate scale (14 loads and streams per block) an
// application on 2.16M cells took 194 us and a product 147 us, now 147 and 102.
constexpr int kBlockWords = 13;
constexpr int kGroupWords = 32 * kBlockWords;
inline int64_t packed_words(int64_t nc, int nslots) { return (nc + 31) / 32 * nslots * kGroupWords; }
// the words of slot s of row i's group
__device__ __forceinline__ const uint32_t* packed_slot(const uint32_t* H, int nslots, int s, int i) {
  return H + ((int64_t)(i >> 5) * nslots + s) * kGroupWords;
}
// word p of row i within its slot
__device__ __forceinline__ int packed_word(int p, int i) {
  return p < 12 ? (p >> 2) * 128 + (i & 31) * 4 + (p & 3) : 384 + (i & 31);
}
__device__ __forceinline__ float packed_scale(uint32_t last) {
  return __uint_as_float(last & 0xffff0000u);
}
struct PackedBlock {
  uint4 q[3];
  uint32_t last;
  // the entries (without the scale); returns the scale
  __device__ __forceinline__ float unpack(float* a) const {
    const uint32_t w[kBlockWords] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z,
                                     q[1].w, q[2].x, q[2].y, q[2].z, q[2].w, last};
#pragma unroll
    for (int p = 0; p < 12; ++p) {
      const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[p]));
      a[2 * p] = f.x;
      a[2 * p + 1] = f.y;
    }
    a[24] = __low2float(*reinterpret_cast<const __half2*>(&w[12]));
    return packed_scale(last);
  }
};

// smallest power of two >= x (x >= 0 and finite); 1 for x == 0
__device__ __forceinline__ float pow2_ceil(float x) {
  if (x == 0.0f) return 1.0f;
  const unsigned b = __float_as_uint(x);
  return __uint_as_float((b + 0x007fffffu) & 0xff800000u);
}

// a (row-major block) into slot s of row i
__device__ __forceinline__ void store_packed(uint32_t* __restrict__ H, int nslots, int s, int i,
                                             const float* a) {
  float mx = 0.0f;
#pragma unroll
  for (int q = 0; q < 25; ++q) mx = fmaxf(mx, fabsf(a[q]));
  const float sc = pow2_ceil(mx);
  const float inv = 1.0f / sc;  // exact: sc is a power of two
  uint32_t w[12];
#pragma unroll
  for (int p = 0; p < 12; ++p) {
    const __half2 h = __floats2half2_rn(a[2 * p] * inv, a[2 * p + 1] * inv);
    w[p] = *reinterpret_cast<const uint32_t*>(&h);
  }
  uint32_t* base = H + ((int64_t)(i >> 5) * nslots + s) * kGroupWords;
#pragma unroll
  for (int p = 0; p < 3; ++p)
    *reinterpret_cast<uint4*>(base + packed_word(4 * p, i)) =
        make_uint4(w[4 * p], w[4 * p + 1], w[4 * p + 2], w[4 * p + 3]);
  base[packed_word(12, i)] =
      (uint32_t)__half_as_ushort(__float2half_rn(a[24] * inv)) | (__float_as_uint(sc) & 0xffff0000u);
}

// block of slot s of row i
__device__ __forceinline__ PackedBlock load_packed(const uint32_t* __restrict__ H, int nslots, int s, int i) {
  const uint32_t* w = packed_slot(H, nslots, s, i);
  PackedBlock b;
#pragma unroll
  for (int p = 0; p < 3; ++p) b.q[p] = *reinterpret_cast<const uint4*>(w + packed_word(4 * p, i));
  b.last = w[packed_word(12, i)];
  return b;
}

// a[k] for a runtime k in [0, 4) without indexing the array (keeps it in registers)
__device__ __forceinline__ int sel4(const int* a, int k) {
  return k == 0 ? a[0] : (k == 1 ? a[1] : (k == 2 ? a[2] : a[3]));
}

// 5x5 inverse by Gauss-Jordan elimination with partial pivoting.
template <class T>
__device__ __forceinline__ void inv5(const T* a, T* inv) {
  T m[5][10];
#pragma unroll
  for (int i = 0; i < 5; ++i)
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      m[i][j] = a[i * 5 + j];
      m[i][5 + j] = (i == j) ? T(1) : T(0);
    }
#pragma unroll
  for (int c = 0; c < 5; ++c) {
    // pivot: the first row r >= c with the largest |m[r][c]|; the swap is written with
    // compile-time row indices (predicated), so m stays in registers
    int p = c;
    T best = fabs(m[c][c]);
#pragma unroll
    for (int r = c + 1; r < 5; ++r)
      if (fabs(m[r][c]) > best) {
        best = fabs(m[r][c]);
        p = r;
      }
#pragma unroll
    for (int r = c + 1; r < 5; ++r)
      if (r == p)
#pragma unroll
        for (int j = 0; j < 10; ++j) {
          const T t = m[r][j];
          m[r][j] = m[c][j];
          m[c][j] = t;
        }
    const T piv = T(1) / m[c][c];
#pragma unroll
    for (int j = 0; j < 10; ++j) m[c][j] *= piv;
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      if (r == c) continue;
      const T f = m[r][c];
#pragma unroll
      for (int j = 0; j < 10; ++j) m[r][j] -= f * m[c][j];
    }
  }
#pragma unroll
  for (int i = 0; i < 5; ++i)
#pragma unroll
    for (int j = 0; j < 5; ++j) inv[i * 5 + j] = m[i][5 + j];
}

// ---------------------------------------------------------------------------------------
// Jacobians and assembly (SolverImplicit::computeFaceFluxes_, src/SolverImplicit.cpp:358-507)
// ---------------------------------------------------------------------------------------
// Per face: dF/dU_L (slot 0) and, for interior faces, dF/dU_R (slot 1) at the FIRST-order states (the
// two cell averages), in the block layout by groups of 32 faces.  A warp writes whole sectors; the
// cells read both blocks of their faces and scale them.  Written per face into the cells' rows
// (scattered blocks and the diagonals' contributions, twice the bytes) and differentiated with
// all five derivatives of every quantity, this took 2.8 ms on 2.16M cells (FP32) and 5.4 ms on
// 518,400 (FP64, bound by the FP64 pipe), now 0.7 and 2.5.
template <class T>
__global__ void __launch_bounds__(128) face_jacobian_kernel(DevMesh m, Params prm,
                                                            const double* __restrict__ U,
                                                            T* __restrict__ Jf) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  const int nc = m.nc, nf = m.nf;
  if (f >= nf) return;
  const int o = m.fown[f];
  double n[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) n[d] = m.fn[(int64_t)d * nf + f];
  T ul[5], ur[5];
#pragma unroll
  for (int v = 0; v < 5; ++v) ul[v] = (T)U[(int64_t)v * nc + o];
  const bool interior = f < m.nf_int;
  if (interior) {
    const int nb = m.fnb[f];
#pragma unroll
    for (int v = 0; v < 5; ++v) ur[v] = (T)U[(int64_t)v * nc + nb];
  }
  const GasConst g = prm.gas;
  if constexpr (std::is_same<T, double>::value) {
    if (interior) {
      T J[25];
      roe_derivative<T>(g, var_side<T>(g, ul, n), fixed_side<T>(g, ur, n), n, J);
      store_block(Jf, 2, 0, f, J);
      roe_derivative<T>(g, fixed_side<T>(g, ul, n), var_side<T>(g, ur, n), n, J);
      store_block(Jf, 2, 1, f, J);
      return;
    }
  }
  typedef Dual<5, T> DT;
  T JL[25], JR[25];
  for (int side = 0; side < (interior ? 2 : 1); ++side) {
    DT dl[5], dr[5], dfl[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      dl[v] = DT(ul[v]);
      dr[v] = DT(interior ? ur[v] : T(0));
      if (side == 0)
        dl[v].d[v] = T(1);
      else
        dr[v].d[v] = T(1);
    }
    if (interior)
      roe_flux(g, dl, dr, n, dfl);
    else if (f < m.nf_int + m.nf_slip)
      slipwall_flux(g, dl, n, dfl);
    else
      freestream_flux(g, dl, prm.pinf_dev, n, dfl);
    T* J = side == 0 ? JL : JR;
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int c = 0; c < 5; ++c) J[r * 5 + c] = dfl[r].d[c];
  }
  store_block(Jf, 2, 0, f, JL);
  if (interior) store_block(Jf, 2, 1, f, JR);
}

// D += m J, `rep` times.  FP32: each product rounded once and added `rep` times, in the order in
// which the system was always formed.  FP64: rep m J with one rounding (the additions would
// take a thousand FP64 instructions per cell).
__device__ __forceinline__ void add_scaled(float* J, float m, int rep, float* D) {
#pragma unroll
  for (int q = 0; q < 25; ++q) J[q] = __fmul_rn(m, J[q]);
#pragma unroll 1
  for (int r = 0; r < rep; ++r)
#pragma unroll
    for (int q = 0; q < 25; ++q) D[q] += J[q];
}
__device__ __forceinline__ void add_scaled(const double* J, double m, int rep, double* D) {
  const double k = (double)rep * m;
#pragma unroll
  for (int q = 0; q < 25; ++q) D[q] = fma(k, J[q], D[q]);
}

struct FaceLocal {
  const int8_t* m_own;  // local face index of the face in its owner
  const int8_t* m_nb;   // ... in its neighbour (-1 on boundary faces)
};

// Outputs of the assembly; null where a context has no use for one.
template <class T>
struct AssembleOut {
  T* A;
  T* LU;          // a second copy, for the factorisation
  T* Dinv;        // inverse diagonal (block Jacobi)
  uint32_t* A16;  // packed A and inverse diagonal
  uint32_t* D16;
};

// Per cell: right-hand side -(dt/V) sum(+-F A) in the reference's face order, the diagonal
// block I + rep * sum of the face contributions (m J_L of the faces it owns, -m J_R of the others,
// m = dt / V * area), the off-diagonal blocks (m J_R, -m J_L, each added `rep` times from zero, as
// the reference's addToBlock sits inside the variable loop, quirk Q9), block-Jacobi inverse
// (optional), and block partial norms of the right-hand side.
template <class T>
__global__ void __launch_bounds__(128) cell_assemble_kernel(
    DevMesh m, FaceLocal fl, const double* __restrict__ FA, const double* __restrict__ dt,
    const unsigned long long* __restrict__ dtmin, int local_dt, int rep, const T* __restrict__ Jf,
    AssembleOut<T> out, double* __restrict__ rhs, T* __restrict__ rhs_t,
    double* __restrict__ partials) {
  const int nc = m.nc;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double b[5] = {0, 0, 0, 0, 0};
  double R[5] = {0, 0, 0, 0, 0};  // unscaled residual sum(+-F A), for convergence monitoring
  if (i < nc) {
    const double dti = local_dt ? dt[i] : __longlong_as_double((long long)*dtmin);
    const double k = dti * m.inv_vol[i];
    T D[25];
#pragma unroll
    for (int q = 0; q < 25; ++q) D[q] = (q % 6 == 0) ? T(1) : T(0);
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
      const int gf = m.gface[s * nc + i];
      if (gf == bes::kNoFace) continue;  // empty slot of a triangle
      const bool own = gf >= 0;
      const int f = own ? gf : ~gf;
      double fa[5];
      load_fa(FA, f, fa);
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        const double y = k * fa[v];
        b[v] = own ? b[v] - y : b[v] + y;
        R[v] = own ? R[v] + fa[v] : R[v] - fa[v];
      }
      const T mf = (T)(k * m.farea[f]), sm = own ? mf : -mf;
      T J[25];
      load_block(Jf, 2, own ? 0 : 1, f, J);
      add_scaled(J, sm, rep, D);
      if (f >= m.nf_int) continue;
      load_block(Jf, 2, own ? 1 : 0, f, J);
      T x[25];
#pragma unroll
      for (int q = 0; q < 25; ++q) x[q] = T(0);
      add_scaled(J, sm, rep, x);
      const int slot = 1 + (own ? fl.m_own[f] : fl.m_nb[f]);
      store_block(out.A, 5, slot, i, x);
      if (out.LU) store_block(out.LU, 5, slot, i, x);
      if constexpr (std::is_same<T, float>::value)
        if (out.A16) store_packed(out.A16, 5, slot, i, x);
    }
    store_block(out.A, 5, 0, i, D);
    if (out.LU) store_block(out.LU, 5, 0, i, D);
    if constexpr (std::is_same<T, float>::value)
      if (out.A16) store_packed(out.A16, 5, 0, i, D);
    if (out.Dinv) {
      T inv[25];
      inv5(D, inv);
      store_block(out.Dinv, 1, 0, i, inv);
      if constexpr (std::is_same<T, float>::value)
        if (out.D16) store_packed(out.D16, 1, 0, i, inv);
    }
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      rhs[(int64_t)v * nc + i] = b[v];
      rhs_t[(int64_t)i * 5 + v] = (T)b[v];
    }
  }
  __shared__ double sh[15][4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const double s2 = warp_sum(b[v] * b[v]);
    const double mx = warp_max(fabs(b[v]));
    const double r2 = warp_sum(R[v] * R[v]);
    if (lane == 0) {
      sh[v][wid] = s2;
      sh[5 + v][wid] = mx;
      sh[10 + v][wid] = r2;
    }
  }
  __syncthreads();
  if (threadIdx.x < 32) {
#pragma unroll
    for (int q = 0; q < 15; ++q) {
      double x = lane < 4 ? sh[q][lane] : 0.0;
      x = (q >= 5 && q < 10) ? warp_max(x) : warp_sum(x);
      // rows: 0-4 sum b^2, 5-9 max |b|, 10-14 sum R^2
      const int row = q < 5 ? q : (q < 10 ? q + 5 : q - 5);
      if (lane == 0) partials[(int64_t)row * gridDim.x + blockIdx.x] = x;
    }
  }
}

// Reduce `nvals` rows of per-block partials (sums, or maxima for rows >= nsum) in a fixed
// order; one block per value.  out[k] = sum (sqrt if sqrt_sums) or max.
static __global__ void __launch_bounds__(256) reduce_rows_kernel(const double* __restrict__ partials,
                                                          int nblocks, int nsum, int sqrt_sums,
                                                          double* __restrict__ out) {
  __shared__ double sh[8];
  const int k = blockIdx.x;
  const bool is_sum = k < nsum;
  double x = is_sum ? 0.0 : 0.0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x) {
    const double y = partials[(int64_t)k * nblocks + b];
    x = is_sum ? x + y : fmax(x, y);
  }
  x = is_sum ? warp_sum(x) : warp_max(x);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = x;
  __syncthreads();
  if (threadIdx.x < 32) {
    x = lane < 8 ? sh[lane] : 0.0;
    x = is_sum ? warp_sum(x) : warp_max(x);
    if (lane == 0) out[k] = (is_sum && sqrt_sums) ? sqrt(x) : x;
  }
}

// Colour-ordered block ILU(0), one colour per launch (rows of one colour are independent).
// IKJ order: the lower blocks of a row are eliminated in increasing factorisation position.
// RANGE: the stage is the contiguous row range [r0, r0 + nrows) and the factorisation
// position is the cell number (colour-major numbering), so no row list or position lookup.
template <class T, bool RANGE = false>
__global__ void __launch_bounds__(128) ilu_factor_kernel(DevMesh m, const int32_t* __restrict__ rows,
                                                         int nrows, const int32_t* __restrict__ pos,
                                                         T* __restrict__ A, T* __restrict__ Dinv,
                                                         int r0 = 0) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nrows) return;
  const int nc = m.nc;
  const int i = RANGE ? r0 + t : rows[t];
  const int pi = RANGE ? i : pos[i];
  int nbr[4], pn[4];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    nbr[s] = m.adj[s * nc + i];
    pn[s] = nbr[s] >= 0 ? (RANGE ? nbr[s] : pos[nbr[s]]) : 0x7fffffff;
  }
  // lower slots in increasing position: rank[s] = number of lower slots before slot s (the
  // neighbours are distinct cells, so positions are distinct).  All indexing of nbr / pn / rank
  // uses compile-time indices, so they stay in registers.
  bool low[4];
  int rank[4], nl = 0;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    low[s] = nbr[s] >= 0 && pn[s] < pi;
    nl += low[s];
  }
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    rank[s] = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t) rank[s] += (low[t] && pn[t] < pn[s]) ? 1 : 0;
  }
  for (int li = 0; li < nl; ++li) {
    int s = 0, j = 0, pj = 0;
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (low[t] && rank[t] == li) {
        s = t;
        j = nbr[t];
        pj = pn[t];
      }
    // blocks are loaded into registers before any store: A is read and written through one
    // pointer, so loads issued after a store could not be batched or reused
    T L[25], Ais[25], Dj[25];
    load_block(A, 5, 1 + s, i, Ais);
    load_block(Dinv, 1, 0, j, Dj);
#pragma unroll
    for (int r = 0; r < 5; ++r)
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        T acc = T(0);
#pragma unroll
        for (int k = 0; k < 5; ++k) acc += Ais[r * 5 + k] * Dj[k * 5 + c];
        L[r * 5 + c] = acc;
      }
    store_block(A, 5, 1 + s, i, L);
    // A_ik -= L_ij U_jk for every k in row i's pattern with pos(k) > pos(j) and (j,k) present
#pragma unroll 1
    for (int kk = -1; kk < 4; ++kk) {
      const int col = kk < 0 ? i : sel4(nbr, kk);
      if (kk >= 0 && (col < 0 || sel4(pn, kk) <= pj)) continue;
      int sj = -1;
      for (int q = 0; q < 4; ++q)
        if (m.adj[q * nc + j] == col) sj = q;
      if (sj < 0) continue;
      const int dst = kk < 0 ? 0 : 1 + kk;
      T U[25], Ad[25];
      load_block(A, 5, 1 + sj, j, U);
      load_block(A, 5, dst, i, Ad);
#pragma unroll
      for (int r = 0; r < 5; ++r)
#pragma unroll
        for (int c = 0; c < 5; ++c) {
          T acc = T(0);
#pragma unroll
          for (int k = 0; k < 5; ++k) acc += L[r * 5 + k] * U[k * 5 + c];
          Ad[r * 5 + c] -= acc;
        }
      store_block(A, 5, dst, i, Ad);
    }
  }
}

// inverse of the factored diagonal block of each row of a stage (after ilu_factor_kernel), and
// the row's packed copies (LU16, D16; null without them)
template <class T, bool RANGE = false>
__global__ void __launch_bounds__(128) ilu_invert_kernel(DevMesh m, const int32_t* __restrict__ rows,
                                                         int nrows, const T* __restrict__ A,
                                                         T* __restrict__ Dinv, uint32_t* __restrict__ LU16,
                                                         uint32_t* __restrict__ D16, int r0 = 0) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nrows) return;
  const int i = RANGE ? r0 + t : rows[t];
  T D[25], inv[25];
  load_block(A, 5, 0, i, D);
  inv5(D, inv);
  store_block(Dinv, 1, 0, i, inv);
  if constexpr (std::is_same<T, float>::value)
    if (LU16) {
      store_packed(D16, 1, 0, i, inv);
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {
        load_block(A, 5, 1 + s, i, D);
        store_packed(LU16, 4, s, i, D);
      }
    }
}

}  // namespace bes
