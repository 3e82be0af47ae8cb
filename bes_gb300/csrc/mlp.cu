// Learned warm start: a FiLM-conditioned coordinate MLP that predicts the converged flow field
// of a freestream condition from the solutions the solver produced for other conditions.
// There is no counterpart in the reference (it always starts from the freestream,
// Solver::setUniversalInitialCondition, include/Solver.hpp:71); the solver still converges
// from the predicted field and judges convergence, and a condition whose prediction is not
// physical (rho <= 0 or p <= 0 in some cell) falls back to the freestream.
//
// Network (the oracle's oracle/mlp_oracle.py restates it in FP64):
//   features  cell centroid x scaled to [-1, 1]^3 by the centroids' bounding box;
//             [sin(pi 2^k x_a), cos(pi 2^k x_a)], k = 0..7, at columns 16a + 2k (+1), x at
//             48..50, zeros up to 64;
//   condition c = (Mach vector - mean) / std over the training conditions;
//   4 hidden layers of width 256: z = h W^T + b; [gamma, beta] = c F^T + g;
//             y = z (1 + gamma) + beta; h = silu(y);
//   output    o = h W4^T + b4 (5 values) = (U - U_inf(c)) / scale.
// GEMMs run on the fifth-generation tensor cores (tcgen05.mma, BF16 operands, FP32
// accumulation in tensor memory) with BF16 copies of the weights and of the activations that
// feed them; everything else is FP32;
// AdamW keeps FP32 master weights.  All reductions are in a fixed order (no atomics), so a
// run is reproducible bit for bit.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "context.hpp"

namespace {

typedef __nv_bfloat16 bf16;

constexpr int kW = 256;        // hidden width
constexpr int kK0 = 64;        // input features
constexpr int kLayers = 4;     // hidden layers
constexpr int kOut = 5;
constexpr int kRowTile = 128;  // rows (samples) per GEMM tile; batches are multiples of it
constexpr int kChunk = 64;     // rows per partial sum of the column reductions

// ---- parameter layout (flat FP32), the order of oracle/mlp_oracle.py layout() ----------------
struct Layout {
  int64_t W[5], b[5], F[4], g[4], n;
  Layout() {
    int64_t off = 0;
    for (int l = 0; l < kLayers; ++l) {
      const int k = l == 0 ? kK0 : kW;
      W[l] = off; off += (int64_t)kW * k;
      b[l] = off; off += kW;
      F[l] = off; off += 2 * kW * 3;
      g[l] = off; off += 2 * kW;
    }
    W[4] = off; off += kOut * kW;
    b[4] = off; off += kOut;
    n = off;
  }
};

// ---- deterministic hashing (splitmix64) ------------------------------------------------------
__host__ __device__ inline uint64_t mix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

__device__ __forceinline__ float silu(float y) { return y / (1.0f + __expf(-y)); }
__device__ __forceinline__ float dsilu(float y) {
  const float s = 1.0f / (1.0f + __expf(-y));
  return s * (1.0f + y * (1.0f - s));
}

// ---- tensor-core GEMM building blocks (tcgen05, accumulators in tensor memory) -----------------
// Every operand is K-major in global memory (the dimension that is summed is contiguous), so
// staging is a copy of 16-byte pieces: a tile of R rows and K values of the summed dimension
// lies in shared memory as 8x8 core matrices without swizzle, value (r, k) at byte
// (r/8) * sbo + (k/8) * 128 + (r%8) * 16 + (k%8) * 2 with sbo = K/8 * 128.  The whole of K (or 512
// values of it) is staged by cp.async at once, one thread issues the tcgen05.mma of all its
// slices of 16 and commits them to an mbarrier, and the warps read the accumulator back with
// tcgen05.ld.  Every wait on the mbarrier gives up after two seconds and sets *err.
constexpr int kCoreBytes = 128;  // an 8 x 8 core matrix of 16-bit values

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: K-major, no swizzle, start address and the two strides (next
// 8 values of k: one core matrix; next 8 rows: sbo)
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr, int sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)((kCoreBytes >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of this architecture
  return d;                // base offset 0, layout type 0 (no swizzle)
}

// instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both K-major, M x N
__host__ __device__ constexpr uint32_t umma_idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ unsigned long long ns_now() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// wait for phase `parity` of the mbarrier; false after two seconds
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  const unsigned long long t0 = ns_now();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
    if (ns_now() - t0 > 2000000000ull) return false;
  }
}

// Stage rows r0 .. r0 + rows - 1, values k0 .. k0 + K - 1 of src [..][ld] into sm (not waited for).
// KC: K where it is known at compile time (the index arithmetic of a piece is then shifts), or 0.
template <int KC>
__device__ __forceinline__ void stage_async(uint32_t sm, const bf16* __restrict__ src, int64_t ld,
                                            int64_t r0, int rows, int64_t k0, int K) {
  const int per = KC ? KC / 8 : K / 8;
  const bf16* base = src + r0 * ld + k0;
#pragma unroll 8
  for (int v = threadIdx.x; v < rows * per; v += blockDim.x) {
    // eight consecutive threads take eight rows of one core matrix (128 consecutive bytes)
    const int r = (v / (8 * per)) * 8 + (v & 7), seg = (v >> 3) % per;
    const uint32_t dst = sm + (r >> 3) * (per * kCoreBytes) + seg * kCoreBytes + (r & 7) * 16;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n"
                 :: "r"(dst), "l"(base + r * ld + seg * 8) : "memory");
  }
}
__device__ __forceinline__ void stage_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// The staged values are there, and visible to the tensor core (async proxy), for every thread.
__device__ __forceinline__ void stage_wait() {
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  __syncthreads();
}

// Tensor memory and the mbarrier of a CTA.
struct TensorCta {
  uint32_t tmem, mbar, phase;
};
template <int COLS>
__device__ __forceinline__ TensorCta tensor_open(uint64_t* mbar, uint32_t* base) {
  const uint32_t mb = smem_u32(mbar);
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n"
                 :: "r"(smem_u32(base)), "n"(COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" :: "r"(mb) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  return TensorCta{*base, mb, 0u};
}
template <int COLS>
__device__ __forceinline__ void tensor_close(const TensorCta& t) {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" :: "r"(t.tmem), "n"(COLS)
                 : "memory");
}
// D (128 x N) = (acc: +=) A B over K staged values, in slices of 16 in increasing k; false if
// the tensor core did not finish within two seconds (the same verdict for every thread).
template <int N>
__device__ __forceinline__ bool tensor_mma(TensorCta& t, uint32_t a, uint32_t b, int K, bool acc) {
  constexpr uint32_t idesc = umma_idesc(128, N);
  if (threadIdx.x == 0) {
    const int sbo = K / 8 * kCoreBytes;
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    for (int kk = 0; kk < K / 16; ++kk) {
      const uint64_t ad = umma_desc(a + kk * 2 * kCoreBytes, sbo);
      const uint64_t bd = umma_desc(b + kk * 2 * kCoreBytes, sbo);
      const uint32_t on = (acc || kk > 0) ? 1u : 0u;
      asm volatile(
          "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
          " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
          :: "r"(t.tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(on) : "memory");
    }
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n"
                 :: "r"(t.mbar) : "memory");
  }
  const int done = mbar_wait(t.mbar, t.phase) ? 1 : 0;
  t.phase ^= 1;
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  return __syncthreads_and(done) != 0;
}
// 16 accumulator columns from c0 of this warp's 32 rows (rows 32 (warp % 4) + lane)
__device__ __forceinline__ void tensor_read16(const TensorCta& t, int c0, float* x) {
  uint32_t r[16];
  const uint32_t addr = t.tmem + ((uint32_t)(((threadIdx.x >> 5) & 3) * 32) << 16) + (uint32_t)c0;
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
        "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int q = 0; q < 16; ++q) x[q] = __uint_as_float(r[q]);
}

// FiLM of one layer and column j (F [512][3], g [512]): gamma, then beta.
struct Film {
  float f0, f1, f2, e0, e1, e2, gj, bj, bias;
};
__device__ __forceinline__ float film_gamma(const Film& f, float c0, float c1, float c2) {
  return f.f0 * c0 + f.f1 * c1 + f.f2 * c2 + f.gj;
}
__device__ __forceinline__ float film_beta(const Film& f, float c0, float c1, float c2) {
  return f.e0 * c0 + f.e1 * c1 + f.e2 * c2 + f.bj;
}
__device__ __forceinline__ Film load_film(const float* __restrict__ bias, const float* __restrict__ F,
                                          const float* __restrict__ g, int j) {
  return Film{F[j * 3], F[j * 3 + 1], F[j * 3 + 2], F[(kW + j) * 3], F[(kW + j) * 3 + 1],
              F[(kW + j) * 3 + 2], g[j], g[kW + j], bias[j]};
}

// ---- forward: all layers of a block of rows in one CTA --------------------------------------------
struct ForwardArgs {
  const bf16* X;              // features [rows][64]
  const bf16* Wb[kLayers];    // BF16 weights [256][K]
  const float* p;             // parameters (biases, FiLM, output layer)
  Layout L;
  const float* C;             // conditions [rows][3] (training)
  float c3[3];                // the condition of every row (inference)
  int64_t ldt;                // row stride of the transposed arrays (training)
  float* ZT[kLayers];         // z = h W^T + b, transposed [256][ldt]
  bf16* HT[kLayers];          // silu(y), transposed [256][ldt]
  const float* T;             // targets [rows][5]
  float* O;                   // outputs [rows][8]
  float* dO;                  // d loss / d output [rows][8]
  double* row_loss;           // squared errors of a row
  float B;                    // rows of the batch
  double* U;                  // inference: predicted states [n][5]
  int64_t n;                  // inference: rows with a cell behind them
  double Uinf[kOut], oscale[kOut];
  int* err;
};

constexpr int kFwdThreads = 1024;
constexpr int kFwdCols = kW / (kFwdThreads / 128);  // columns of a warp's epilogue
constexpr int kSmW = kW * kW * 2, kSmA = kRowTile * kW * 2;
constexpr int kSmFilm = 2 * kW * 12 * 4, kSmC = kRowTile * 3 * 4, kSmW4 = kOut * kW * 4;
constexpr int kFwdSmem = kSmW + kSmA + kSmFilm + kSmC + kSmW4 + kRowTile * kOut * 4;

// A CTA owns ROWS rows and every column: the activations stay in shared memory as the next
// layer's A operand (rows beyond ROWS of the 128-row MMA are not read back), the next layer's
// weights are fetched while a layer's epilogue (FiLM, SiLU) runs, and the output layer ends the
// kernel.  Four GEMM and four FiLM launches took 100 us on 8,192 rows, bound by waiting for one
// 64-wide slice after the other and by writing and reading z; what bounds it now is the
// epilogue's exponentials and divisions.  ROWS 64 where 128 would leave SMs idle.
template <int ROWS, bool TRAIN>
__global__ void __launch_bounds__(kFwdThreads, 1) mlp_forward_kernel(const __grid_constant__ ForwardArgs a) {
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t* sW = sm;
  uint8_t* sA = sm + kSmW;
  float* film = reinterpret_cast<float*>(sm + kSmW + kSmA);  // two layers of [256][12]
  float* sC = film + 2 * kW * 12;
  float* w4 = sC + kRowTile * 3;
  float* so = w4 + kOut * kW;
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t r0 = (int64_t)blockIdx.x * ROWS;
  const uint32_t uW = smem_u32(sW), uA = smem_u32(sA);
  stage_async<kK0>(uA, a.X, kK0, r0, ROWS, 0, kK0);
  stage_async<kK0>(uW, a.Wb[0], kK0, 0, kW, 0, kK0);
  stage_commit();
  auto load_layer = [&](int l) {
    if (tid < kW) {
      const Film f = load_film(a.p + a.L.b[l], a.p + a.L.F[l], a.p + a.L.g[l], tid);
      float* d = film + ((l & 1) * kW + tid) * 12;
      if (!TRAIN) {
        // one condition for every row: gamma and beta are the column's
        reinterpret_cast<float4*>(d)[0] =
            make_float4(f.bias, film_gamma(f, a.c3[0], a.c3[1], a.c3[2]), film_beta(f, a.c3[0], a.c3[1], a.c3[2]), 0.0f);
        return;
      }
      reinterpret_cast<float4*>(d)[0] = make_float4(f.bias, f.f0, f.f1, f.f2);
      reinterpret_cast<float4*>(d)[1] = make_float4(f.gj, f.e0, f.e1, f.e2);
      d[8] = f.bj;
    }
  };
  load_layer(0);
  for (int q = tid; q < ROWS * 3; q += kFwdThreads) sC[q] = TRAIN ? a.C[r0 * 3 + q] : a.c3[q % 3];
  for (int q = tid; q < kOut * kW; q += kFwdThreads) w4[q] = a.p[a.L.W[kLayers] + q];
  TensorCta t = tensor_open<kW>(&mbar, &tmem_base);
  const int row = (warp & 3) * 32 + lane, col0 = (warp >> 2) * kFwdCols;
  bool ok = true;
  for (int l = 0; l < kLayers && ok; ++l) {
    const int K = l == 0 ? kK0 : kW;
    stage_wait();
    ok = tensor_mma<kW>(t, uA, uW, K, false);
    if (!ok) break;
    if (l + 1 < kLayers) {
      stage_async<kW>(uW, a.Wb[l + 1], kW, 0, kW, 0, kW);
      stage_commit();
      load_layer(l + 1);
    }
    if ((warp & 3) * 32 < ROWS) {
      const float c0 = sC[row * 3], c1 = sC[row * 3 + 1], c2 = sC[row * 3 + 2];
      const float* fl = film + (l & 1) * kW * 12;
#pragma unroll 1
      for (int cc = 0; cc < kFwdCols; cc += 16) {
        float x[16];
        tensor_read16(t, col0 + cc, x);
        uint32_t packed[8];
#pragma unroll
        for (int q = 0; q < 16; ++q) {
          const int j = col0 + cc + q;
          const float4 fa = reinterpret_cast<const float4*>(fl + j * 12)[0];
          float gam = fa.y, bet = fa.z;
          if (TRAIN) {
            const float4 fb = reinterpret_cast<const float4*>(fl + j * 12)[1];
            const Film f{fa.y, fa.z, fa.w, fb.y, fb.z, fb.w, fb.x, fl[j * 12 + 8], fa.x};
            gam = film_gamma(f, c0, c1, c2);
            bet = film_beta(f, c0, c1, c2);
          }
          const float z = x[q] + fa.x;
          const float y = z * (1.0f + gam) + bet;
          const bf16 h = __float2bfloat16(silu(y));
          if (TRAIN) {
            a.ZT[l][j * a.ldt + r0 + row] = z;
            a.HT[l][j * a.ldt + r0 + row] = h;
          }
          const uint32_t hb = (uint32_t)__bfloat16_as_ushort(h);
          if (q & 1) packed[q >> 1] |= hb << 16;
          else packed[q >> 1] = hb;
        }
        uint8_t* dst = sA + (row >> 3) * (kW / 8 * kCoreBytes) + ((col0 + cc) >> 3) * kCoreBytes + (row & 7) * 16;
        *reinterpret_cast<uint4*>(dst) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        *reinterpret_cast<uint4*>(dst + kCoreBytes) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  }
  if (!ok && tid == 0) atomicExch(a.err, 1);
  __syncthreads();
  // output layer: one thread per row and output, k in increasing order
  for (int q = tid; ok && q < ROWS * kOut; q += kFwdThreads) {
    const int v = q / ROWS, r = q - v * ROWS;
    float o = a.p[a.L.b[kLayers] + v];
    const uint8_t* src = sA + (r >> 3) * (kW / 8 * kCoreBytes) + (r & 7) * 16;
    for (int k = 0; k < kW; k += 8) {
      const uint4 x = *reinterpret_cast<const uint4*>(src + (k >> 3) * kCoreBytes);
      const bf16* e = reinterpret_cast<const bf16*>(&x);
#pragma unroll
      for (int i = 0; i < 8; ++i) o += __bfloat162float(e[i]) * w4[v * kW + k + i];
    }
    if (TRAIN) {
      so[r * kOut + v] = o;
    } else if (r0 + r < a.n) {
      // on the host's arithmetic: no contraction
      a.U[(r0 + r) * kOut + v] = __dadd_rn(a.Uinf[v], __dmul_rn(a.oscale[v], (double)o));
    }
  }
  if (TRAIN) {
    __syncthreads();
    if (ok && tid < ROWS) {
      double l = 0.0;
#pragma unroll
      for (int v = 0; v < kOut; ++v) {
        const float o = so[tid * kOut + v];
        const float d = o - a.T[(r0 + tid) * kOut + v];
        a.O[(r0 + tid) * 8 + v] = o;
        a.dO[(r0 + tid) * 8 + v] = 2.0f * d / (5.0f * a.B);
        l += (double)d * (double)d;
      }
      a.row_loss[r0 + tid] = l;
    }
  }
  tensor_close<kW>(t);
}

// ---- backward ----------------------------------------------------------------------------------------

// dH (transposed [256][ldt]) = dZ [rows][256] W: 128 rows and 128 columns per CTA, all of K staged
// at once.  WT: W transposed [256 (n)][256 (k)].
constexpr int kDhSmem = 2 * kRowTile * kW * 2;
__global__ void __launch_bounds__(256, 1) mlp_dh_kernel(const bf16* __restrict__ dZ,
                                                        const bf16* __restrict__ WT,
                                                        float* __restrict__ dHT, int64_t ldt, int* err) {
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_base;
  const int64_t r0 = (int64_t)blockIdx.y * kRowTile;
  const int n0 = blockIdx.x * 128;
  const uint32_t uA = smem_u32(sm), uB = uA + kRowTile * kW * 2;
  stage_async<kW>(uA, dZ, kW, r0, kRowTile, 0, kW);
  stage_async<kW>(uB, WT, kW, n0, 128, 0, kW);
  stage_commit();
  TensorCta t = tensor_open<128>(&mbar, &tmem_base);
  stage_wait();
  const bool ok = tensor_mma<128>(t, uA, uB, kW, false);
  if (!ok && threadIdx.x == 0) atomicExch(err, 1);
  if (ok) {
    const int warp = threadIdx.x >> 5, row = (warp & 3) * 32 + (threadIdx.x & 31), c0 = (warp >> 2) * 64;
#pragma unroll
    for (int cc = 0; cc < 64; cc += 16) {
      float x[16];
      tensor_read16(t, c0 + cc, x);
#pragma unroll
      for (int q = 0; q < 16; ++q) dHT[(int64_t)(n0 + c0 + cc + q) * ldt + r0 + row] = x[q];
    }
  }
  tensor_close<128>(t);
}

// Weight gradients dW_l = dZ_l^T H_l of every layer: a CTA takes 128 x 64 of one layer's matrix and
// one split of the rows (512 of them, or the whole batch in pieces of 512), both operands from
// their transposed copies.  wpart: per layer [split][256][K_l].
struct DwArgs {
  const bf16 *dZT[kLayers], *HT[kLayers];  // [256][ldt], [K_l][ldt]
  float* wpart[kLayers];
  int64_t ldt, k_split;
  int splits;
  int* err;
};
constexpr int kDwSlice = 512;
constexpr int kDwSmem = (128 + 64) * kDwSlice * 2;
__global__ void __launch_bounds__(256, 1) mlp_dw_kernel(const __grid_constant__ DwArgs a) {
  extern __shared__ __align__(1024) uint8_t sm[];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ uint32_t tmem_base;
  // tiles of a split: 2 x 4 of each layer above the first, 2 x 1 of the first
  const int tile = blockIdx.x, l = tile < 24 ? 1 + tile / 8 : 0;
  const int m0 = ((tile < 24 ? tile % 8 : tile - 24) & 1) * 128;
  const int n0 = l == 0 ? 0 : ((tile % 8) >> 1) * 64;
  const int K = l == 0 ? kK0 : kW;
  const int64_t k_begin = (int64_t)blockIdx.y * a.k_split, k_end = k_begin + a.k_split;
  const uint32_t uA = smem_u32(sm), uB = uA + 128 * kDwSlice * 2;
  TensorCta t = tensor_open<64>(&mbar, &tmem_base);
  bool ok = true;
  for (int64_t k0 = k_begin; k0 < k_end && ok; k0 += kDwSlice) {
    const int n = (int)(k_end - k0 < kDwSlice ? k_end - k0 : kDwSlice);
    if (n == kDwSlice) {
      stage_async<kDwSlice>(uA, a.dZT[l], a.ldt, m0, 128, k0, n);
      stage_async<kDwSlice>(uB, a.HT[l], a.ldt, n0, 64, k0, n);
    } else {
      stage_async<0>(uA, a.dZT[l], a.ldt, m0, 128, k0, n);
      stage_async<0>(uB, a.HT[l], a.ldt, n0, 64, k0, n);
    }
    stage_commit();
    stage_wait();
    ok = tensor_mma<64>(t, uA, uB, n, k0 > k_begin);
  }
  if (!ok && threadIdx.x == 0) atomicExch(a.err, 1);
  if (ok) {
    const int warp = threadIdx.x >> 5, row = (warp & 3) * 32 + (threadIdx.x & 31), c0 = (warp >> 2) * 32;
    float* dst = a.wpart[l] + ((int64_t)blockIdx.y * kW + m0 + row) * K + n0 + c0;
#pragma unroll
    for (int cc = 0; cc < 32; cc += 16) {
      float x[16];
      tensor_read16(t, c0 + cc, x);
#pragma unroll
      for (int q = 0; q < 16; q += 4)
        *reinterpret_cast<float4*>(dst + cc + q) = make_float4(x[q], x[q + 1], x[q + 2], x[q + 3]);
    }
  }
  tensor_close<64>(t);
}

// ---- elementwise and reduction kernels -------------------------------------------------------

// features of every cell: bf16 [n_rows][64] (rows beyond n_cells are zero)
__global__ void encode_kernel(int n_cells, int n_rows, const float* __restrict__ xn,
                              bf16* __restrict__ feat) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_rows) return;
  float f[kK0];
#pragma unroll
  for (int q = 0; q < kK0; ++q) f[q] = 0.0f;
  if (i < n_cells) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const double x = xn[i * 3 + a];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const double w = 3.141592653589793 * (double)(1 << k) * x;
        f[16 * a + 2 * k] = (float)sin(w);
        f[16 * a + 2 * k + 1] = (float)cos(w);
      }
      f[48 + a] = (float)x;
    }
  }
#pragma unroll
  for (int q = 0; q < kK0; ++q) feat[(size_t)i * kK0 + q] = __float2bfloat16(f[q]);
}

// One row of a batch: its features (and their transposed copy, the weight gradient's operand).
__device__ __forceinline__ void gather_row(int64_t r, int64_t cell, int64_t ldt, const bf16* __restrict__ feat,
                                           bf16* __restrict__ H0, bf16* __restrict__ H0T) {
  const uint4* src = reinterpret_cast<const uint4*>(feat + cell * kK0);
  uint4* dst = reinterpret_cast<uint4*>(H0 + r * kK0);
#pragma unroll
  for (int q = 0; q < kK0 / 8; ++q) {
    const uint4 x = src[q];
    dst[q] = x;
    const bf16* e = reinterpret_cast<const bf16*>(&x);
#pragma unroll
    for (int i = 0; i < 8; ++i) H0T[(q * 8 + i) * ldt + r] = e[i];
  }
}

// Training batch: row r draws (sample, cell) from a hash of (seed, step, r).
__global__ void gather_kernel(int B, uint64_t seed, int64_t step, int n_samples, int n_cells,
                              const bf16* __restrict__ feat, const float* __restrict__ targets,
                              const float* __restrict__ cond, bf16* __restrict__ H0,
                              bf16* __restrict__ H0T, int64_t ldt, float* __restrict__ C,
                              float* __restrict__ T) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= B) return;
  const uint64_t h = mix64(seed ^ mix64((uint64_t)step * 0x100000001B3ull + (uint64_t)r));
  const int s = (int)((h & 0xffffffffull) % (uint64_t)n_samples);
  const int c = (int)((h >> 32) % (uint64_t)n_cells);
  gather_row(r, c, ldt, feat, H0, H0T);
#pragma unroll
  for (int a = 0; a < 3; ++a) C[r * 3 + a] = cond[s * 3 + a];
#pragma unroll
  for (int v = 0; v < kOut; ++v) T[r * kOut + v] = targets[((size_t)s * n_cells + c) * kOut + v];
}
// Rows given by their cells.
__global__ void gather_cells_kernel(int B, const int64_t* __restrict__ cells, const bf16* __restrict__ feat,
                                    bf16* __restrict__ H0, bf16* __restrict__ H0T, int64_t ldt) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r < B) gather_row(r, cells[r], ldt, feat, H0, H0T);
}
// Training targets (U - U_inf) / scale in FP32, from the solutions as given.
__global__ void targets_kernel(int64_t per_sample, int64_t n, const double* __restrict__ U,
                               const double* __restrict__ Uinf, const double* __restrict__ oscale,
                               float* __restrict__ T) {
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (int64_t)gridDim.x * blockDim.x) {
    const int v = (int)(k % kOut);
    T[k] = (float)((U[k] - Uinf[k / per_sample * kOut + v]) / oscale[v]);
  }
}

// FiLM + SiLU backward of layer l for a chunk of 64 rows, thread j the column j, rows in increasing
// order: dZ in BF16 (by rows, the next dH GEMM's operand, and transposed, the weight gradient's)
// and the chunk's partial sums part[chunk][9][256]: row 0 db, rows 1..3 dF of gamma, rows 4..6 dF of
// beta, row 7 dg of gamma, row 8 dg of beta.  OUT: the last layer; dH = dO W4 is formed here,
// with the partials part4[chunk][5*256 + 5] of dW4 / db4, and the first blocks add up the rows'
// losses (256 rows per partial).  The transposed inputs give a thread its rows in 16-byte loads
// that do not wait for one another (one row after the other: 53 us on 8,192 rows).
struct FilmBackArgs {
  int B;
  int64_t ldt;
  const float* dHT;           // [256][ldt]
  const float* ZT;
  const float *bias, *F, *g, *C;
  bf16 *dZ, *dZT;             // dZ null for the first layer
  float* part;
  const float *dO, *W4;       // OUT
  const bf16* HT;
  float* part4;
  const double* row_loss;
  double* loss_part;
};
template <bool OUT>
__global__ void __launch_bounds__(256) film_backward_kernel(const __grid_constant__ FilmBackArgs a) {
  __shared__ float sC[kChunk * 3], sdO[kChunk * kOut];
  const int j = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.x * kChunk;  // B is a multiple of 128
  for (int q = j; q < kChunk * 3; q += kW) sC[q] = a.C[r0 * 3 + q];
  if (OUT)
    for (int q = j; q < kChunk * kOut; q += kW) sdO[q] = a.dO[(r0 + q / kOut) * 8 + q % kOut];
  const Film f = load_film(a.bias, a.F, a.g, j);
  float w[kOut] = {}, aw[kOut] = {}, ab[kOut] = {};
  if (OUT)
#pragma unroll
    for (int v = 0; v < kOut; ++v) w[v] = a.W4[v * kW + j];
  float s8[8] = {0, 0, 0, 0, 0, 0, 0, 0}, db = 0.0f;
  __syncthreads();
  const float4* zp = reinterpret_cast<const float4*>(a.ZT + j * a.ldt + r0);
  const float4* hp = OUT ? nullptr : reinterpret_cast<const float4*>(a.dHT + j * a.ldt + r0);
  const uint4* h4 = OUT ? reinterpret_cast<const uint4*>(a.HT + j * a.ldt + r0) : nullptr;
#pragma unroll 2
  for (int q = 0; q < kChunk / 8; ++q) {
    const float4 z0 = zp[2 * q], z1 = zp[2 * q + 1];
    const float zz[8] = {z0.x, z0.y, z0.z, z0.w, z1.x, z1.y, z1.z, z1.w};
    float dh[8];
    uint4 hw = make_uint4(0, 0, 0, 0);
    if (OUT) {
      hw = h4[q];
    } else {
      const float4 d0 = hp[2 * q], d1 = hp[2 * q + 1];
      dh[0] = d0.x; dh[1] = d0.y; dh[2] = d0.z; dh[3] = d0.w;
      dh[4] = d1.x; dh[5] = d1.y; dh[6] = d1.z; dh[7] = d1.w;
    }
    const bf16* he = reinterpret_cast<const bf16*>(&hw);
    uint32_t packed[4];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = q * 8 + i;
      if (OUT) {
        const float h = __bfloat162float(he[i]);
        float s = 0.0f;
#pragma unroll
        for (int v = 0; v < kOut; ++v) {
          const float d = sdO[r * kOut + v];
          s += d * w[v];
          aw[v] += d * h;
          ab[v] += d;
        }
        dh[i] = s;
      }
      const float c0 = sC[r * 3], c1 = sC[r * 3 + 1], c2 = sC[r * 3 + 2];
      const float gam = film_gamma(f, c0, c1, c2), bet = film_beta(f, c0, c1, c2);
      const float z = zz[i];
      const float y = z * (1.0f + gam) + bet;
      const float dy = dh[i] * dsilu(y);
      const float dz = dy * (1.0f + gam);
      const float dgam = dy * z;
      const bf16 b = __float2bfloat16(dz);
      if (a.dZ) a.dZ[(r0 + r) * kW + j] = b;
      const uint32_t bits = (uint32_t)__bfloat16_as_ushort(b);
      if (i & 1) packed[i >> 1] |= bits << 16;
      else packed[i >> 1] = bits;
      db += dz;
      s8[0] += dgam * c0;
      s8[1] += dgam * c1;
      s8[2] += dgam * c2;
      s8[3] += dy * c0;
      s8[4] += dy * c1;
      s8[5] += dy * c2;
      s8[6] += dgam;
      s8[7] += dy;
    }
    *reinterpret_cast<uint4*>(a.dZT + j * a.ldt + r0 + q * 8) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
  }
  float* p = a.part + (size_t)blockIdx.x * 9 * kW;
  p[j] = db;
#pragma unroll
  for (int k = 0; k < 8; ++k) p[(1 + k) * kW + j] = s8[k];
  if (OUT) {
    float* p4 = a.part4 + (size_t)blockIdx.x * (kOut * kW + kOut);
#pragma unroll
    for (int v = 0; v < kOut; ++v) p4[v * kW + j] = aw[v];
#pragma unroll
    for (int v = 0; v < kOut; ++v)
      if (j == v) p4[kOut * kW + v] = ab[v];
    // the loss of rows 256 b .. 256 b + 255, summed as a tree
    if ((int64_t)blockIdx.x * 256 < a.B) {
      __shared__ double red[256];
      const int64_t r = (int64_t)blockIdx.x * 256 + j;
      red[j] = r < a.B ? a.row_loss[r] : 0.0;
      __syncthreads();
      for (int s = 128; s > 0; s >>= 1) {
        if (j < s) red[j] += red[j + s];
        __syncthreads();
      }
      if (j == 0) a.loss_part[blockIdx.x] = red[0] / (5.0 * (double)a.B);
    }
  }
}

// AdamW on one parameter (decoupled weight decay where decay != 0).
__device__ __forceinline__ float adamw_one(float p, float gi, float* __restrict__ m, float* __restrict__ v,
                                           bool decay, float lr, float wd, float bc1, float bc2) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float mi = b1 * *m + (1.0f - b1) * gi;
  const float vi = b2 * *v + (1.0f - b2) * gi * gi;
  *m = mi;
  *v = vi;
  const float upd = (mi / bc1) / (sqrtf(vi / bc2) + eps) + (decay ? wd * p : 0.0f);
  return p - lr * upd;
}

struct UpdateArgs {
  Layout L;
  int64_t n;
  float *p, *grad, *m, *v;
  const uint8_t* decay;
  bf16 *Wb[kLayers], *WT[kLayers];  // BF16 copies of the hidden weights, as they are and transposed
  // partial sums of the gradient (REDUCE)
  const float* wpart[kLayers];
  const float* part[kLayers];
  const float* part4;
  int splits, chunks;
  float lr, wd, bc1, bc2;
};
// out = sum over q < n of src[q * stride], in increasing q, the loads sixteen at a time
__device__ __forceinline__ float sum_rows(const float* __restrict__ src, int64_t stride, int n) {
  float s = 0.0f;
  int q = 0;
  for (; q + 16 <= n; q += 16) {
    float x[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) x[e] = src[(q + e) * stride];
#pragma unroll
    for (int e = 0; e < 16; ++e) s += x[e];
  }
  for (; q < n; ++q) s += src[q * stride];
  return s;
}
// One thread per parameter: its gradient from the partial sums (REDUCE), the AdamW step (STEP) and
// the BF16 copies.
template <bool REDUCE, bool STEP>
__global__ void __launch_bounds__(256) update_params_kernel(const __grid_constant__ UpdateArgs a) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.n) return;
  int l = 0;
  while (l < kLayers && i >= a.L.W[l + 1]) ++l;  // the layer of parameter i (kLayers: output layer)
  const int64_t e = i - a.L.W[l];
  const int K = l == 0 ? kK0 : kW;
  const bool weight = l < kLayers && e < (int64_t)kW * K;
  float gi;
  if (REDUCE) {
    if (l == kLayers) {
      gi = sum_rows(a.part4 + e, kOut * kW + kOut, a.chunks);
    } else if (weight) {
      gi = sum_rows(a.wpart[l] + e, (int64_t)kW * K, a.splits);
    } else {
      // position in the partial sums [9][256]
      int at;
      if (i < a.L.F[l]) {
        at = (int)(i - a.L.b[l]);
      } else if (i < a.L.g[l]) {
        const int q = (int)(i - a.L.F[l]), j = q / 3, d = q - 3 * j;
        at = j < kW ? (1 + d) * kW + j : (4 + d) * kW + j - kW;
      } else {
        const int q = (int)(i - a.L.g[l]);
        at = q < kW ? 7 * kW + q : 8 * kW + q - kW;
      }
      gi = sum_rows(a.part[l] + at, 9 * kW, a.chunks);
    }
    a.grad[i] = gi;
  } else {
    gi = a.grad[i];
  }
  float p = a.p[i];
  if (STEP) {
    p = adamw_one(p, gi, a.m + i, a.v + i, a.decay[i] != 0, a.lr, a.wd, a.bc1, a.bc2);
    a.p[i] = p;
  }
  if (weight && (STEP || !REDUCE)) {
    const bf16 b = __float2bfloat16(p);
    a.Wb[l][e] = b;
    const int64_t m = e / K, k = e - m * K;
    a.WT[l][k * kW + m] = b;
  }
}

}  // namespace

// ---- the handle ------------------------------------------------------------------------------
struct bes_mlp {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string last_error;
  std::vector<void*> allocs, batch_allocs;
  int64_t nc = 0, n_rows = 0;  // cells, cells rounded up to the row tile
  double gamma = 1.4, R = 287.0;
  Layout L;
  float* feat_xn = nullptr;  // [nc][3] scaled centroids (reference numbering)
  bf16* feat = nullptr;      // [n_rows][64]
  float* p = nullptr;        // parameters, gradient, AdamW moments
  float* grad = nullptr;
  float* m = nullptr;
  float* v = nullptr;
  uint8_t* decay = nullptr;
  bf16 *Wb[kLayers] = {}, *WT[kLayers] = {};  // BF16 copies of the hidden weights, as they are and transposed
  int64_t t = 0;             // AdamW steps taken
  double cmean[3] = {0, 0, 0}, csd[3] = {1, 1, 1}, oscale[kOut] = {1, 1, 1, 1, 1};
  double* ustage[2] = {};    // fields [nc][5] on their way to or from the caller
  cudaStream_t copy = nullptr;               // the predictions' way out
  cudaEvent_t ready[2] = {}, taken[2] = {};  // a field is complete, is copied
  // batch buffers (capacity in rows; transposed arrays have rows of `cap` values)
  int cap = 0;
  bf16 *H0 = nullptr, *H0T = nullptr;  // features of the batch
  float* ZT[kLayers] = {};
  bf16 *HT[kLayers] = {}, *dZT[kLayers] = {};
  float *C = nullptr, *T = nullptr, *O = nullptr, *dO = nullptr, *dHT = nullptr;
  bf16* dZ = nullptr;
  float *part[kLayers] = {}, *part4 = nullptr, *wpart[kLayers] = {};
  double *row_loss = nullptr, *loss_part = nullptr;
  int* gemm_err = nullptr;   // set by a GEMM whose tensor-core wait gave up
};

namespace {

#define MLP_TRY(h, call)                                                         \
  do {                                                                           \
    cudaError_t e_ = (call);                                                     \
    if (e_ != cudaSuccess) {                                                     \
      (h)->last_error = std::string(#call) + ": " + cudaGetErrorString(e_);      \
      return BES_ERR_CUDA;                                                       \
    }                                                                            \
  } while (0)

// BES_ERR_TIMEOUT (and the flag cleared) if a GEMM's wait on the tensor core gave up
int gemm_status(bes_mlp* h) {
  int e = 0;
  MLP_TRY(h, cudaMemcpy(&e, h->gemm_err, sizeof(int), cudaMemcpyDeviceToHost));
  if (!e) return BES_OK;
  cudaMemset(h->gemm_err, 0, sizeof(int));
  h->last_error = "a tensor-core GEMM stopped waiting for its products after two seconds";
  return BES_ERR_TIMEOUT;
}

template <class X>
int mlp_alloc(bes_mlp* h, X** ptr, size_t count, std::vector<void*>& list) {
  *ptr = nullptr;
  cudaError_t e = cudaMalloc((void**)ptr, std::max<size_t>(count, 1) * sizeof(X));
  if (e != cudaSuccess) {
    cudaGetLastError();  // not the next call's
    h->last_error = std::string("cudaMalloc: ") + cudaGetErrorString(e);
    return BES_ERR_CUDA;
  }
  list.push_back(*ptr);
  return BES_OK;
}
template <class X>
int mlp_alloc(bes_mlp* h, X** ptr, size_t count) {
  return mlp_alloc(h, ptr, count, h->allocs);
}

void free_batch(bes_mlp* h) {
  for (void* q : h->batch_allocs) cudaFree(q);
  h->batch_allocs.clear();
  h->cap = 0;
}

// Buffers for batches of B rows: all of them or none, in place of smaller ones.
int ensure_batch(bes_mlp* h, int B) {
  if (B <= h->cap) return BES_OK;
  free_batch(h);
  int rc = 0;
  auto alloc = [&](auto** ptr, size_t count) { rc |= mlp_alloc(h, ptr, count, h->batch_allocs); };
  alloc(&h->H0, (size_t)B * kK0);
  alloc(&h->H0T, (size_t)B * kK0);
  const int chunks = B / kChunk;
  for (int l = 0; l < kLayers; ++l) {
    alloc(&h->ZT[l], (size_t)B * kW);
    alloc(&h->HT[l], (size_t)B * kW);
    alloc(&h->dZT[l], (size_t)B * kW);
    alloc(&h->part[l], (size_t)chunks * 9 * kW);
    // split-K partials of dW: B / 512 splits of [256][K]
    alloc(&h->wpart[l], (size_t)std::max(1, B / 512) * kW * (l == 0 ? kK0 : kW));
  }
  alloc(&h->C, (size_t)B * 3);
  alloc(&h->T, (size_t)B * kOut);
  alloc(&h->O, (size_t)B * 8);
  alloc(&h->dO, (size_t)B * 8);
  alloc(&h->dHT, (size_t)B * kW);
  alloc(&h->dZ, (size_t)B * kW);
  alloc(&h->part4, (size_t)chunks * (kOut * kW + kOut));
  alloc(&h->row_loss, (size_t)B);
  alloc(&h->loss_part, (size_t)(B + 255) / 256);
  if (rc) {
    free_batch(h);
    return BES_ERR_CUDA;
  }
  h->cap = B;
  return BES_OK;
}

inline int nblk(int64_t n, int b) { return (int)((n + b - 1) / b); }

// Rows per CTA of the forward kernel: 128, or 64 while 128 would leave SMs without a CTA (8,192
// rows: 64 CTAs of 128 rows against 128 of 64).
inline bool narrow_rows(int64_t rows) { return rows / 128 < 152; }

template <bool TRAIN>
void launch_forward(bes_mlp* h, const ForwardArgs& a, int64_t rows) {
  if (narrow_rows(rows))
    mlp_forward_kernel<64, TRAIN><<<(unsigned)(rows / 64), kFwdThreads, kFwdSmem, h->stream>>>(a);
  else
    mlp_forward_kernel<128, TRAIN><<<(unsigned)(rows / 128), kFwdThreads, kFwdSmem, h->stream>>>(a);
}

int set_smem_limits(bes_mlp* h) {
  const auto dyn = cudaFuncAttributeMaxDynamicSharedMemorySize;
  MLP_TRY(h, cudaFuncSetAttribute(mlp_forward_kernel<64, true>, dyn, kFwdSmem));
  MLP_TRY(h, cudaFuncSetAttribute(mlp_forward_kernel<128, true>, dyn, kFwdSmem));
  MLP_TRY(h, cudaFuncSetAttribute(mlp_forward_kernel<64, false>, dyn, kFwdSmem));
  MLP_TRY(h, cudaFuncSetAttribute(mlp_forward_kernel<128, false>, dyn, kFwdSmem));
  MLP_TRY(h, cudaFuncSetAttribute(mlp_dh_kernel, dyn, kDhSmem));
  MLP_TRY(h, cudaFuncSetAttribute(mlp_dw_kernel, dyn, kDwSmem));
  return BES_OK;
}

ForwardArgs forward_args(bes_mlp* h) {
  ForwardArgs a;
  std::memset(&a, 0, sizeof(a));
  for (int l = 0; l < kLayers; ++l) a.Wb[l] = h->Wb[l];
  a.p = h->p;
  a.L = h->L;
  a.err = h->gemm_err;
  return a;
}

// forward of B rows whose features are in h->H0, conditions in h->C and targets in h->T
void forward(bes_mlp* h, int B) {
  ForwardArgs a = forward_args(h);
  a.X = h->H0;
  a.C = h->C;
  a.ldt = h->cap;
  for (int l = 0; l < kLayers; ++l) {
    a.ZT[l] = h->ZT[l];
    a.HT[l] = h->HT[l];
  }
  a.T = h->T;
  a.O = h->O;
  a.dO = h->dO;
  a.row_loss = h->row_loss;
  a.B = (float)B;
  launch_forward<true>(h, a, B);
}

// partial sums of the gradient of the batch after forward(); loss partials in loss_part
void backward(bes_mlp* h, int B, double* loss_part) {
  cudaStream_t s = h->stream;
  const Layout& L = h->L;
  const int chunks = B / kChunk;
  FilmBackArgs f;
  std::memset(&f, 0, sizeof(f));
  f.B = B;
  f.ldt = h->cap;
  f.C = h->C;
  f.dO = h->dO;
  f.W4 = h->p + L.W[kLayers];
  f.part4 = h->part4;
  f.row_loss = h->row_loss;
  f.loss_part = loss_part;
  f.dHT = h->dHT;
  f.HT = h->HT[kLayers - 1];
  for (int l = kLayers - 1; l >= 0; --l) {
    f.ZT = h->ZT[l];
    f.bias = h->p + L.b[l];
    f.F = h->p + L.F[l];
    f.g = h->p + L.g[l];
    f.dZ = l > 0 ? h->dZ : nullptr;
    f.dZT = h->dZT[l];
    f.part = h->part[l];
    if (l == kLayers - 1) film_backward_kernel<true><<<chunks, kW, 0, s>>>(f);
    else film_backward_kernel<false><<<chunks, kW, 0, s>>>(f);
    // dH_l = dZ W_l
    if (l > 0)
      mlp_dh_kernel<<<dim3(2, B / kRowTile), 256, kDhSmem, s>>>(h->dZ, h->WT[l], h->dHT, h->cap, h->gemm_err);
  }
  // dW_l = dZ_l^T H_l, split over the rows in chunks of 512 when they divide the batch
  DwArgs d;
  std::memset(&d, 0, sizeof(d));
  for (int l = 0; l < kLayers; ++l) {
    d.dZT[l] = h->dZT[l];
    d.HT[l] = l == 0 ? h->H0T : h->HT[l - 1];
    d.wpart[l] = h->wpart[l];
  }
  d.ldt = h->cap;
  d.splits = B % 512 == 0 ? B / 512 : 1;
  d.k_split = B / d.splits;
  d.err = h->gemm_err;
  mlp_dw_kernel<<<dim3(26, d.splits), 256, kDwSmem, s>>>(d);
}

UpdateArgs update_args(bes_mlp* h, int B) {
  UpdateArgs u;
  std::memset(&u, 0, sizeof(u));
  u.L = h->L;
  u.n = h->L.n;
  u.p = h->p;
  u.grad = h->grad;
  u.m = h->m;
  u.v = h->v;
  u.decay = h->decay;
  for (int l = 0; l < kLayers; ++l) {
    u.Wb[l] = h->Wb[l];
    u.WT[l] = h->WT[l];
    u.wpart[l] = h->wpart[l];
    u.part[l] = h->part[l];
  }
  u.part4 = h->part4;
  u.splits = B % 512 == 0 ? B / 512 : 1;
  u.chunks = B / kChunk;
  return u;
}

// AdamW step; with B > 0 the gradient is first added up from the batch's partial sums
void adamw(bes_mlp* h, double lr, double wd, int B) {
  h->t += 1;
  UpdateArgs u = update_args(h, B);
  u.lr = (float)lr;
  u.wd = (float)wd;
  u.bc1 = (float)(1.0 - std::pow(0.9, (double)h->t));
  u.bc2 = (float)(1.0 - std::pow(0.999, (double)h->t));
  if (B > 0) update_params_kernel<true, true><<<nblk(u.n, 256), 256, 0, h->stream>>>(u);
  else update_params_kernel<false, true><<<nblk(u.n, 256), 256, 0, h->stream>>>(u);
}
// the BF16 copies of the parameters
void refresh_weights(bes_mlp* h) {
  const UpdateArgs u = update_args(h, 0);
  update_params_kernel<false, false><<<nblk(u.n, 256), 256, 0, h->stream>>>(u);
}

void freestream_conserved(double gamma, double R, const double* mach, double* U) {
  // rho = 1, p = 1/gamma, T = 1/(gamma R) (Config.cpp:480-488), cv = R/(gamma-1)
  const double cv = R / (gamma - 1.0), T = 1.0 / (gamma * R);
  double q = 0.0;
  for (int d = 0; d < 3; ++d) q += mach[d] * mach[d];
  U[0] = 1.0;
  for (int d = 0; d < 3; ++d) U[1 + d] = mach[d];
  U[4] = cv * T + q / 2.0;
}

int check_rows(bes_mlp* h, int64_t B) {
  if (B < kRowTile || B % kRowTile != 0 || B > (1 << 22)) {
    h->last_error = "batch must be a positive multiple of 128 rows and at most 4,194,304";
    return BES_ERR_INVALID;
  }
  return BES_OK;
}

}  // namespace

extern "C" {

int bes_mlp_create(const bes_ctx* ctx, uint64_t seed, bes_mlp** out) {
  if (!ctx || !out) return BES_ERR_INVALID;
  *out = nullptr;
  bes_mlp* h = new bes_mlp();
  h->device = ctx->device;
  cudaSetDevice(h->device);
  bool made = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaStreamCreateWithFlags(&h->copy, cudaStreamNonBlocking) == cudaSuccess;
  for (int b = 0; b < 2 && made; ++b)
    made = cudaEventCreateWithFlags(&h->ready[b], cudaEventDisableTiming) == cudaSuccess &&
           cudaEventCreateWithFlags(&h->taken[b], cudaEventDisableTiming) == cudaSuccess;
  if (!made) {
    bes_mlp_destroy(h);
    return BES_ERR_CUDA;
  }
  h->gamma = ctx->opt.specific_heat_ratio;
  h->R = ctx->opt.gas_constant;
  h->nc = ctx->ref.nc;
  h->n_rows = (h->nc + kRowTile - 1) / kRowTile * kRowTile;
  // centroids scaled by their bounding box (reference numbering)
  std::vector<float> xn((size_t)h->nc * 3);
  for (int a = 0; a < 3; ++a) {
    double lo = 1e300, hi = -1e300;
    for (int64_t i = 0; i < h->nc; ++i) {
      lo = std::min(lo, ctx->ref.centroid[i * 3 + a]);
      hi = std::max(hi, ctx->ref.centroid[i * 3 + a]);
    }
    const double span = hi > lo ? hi - lo : 1.0;
    for (int64_t i = 0; i < h->nc; ++i)
      xn[i * 3 + a] = (float)(2.0 * (ctx->ref.centroid[i * 3 + a] - lo) / span - 1.0);
  }
  const Layout& L = h->L;
  int rc = 0;
  rc |= mlp_alloc(h, &h->feat_xn, xn.size());
  rc |= mlp_alloc(h, &h->feat, (size_t)h->n_rows * kK0);
  rc |= mlp_alloc(h, &h->p, L.n);
  rc |= mlp_alloc(h, &h->grad, L.n);
  rc |= mlp_alloc(h, &h->m, L.n);
  rc |= mlp_alloc(h, &h->v, L.n);
  rc |= mlp_alloc(h, &h->decay, L.n);
  for (int l = 0; l < kLayers; ++l) {
    rc |= mlp_alloc(h, &h->Wb[l], (size_t)kW * (l == 0 ? kK0 : kW));
    rc |= mlp_alloc(h, &h->WT[l], (size_t)kW * (l == 0 ? kK0 : kW));
  }
  for (double*& u : h->ustage) rc |= mlp_alloc(h, &u, (size_t)h->nc * kOut);
  rc |= mlp_alloc(h, &h->gemm_err, 1);
  rc |= set_smem_limits(h);
  if (rc) {
    bes_mlp_destroy(h);
    return BES_ERR_CUDA;
  }
  cudaMemset(h->gemm_err, 0, sizeof(int));
  // Glorot-uniform weights from the seed, zero biases, identity FiLM (F = 0, g = 0), a small
  // output layer
  std::vector<float> p(L.n, 0.0f);
  std::vector<uint8_t> decay(L.n, 0);
  uint64_t st = seed * 0x9E3779B97F4A7C15ull + 12345;
  auto uni = [&]() { st = mix64(st); return (double)(st >> 11) * (1.0 / 9007199254740992.0); };
  for (int l = 0; l <= kLayers; ++l) {
    const int fin = l == 0 ? kK0 : kW, fout = l == kLayers ? kOut : kW;
    const double a = std::sqrt(6.0 / (fin + fout)) * (l == kLayers ? 0.1 : 1.0);
    for (int64_t q = 0; q < (int64_t)fin * fout; ++q) {
      p[L.W[l] + q] = (float)((2.0 * uni() - 1.0) * a);
      decay[L.W[l] + q] = 1;
    }
  }
  cudaMemcpy(h->feat_xn, xn.data(), xn.size() * sizeof(float), cudaMemcpyHostToDevice);
  cudaMemcpy(h->p, p.data(), L.n * sizeof(float), cudaMemcpyHostToDevice);
  cudaMemcpy(h->decay, decay.data(), L.n, cudaMemcpyHostToDevice);
  cudaMemset(h->m, 0, L.n * sizeof(float));
  cudaMemset(h->v, 0, L.n * sizeof(float));
  cudaMemset(h->grad, 0, L.n * sizeof(float));
  encode_kernel<<<nblk(h->n_rows, 128), 128, 0, h->stream>>>((int)h->nc, (int)h->n_rows,
                                                             h->feat_xn, h->feat);
  refresh_weights(h);
  if (cudaStreamSynchronize(h->stream) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
    bes_mlp_destroy(h);
    return BES_ERR_CUDA;
  }
  *out = h;
  return BES_OK;
}

void bes_mlp_destroy(bes_mlp* h) {
  if (!h) return;
  for (cudaStream_t s : {h->stream, h->copy})
    if (s) cudaStreamSynchronize(s);
  free_batch(h);
  for (void* q : h->allocs) cudaFree(q);
  for (int b = 0; b < 2; ++b) {
    if (h->ready[b]) cudaEventDestroy(h->ready[b]);
    if (h->taken[b]) cudaEventDestroy(h->taken[b]);
  }
  for (cudaStream_t s : {h->stream, h->copy})
    if (s) cudaStreamDestroy(s);
  delete h;
}

const char* bes_mlp_last_error(const bes_mlp* h) { return h ? h->last_error.c_str() : "null"; }

int bes_mlp_params(bes_mlp* h, float* get, const float* set, int64_t* n_params) {
  if (!h) return BES_ERR_INVALID;
  if (n_params) *n_params = h->L.n;
  if (set) {
    MLP_TRY(h, cudaMemcpy(h->p, set, h->L.n * sizeof(float), cudaMemcpyHostToDevice));
    refresh_weights(h);
    MLP_TRY(h, cudaStreamSynchronize(h->stream));
  }
  if (get) MLP_TRY(h, cudaMemcpy(get, h->p, h->L.n * sizeof(float), cudaMemcpyDeviceToHost));
  return BES_OK;
}

int bes_mlp_features(bes_mlp* h, float* xn) {
  if (!h || !xn) return BES_ERR_INVALID;
  MLP_TRY(h, cudaMemcpy(xn, h->feat_xn, h->nc * 3 * sizeof(float), cudaMemcpyDeviceToHost));
  return BES_OK;
}

int bes_mlp_loss_grad(bes_mlp* h, int32_t n_rows, const int64_t* cells, const double* cond,
                      const double* targets, double* loss, float* grad, double* outputs) {
  if (!h || !cells || !cond) return BES_ERR_INVALID;
  int rc = check_rows(h, n_rows);
  if (rc) return rc;
  if ((rc = ensure_batch(h, n_rows))) return rc;
  const int B = n_rows;
  // rows from the feature table, conditions and targets as given
  std::vector<float> C((size_t)B * 3), T((size_t)B * kOut, 0.0f);
  for (int r = 0; r < B; ++r) {
    if (cells[r] < 0 || cells[r] >= h->nc) {
      h->last_error = "cell index out of range";
      return BES_ERR_INVALID;
    }
    for (int a = 0; a < 3; ++a) C[r * 3 + a] = (float)cond[r * 3 + a];
    if (targets)
      for (int v = 0; v < kOut; ++v) T[r * kOut + v] = (float)targets[r * kOut + v];
  }
  int64_t* dcells = nullptr;
  MLP_TRY(h, cudaMallocAsync((void**)&dcells, (size_t)B * sizeof(int64_t), h->stream));
  MLP_TRY(h, cudaMemcpyAsync(dcells, cells, (size_t)B * sizeof(int64_t), cudaMemcpyHostToDevice, h->stream));
  gather_cells_kernel<<<nblk(B, 128), 128, 0, h->stream>>>(B, dcells, h->feat, h->H0, h->H0T, h->cap);
  MLP_TRY(h, cudaFreeAsync(dcells, h->stream));
  MLP_TRY(h, cudaMemcpyAsync(h->C, C.data(), C.size() * 4, cudaMemcpyHostToDevice, h->stream));
  MLP_TRY(h, cudaMemcpyAsync(h->T, T.data(), T.size() * 4, cudaMemcpyHostToDevice, h->stream));
  forward(h, B);
  backward(h, B, h->loss_part);
  const UpdateArgs u = update_args(h, B);
  update_params_kernel<true, false><<<nblk(u.n, 256), 256, 0, h->stream>>>(u);
  std::vector<double> lp((B + 255) / 256);
  MLP_TRY(h, cudaMemcpyAsync(lp.data(), h->loss_part, lp.size() * 8, cudaMemcpyDeviceToHost, h->stream));
  std::vector<float> o((size_t)B * 8);
  MLP_TRY(h, cudaMemcpyAsync(o.data(), h->O, o.size() * 4, cudaMemcpyDeviceToHost, h->stream));
  if (grad) MLP_TRY(h, cudaMemcpyAsync(grad, h->grad, h->L.n * 4, cudaMemcpyDeviceToHost, h->stream));
  MLP_TRY(h, cudaStreamSynchronize(h->stream));
  MLP_TRY(h, cudaGetLastError());
  if (loss) {
    double s = 0.0;
    for (double x : lp) s += x;
    *loss = s;
  }
  if (outputs)
    for (int r = 0; r < B; ++r)
      for (int v = 0; v < kOut; ++v) outputs[r * kOut + v] = o[r * 8 + v];
  return gemm_status(h);
}

int bes_mlp_apply_grad(bes_mlp* h, const float* grad, double lr, double weight_decay) {
  if (!h || !grad) return BES_ERR_INVALID;
  MLP_TRY(h, cudaMemcpyAsync(h->grad, grad, h->L.n * 4, cudaMemcpyHostToDevice, h->stream));
  adamw(h, lr, weight_decay, 0);
  MLP_TRY(h, cudaStreamSynchronize(h->stream));
  MLP_TRY(h, cudaGetLastError());
  return BES_OK;
}

int bes_mlp_train(bes_mlp* h, int32_t n_samples, const double* mach, const double* U,
                  int64_t steps, int32_t batch, double lr, double weight_decay, uint64_t seed,
                  double* loss_history) {
  if (!h || !mach || !U || n_samples < 1 || steps < 0) return BES_ERR_INVALID;
  int rc = check_rows(h, batch);
  if (rc) return rc;
  if ((rc = ensure_batch(h, batch))) return rc;
  const int64_t nc = h->nc;
  // normalisation from the training set: condition mean / std, output scale = std of U - U_inf
  for (int a = 0; a < 3; ++a) {
    double s = 0, s2 = 0;
    for (int q = 0; q < n_samples; ++q) s += mach[q * 3 + a];
    const double mu = s / n_samples;
    for (int q = 0; q < n_samples; ++q) s2 += (mach[q * 3 + a] - mu) * (mach[q * 3 + a] - mu);
    const double sd = std::sqrt(s2 / n_samples);
    h->cmean[a] = mu;
    h->csd[a] = sd > 1e-6 ? sd : 1.0;
  }
  std::vector<double> Uinf((size_t)n_samples * kOut);
  for (int q = 0; q < n_samples; ++q) freestream_conserved(h->gamma, h->R, &mach[q * 3], &Uinf[q * kOut]);
  {
    // (one accumulator per variable, each in the order of the samples and cells)
    double s2[kOut] = {0, 0, 0, 0, 0};
    for (int q = 0; q < n_samples; ++q)
      for (int64_t i = 0; i < nc; ++i)
        for (int v = 0; v < kOut; ++v) {
          const double d = U[((size_t)q * nc + i) * kOut + v] - Uinf[q * kOut + v];
          s2[v] += d * d;
        }
    for (int v = 0; v < kOut; ++v) {
      const double sd = std::sqrt(s2[v] / ((double)n_samples * nc));
      h->oscale[v] = sd > 1e-6 ? sd : 1e-6;
    }
  }
  std::vector<float> cnd((size_t)n_samples * 3);
  for (int q = 0; q < n_samples; ++q)
    for (int a = 0; a < 3; ++a) cnd[q * 3 + a] = (float)((mach[q * 3 + a] - h->cmean[a]) / h->csd[a]);
  const size_t n_tgt = (size_t)n_samples * nc * kOut;
  float *dt = nullptr, *dc = nullptr;
  double* dscale = nullptr;  // U_inf of the samples, then the output scale
  const std::vector<double> scale = [&] {
    std::vector<double> x(Uinf);
    x.insert(x.end(), h->oscale, h->oscale + kOut);
    return x;
  }();
  MLP_TRY(h, cudaMalloc((void**)&dt, n_tgt * sizeof(float)));
  if (cudaMalloc((void**)&dc, cnd.size() * sizeof(float)) != cudaSuccess ||
      cudaMalloc((void**)&dscale, scale.size() * sizeof(double)) != cudaSuccess) {
    cudaFree(dt);
    cudaFree(dc);
    h->last_error = "cudaMalloc of the condition table failed";
    return BES_ERR_CUDA;
  }
  cudaMemcpyAsync(dc, cnd.data(), cnd.size() * 4, cudaMemcpyHostToDevice, h->stream);
  cudaMemcpyAsync(dscale, scale.data(), scale.size() * 8, cudaMemcpyHostToDevice, h->stream);
  for (int q = 0; q < n_samples; ++q) {
    const int64_t n = nc * kOut;
    cudaMemcpyAsync(h->ustage[0], U + (size_t)q * n, n * sizeof(double), cudaMemcpyHostToDevice, h->stream);
    targets_kernel<<<1024, 256, 0, h->stream>>>(n, n, h->ustage[0], dscale + q * kOut,
                                                dscale + n_samples * kOut, dt + (size_t)q * n);
  }
  const size_t n_lp = (batch + 255) / 256;
  double* dloss = nullptr;
  if (loss_history && steps > 0) cudaMalloc((void**)&dloss, steps * n_lp * sizeof(double));
  for (int64_t s = 0; s < steps; ++s) {
    gather_kernel<<<nblk(batch, 128), 128, 0, h->stream>>>(batch, seed, s, n_samples, (int)nc, h->feat, dt,
                                                           dc, h->H0, h->H0T, h->cap, h->C, h->T);
    forward(h, batch);
    backward(h, batch, dloss ? dloss + s * n_lp : h->loss_part);
    adamw(h, lr, weight_decay, batch);
  }
  cudaError_t e = cudaStreamSynchronize(h->stream);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess && dloss) {
    std::vector<double> all(steps * n_lp);
    e = cudaMemcpy(all.data(), dloss, all.size() * 8, cudaMemcpyDeviceToHost);
    for (int64_t s = 0; s < steps; ++s) {
      double x = 0.0;
      for (size_t q = 0; q < n_lp; ++q) x += all[s * n_lp + q];
      loss_history[s] = x;
    }
  }
  cudaFree(dt);
  cudaFree(dc);
  cudaFree(dscale);
  if (dloss) cudaFree(dloss);
  if (e != cudaSuccess) {
    h->last_error = std::string("training: ") + cudaGetErrorString(e);
    return BES_ERR_CUDA;
  }
  return gemm_status(h);
}

int bes_mlp_infer(bes_mlp* h, int32_t n, const double* mach, double* U) {
  if (!h || !mach || !U || n < 0) return BES_ERR_INVALID;
  ForwardArgs a = forward_args(h);
  a.X = h->feat;
  a.n = h->nc;
  for (int v = 0; v < kOut; ++v) a.oscale[v] = h->oscale[v];
  // The copy to the caller's memory takes longer than the kernel (pageable memory, and the call
  // returns when it is done): the next condition's kernel is launched before it, on the other field.
  for (int q = 0; q <= n; ++q) {
    if (q < n) {
      const int b = q & 1;
      for (int d = 0; d < 3; ++d) a.c3[d] = (float)((mach[q * 3 + d] - h->cmean[d]) / h->csd[d]);
      freestream_conserved(h->gamma, h->R, &mach[q * 3], a.Uinf);
      a.U = h->ustage[b];
      if (q >= 2) MLP_TRY(h, cudaStreamWaitEvent(h->stream, h->taken[b], 0));
      launch_forward<false>(h, a, h->n_rows);
      MLP_TRY(h, cudaEventRecord(h->ready[b], h->stream));
    }
    if (q > 0) {
      const int b = (q - 1) & 1;
      MLP_TRY(h, cudaStreamWaitEvent(h->copy, h->ready[b], 0));
      MLP_TRY(h, cudaMemcpyAsync(U + (size_t)(q - 1) * h->nc * kOut, h->ustage[b],
                                 (size_t)h->nc * kOut * sizeof(double), cudaMemcpyDeviceToHost, h->copy));
      MLP_TRY(h, cudaEventRecord(h->taken[b], h->copy));
    }
  }
  MLP_TRY(h, cudaStreamSynchronize(h->copy));
  MLP_TRY(h, cudaStreamSynchronize(h->stream));
  MLP_TRY(h, cudaGetLastError());
  return gemm_status(h);
}

int bes_mlp_init_state(bes_mlp* h, bes_ctx* ctx, int32_t* used) {
  if (!h || !ctx) return BES_ERR_INVALID;
  if (ctx->ref.nc != h->nc) {
    h->last_error = "the context's mesh differs from the network's";
    return BES_ERR_INVALID;
  }
  const int nb = ctx->nb;
  const int64_t nc = h->nc;
  std::vector<double> mach((size_t)nb * 3);
  for (int b = 0; b < nb; ++b)
    for (int d = 0; d < 3; ++d) mach[b * 3 + d] = ctx->pinf0_host[6 * b + 1 + d];
  std::vector<double> U((size_t)nb * nc * kOut);
  int rc = bes_mlp_infer(h, nb, mach.data(), U.data());
  if (rc) return rc;
  // a prediction that is not physical falls back to the freestream for that condition
  std::vector<double> Uf((size_t)nb * nc * kOut);
  rc = bes_set_freestream_state(ctx);
  if (rc) return rc;
  rc = bes_get_state(ctx, Uf.data());
  if (rc) return rc;
  const double gm1 = h->gamma - 1.0;
  for (int b = 0; b < nb; ++b) {
    bool ok = true;
    for (int64_t i = 0; i < nc && ok; ++i) {
      const double* u = &U[((size_t)b * nc + i) * kOut];
      const double p = gm1 * (u[4] - (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) / (2.0 * u[0]));
      ok = u[0] > 0.0 && p > 0.0 && std::isfinite(p);
    }
    if (used) used[b] = ok ? 1 : 0;
    if (!ok)
      std::copy(Uf.begin() + (size_t)b * nc * kOut, Uf.begin() + (size_t)(b + 1) * nc * kOut,
                U.begin() + (size_t)b * nc * kOut);
  }
  return bes_set_state(ctx, U.data());
}

int bes_mlp_normalisation(const bes_mlp* h, double* out) {
  if (!h || !out) return BES_ERR_INVALID;
  for (int a = 0; a < 3; ++a) {
    out[a] = h->cmean[a];
    out[3 + a] = h->csd[a];
  }
  for (int v = 0; v < kOut; ++v) out[6 + v] = h->oscale[v];
  return BES_OK;
}

}  // extern "C"
