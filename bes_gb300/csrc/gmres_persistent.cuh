// One cooperative launch for the linear solves of a step: every restart cycle, Arnoldi step,
// preconditioner sweep and GMRES decision of all slots.
//
// On meshes whose phases take a few microseconds the step graph's solve is bound by its nodes:
// an Arnoldi step with block ILU is 12 kernels (eight of them the colour sweep's) and two conditional
// nodes: 57 to 80 us from 1,152 to 50,000 cells in FP32, 95 to 139 in FP64.  Here nothing is launched between Arnoldi steps: rows wait for
// the entries they need (below), four grid barriers (an atomic and a poll of one word in L2, about
// 2 us) separate the product, the dot products, their reduction and the new basis vector, and
// the decisions are taken by every block from the same values.  What is left is a chain of
// round trips to L2: an Arnoldi step takes 41 to 50 us in FP32 (7,000 cells: sweeps 20, product
// 5, Gram-Schmidt 17), 48 to 50 in FP64 up to 7,000 cells and 85 at 31,000.
//
// Every value is computed as by the graph's kernels, bit for bit: rows in the order of the row
// functions, reductions over the same kRedBlocks x 256 threads ("virtual blocks", dealt out to
// the blocks of the grid), the GMRES control by the same statements.
#pragma once
#include "krylov_kernels.cuh"

namespace bes {

// Grid barrier on a counter that only grows during a launch (zeroed before it).  A wait gives
// up after one second and sets the error flag (BES_ERR_TIMEOUT for the host); once it is set
// every later wait of every launch returns at once, so no launch can hang.
struct GridBar {
  unsigned* count;
  int* error;
};

template <class T, class B>
struct SolveArgs {
  DevMesh m;
  SweepPlan plan;       // colour stages (block ILU)
  SweepOps<T> ops;      // factors (block ILU) or inverse diagonal (block Jacobi)
  int ilu;
  SlotPtr<const uint32_t> A16;  // packed matrix
  SlotPtr<const T> A;          // matrix in T
  SlotPtr<const T> b;
  SlotPtr<T> Y, Z, W, X, Vx;
  B* V;
  int64_t sV, ldv, N;
  double* red;          // per slot: rows of kRedBlocks partials
  int64_t sred;         // values per slot
  GmresDev g;
  GmresParam P;
  int nslot;
  int lane_spmv;        // the products with one component per lane (else one row per thread)
  const int32_t* act;
  const int* nan_flag;
  const int32_t* guard;
  GridBar bar;
  unsigned long long* prof;  // category stamps, or null
};

// All blocks arrive before any leaves; false if a wait gave up.  target: thread 0's count.
__device__ __forceinline__ bool grid_barrier(const GridBar& b, unsigned& target) {
  __syncthreads();
  int good = 1;
  if (threadIdx.x == 0) {
    target += gridDim.x;
    unsigned old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(b.count) : "memory");
    if ((int)(old + 1u - target) < 0) {
      unsigned long long t0 = 0;
      int spin = 0;
      while ((int)(ld_acquire(b.count) - target) < 0) {
        if ((++spin & 63) != 0) continue;
        if (*(volatile int*)b.error) {
          good = 0;
          break;
        }
        const unsigned long long t = global_ns();
        if (t0 == 0) t0 = t;
        if (t - t0 > 1000000000ull) {
          atomicExch(b.error, 1);
          good = 0;
          break;
        }
      }
    }
  }
  return __syncthreads_and(good) != 0;
}

// ---- vector loads through L2 (other blocks of the launch write these vectors) --------------------
template <class T, class B, class A>
__device__ __forceinline__ void basis_load_cg(const B* V, int64_t g, A* x) {
  const uint4 u = __ldcg(reinterpret_cast<const uint4*>(V) + g);
  if constexpr (std::is_same<T, B>::value) {
    const Pack16<T> p = *reinterpret_cast<const Pack16<T>*>(&u);
#pragma unroll
    for (int e = 0; e < Pack16<T>::W; ++e) x[e] = (A)p.v[e];
  } else {
    BasisIO<T, B>::unpack(u, x);
  }
}
template <class T, class A>
__device__ __forceinline__ void vec_load_cg(const T* w, int64_t pack, A* x) {
  const uint4 u = __ldcg(reinterpret_cast<const uint4*>(w) + pack);
  const Pack16<T> p = *reinterpret_cast<const Pack16<T>*>(&u);
#pragma unroll
  for (int e = 0; e < Pack16<T>::W; ++e) x[e] = (A)p.v[e];
}
template <class T, class B, class A>
__device__ __forceinline__ A basis_get_cg(const B* V, int64_t i) {
  if constexpr (std::is_same<T, B>::value) return (A)__ldcg(V + i);
  else {
    const __half h = __ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(V) + i));
    return BasisIO<T, B>::template get<A>(&h, 0);
  }
}

// ---- vector entries that are waited for ----------------------------------------------------------
// The sweeps and the product behind them have no barriers between their stages: an entry of Y
// (forward solve) or Z (backward solve) that has not been computed yet holds a mark, a NaN that
// no arithmetic produces, and whoever needs it reads again until the mark is gone.  Every warp
// walks the stages in order and all blocks are resident, so a row waits only for rows that are
// being worked on.  A stage then costs one store and one load through L2 (about 1 us) instead of
// a grid barrier and a round of loads behind it (3.5 us).  The marks are set again while the
// vectors are not in use, with a barrier on both sides.
template <class T> struct Mark;
template <> struct Mark<float> {
  typedef unsigned Bits;
  static constexpr Bits value = 0x7fadbeefu;
  __device__ static __forceinline__ Bits bits(float x) { return __float_as_uint(x); }
  __device__ static __forceinline__ float make() { return __uint_as_float(value); }
  __device__ static __forceinline__ float nan() { return __uint_as_float(0x7fffffffu); }
};
template <> struct Mark<double> {
  typedef unsigned long long Bits;
  static constexpr Bits value = 0x7ff5deadbeef0001ull;
  __device__ static __forceinline__ Bits bits(double x) { return (Bits)__double_as_longlong(x); }
  __device__ static __forceinline__ double make() { return __longlong_as_double((long long)value); }
  __device__ static __forceinline__ double nan() { return __longlong_as_double((long long)0xfff8000000000000ull); }
};
template <class T>
__device__ __forceinline__ bool is_mark(T x) { return Mark<T>::bits(x) == Mark<T>::value; }

__device__ __forceinline__ float4 ld_relaxed(const float4* p) {
  float4 v;
  asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ double2 ld_relaxed(const double2* p) {
  double2 v;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float ld_relaxed(const float* p) {
  float v;
  asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ double ld_relaxed(const double* p) {
  double v;
  asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
  return v;
}
// An entry that other blocks may be polling: a strong store, as their loads are (a weak one beside
// them would be a data race).
__device__ __forceinline__ void st_relaxed(float* p, float v) {
  asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" : : "l"(p), "f"(v) : "memory");
}
__device__ __forceinline__ void st_relaxed(double* p, double v) {
  asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" : : "l"(p), "d"(v) : "memory");
}
// gather5 of entries that may not be there yet; false while one is missing
__device__ __forceinline__ bool try_gather5(const float* x, int j, float* y) {
  const int64_t e0 = (int64_t)j * 5;
  const float4* p = reinterpret_cast<const float4*>(x) + (e0 >> 2);
  const float4 a = ld_relaxed(p), b = ld_relaxed(p + 1);
  const float w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  const int o = (int)(e0 & 3);
  bool ok = true;
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    float t = w[v];
    t = o == 1 ? w[v + 1] : t;
    t = o == 2 ? w[v + 2] : t;
    t = o == 3 ? w[v + 3] : t;
    y[v] = t;
    ok = ok && !is_mark(t);
  }
  return ok;
}
__device__ __forceinline__ bool try_gather5(const double* x, int j, double* y) {
  const int64_t e0 = (int64_t)j * 5;
  const double2* p = reinterpret_cast<const double2*>(x) + (e0 >> 1);
  const double2 a = ld_relaxed(p), b = ld_relaxed(p + 1), c = ld_relaxed(p + 2);
  const double w[6] = {a.x, a.y, b.x, b.y, c.x, c.y};
  const bool odd = e0 & 1;
  bool ok = true;
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    y[v] = odd ? w[v + 1] : w[v];
    ok = ok && !is_mark(y[v]);
  }
  return ok;
}
// One more turn of a wait: false when it has to be given up (after a second, or because another
// wait of the launch has been).
struct Spin {
  int n = 0;
  unsigned long long t0 = 0;
  __device__ __forceinline__ bool turn(int* error) {
    if ((++n & 63) != 0) return true;
    if (*(volatile int*)error) return false;
    const unsigned long long t = global_ns();
    if (t0 == 0) t0 = t;
    if (t - t0 < 1000000000ull) return true;
    atomicExch(error, 1);
    return false;
  }
};
template <class T>
__device__ __forceinline__ void wait_gather5(const T* x, int j, T* y, int* error) {
  Spin spin;
  while (!try_gather5(x, j, y) && spin.turn(error)) {
  }
}
template <class T>
__device__ __forceinline__ T wait_entry(const T* x, int* error) {
  Spin spin;
  T v = ld_relaxed(x);
  while (is_mark(v) && spin.turn(error)) v = ld_relaxed(x);
  return v;
}
template <class T>
__device__ __forceinline__ void put_entry(T* x, T v) {
  st_relaxed(x, is_mark(v) ? Mark<T>::nan() : v);
}

// ---- rows ----------------------------------------------------------------------------------------
// Two ways to deal out rows.  One component per lane: a warp takes six rows, lane 5 q + r the
// component r of row q (lanes 30 and 31 idle), so that a lane's part of a row is 20 to 25 words,
// loaded while the row before it waits for its neighbours: the shorter time per row, where a
// stage's rows fit the grid about at once.  One row per thread (32 consecutive rows per warp): a
// third of the load instructions and whole sectors, for more rows.  Each component is
// accumulated in the order of the row functions (slots, then columns).
constexpr int kRowsPerWarp = 6;

// A lane's words of one block row: five values of T, or three words of a packed block and its
// scale (entries 5 r .. 5 r + 4 of the row-major block).
template <class T, bool PACKED>
struct LaneBlock {
  T a[5];
  __device__ __forceinline__ void load(const T* __restrict__ A, int nslots, int s, int i, int r) {
    // (entry by entry: 16-byte words and selecting from them cost more than they save here)
    const T* p = A + block_at<T>(nslots, s, 0, i - (i & 31));
#pragma unroll
    for (int c = 0; c < 5; ++c) a[c] = p[block_at<T>(1, 0, 5 * r + c, i & 31)];
  }
  __device__ __forceinline__ T entry(int c, int) const { return a[c]; }
  __device__ __forceinline__ T scale() const { return T(1); }
};
template <>
struct LaneBlock<float, true> {
  uint32_t w[3];
  float sc;
  __device__ __forceinline__ void load(const uint32_t* __restrict__ H, int nslots, int s, int i, int r) {
    const uint32_t* h = packed_slot(H, nslots, s, i);
    const int p0 = (5 * r) >> 1;
#pragma unroll
    for (int p = 0; p < 3; ++p) w[p] = h[packed_word(p0 + p, i)];
    sc = packed_scale(h[packed_word(12, i)]);
  }
  // entry c of the row: half 5 r + c of the block, and 5 r starts in the second half for odd r
  __device__ __forceinline__ float entry(int c, int r) const {
    const bool odd = r & 1;
    const float2 even = __half22float2(*reinterpret_cast<const __half2*>(&w[c >> 1]));
    const float2 next = __half22float2(*reinterpret_cast<const __half2*>(&w[(c + 1) >> 1]));
    const float e = (c & 1) ? even.y : even.x;         // half c of the words
    const float o = ((c + 1) & 1) ? next.y : next.x;   // half c + 1
    return odd ? o : e;
  }
  __device__ __forceinline__ float scale() const { return sc; }
};

struct RowItem {
  int k, i;  // slot and row; i < 0: none
};
template <bool LANES>
__device__ __forceinline__ int row_chunks(int n) {
  return LANES ? (n + kRowsPerWarp - 1) / kRowsPerWarp : (n + 31) >> 5;
}
// Slot and row of this lane in warp item `it` of rows [r0, r1).
template <bool LANES>
__device__ __forceinline__ RowItem row_item(int64_t it, int r0, int r1, int nslot, const int* run) {
  const int lane = threadIdx.x & 31, q = LANES ? lane / 5 : lane, chunks = row_chunks<LANES>(r1 - r0);
  RowItem o;
  o.k = nslot == 1 ? 0 : (int)(it / chunks);
  if (o.k >= nslot || it >= (int64_t)chunks * nslot) return RowItem{0, -1};
  o.i = r0 + (int)(it - (int64_t)o.k * chunks) * (LANES ? kRowsPerWarp : 32) + q;
  if ((LANES && q >= kRowsPerWarp) || o.i >= r1 || run[o.k] == 0) o.i = -1;
  return o;
}
__device__ __forceinline__ int64_t first_item() {
  return (int64_t)(threadIdx.x >> 5) * gridDim.x + blockIdx.x;  // spread over the SMs first
}
__device__ __forceinline__ int64_t item_stride() { return (int64_t)gridDim.x * (blockDim.x >> 5); }

// A lane's part of a sweep row.
template <class T, bool PACKED>
struct SweepLane {
  RowItem q;
  int j[4];
  LaneBlock<T, PACKED> blk[4], inv;
};

// Virtual blocks of the vector kernels: f(slot, vb) for the first nvb of kRedBlocks (the
// others have no elements and their partial sums are zero).
template <class F>
__device__ __forceinline__ void for_vblocks(int nvb, int nslot, const int* run, F&& f) {
  for (int it = blockIdx.x; it < nvb * nslot; it += gridDim.x) {
    const int k = nslot == 1 ? 0 : it / nvb;
    if (run[k] == 0) continue;
    f(k, it - k * nvb);
  }
}

__device__ __forceinline__ int active_vblocks(int64_t n) {
  const int64_t v = (n + 255) / 256;
  return (int)(v < kRedBlocks ? (v < 1 ? 1 : v) : kRedBlocks);
}

template <class T, class B, bool PACKED>
__device__ __forceinline__ void sweep_lane_load(const SolveArgs<T, B>& S, int st, int64_t it, int r,
                                                const int* run, SweepLane<T, PACKED>& L) {
  const int nc = S.m.nc;
  L.q = row_item<true>(it, S.plan.r0[st], S.plan.r1[st], S.nslot, run);
  if (L.q.i < 0) return;
  // every slot's words: which of them the stage uses is known only behind the neighbour ids
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    L.j[s] = S.m.adj[s * nc + L.q.i];
    if constexpr (PACKED) L.blk[s].load(S.ops.H.of(L.q.k), 4, s, L.q.i, r);
    else L.blk[s].load(S.ops.L.of(L.q.k), 5, 1 + s, L.q.i, r);
  }
  if constexpr (PACKED) L.inv.load(S.ops.D.of(L.q.k), 1, 0, L.q.i, r);
  else L.inv.load(S.ops.Dinv.of(L.q.k), 1, 0, L.q.i, r);
}
// One row of a stage by one component per lane (ilu_colour_row / ilu_colour_packed_row).  Every
// lane of the warp calls.
template <class T, class B, bool PACKED>
__device__ __forceinline__ void sweep_lane_row(const SolveArgs<T, B>& S, int st, int r, const T* in0,
                                               int64_t in_stride, const SweepLane<T, PACKED>& L) {
  const int r0 = S.plan.r0[st], r1 = S.plan.r1[st], kind = S.plan.kind[st], s1 = S.plan.s1;
  int* err = S.bar.error;
  const int i = L.q.i;
  T acc = T(0);
  if (i >= 0) {
    const T* in = in0 + L.q.k * in_stride;
    const T *Y = S.Y.of(L.q.k), *Z = S.Z.of(L.q.k);
    T y[4][5];
    bool use[4], ok;
    Spin spin;
    do {
      ok = true;
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int j = L.j[s];
        const bool lower = kind != 2 && j >= 0 && j < r0;
        use[s] = lower || (kind != 0 && j >= r1);
        if (use[s]) ok = try_gather5(lower ? (j < s1 ? in : Y) : Z, j, y[s]) && ok;
      }
    } while (!ok && spin.turn(err));
    acc = (kind != 2 || r0 == 0) ? __ldcg(in + (int64_t)i * 5 + r) : wait_entry(Y + (int64_t)i * 5 + r, err);
#pragma unroll
    for (int s = 0; s < 4; ++s)
      if (use[s])
#pragma unroll
        for (int c = 0; c < 5; ++c)
          acc = fma_t(-L.blk[s].entry(c, r), PACKED ? y[s][c] * L.blk[s].scale() : y[s][c], acc);
  }
  if (kind != 0) {
    __syncwarp();
    const int base = (threadIdx.x & 31) - r;
    T x = T(0);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const T ac = __shfl_sync(0xffffffffu, acc, base + c < 31 ? base + c : 31);
      if (i >= 0) x = fma_t(L.inv.entry(c, r), ac, x);
    }
    if (i >= 0) put_entry(S.Z.of(L.q.k) + (int64_t)i * 5 + r, PACKED ? L.inv.scale() * x : x);
  } else if (i >= 0) {
    put_entry(S.Y.of(L.q.k) + (int64_t)i * 5 + r, acc);
  }
}
// Block Jacobi.
template <class T, class B, bool PACKED>
__device__ __noinline__ void phase_jacobi(const SolveArgs<T, B>& S, const T* in, int64_t in_stride,
                                const int* run) {
  const int nc = S.m.nc, lane = threadIdx.x & 31, r = lane - 5 * (lane / 5);
  const int64_t items = (int64_t)row_chunks<true>(nc) * S.nslot;
  for (int64_t it = first_item(); it < items; it += item_stride()) {
    const RowItem q = row_item<true>(it, 0, nc, S.nslot, run);
    if (q.i < 0) continue;
    LaneBlock<T, PACKED> D;
    if constexpr (PACKED) D.load(S.ops.D.of(q.k), 1, 0, q.i, r);
    else D.load(S.ops.Dinv.of(q.k), 1, 0, q.i, r);
    T x[5], acc = T(0);
    gather5<true>(in + q.k * in_stride, q.i, x);
#pragma unroll
    for (int c = 0; c < 5; ++c) acc = fma_t(D.entry(c, r), x[c], acc);
    put_entry(S.Z.of(q.k) + (int64_t)q.i * 5 + r, PACKED ? D.scale() * acc : acc);
  }
}

// The colour sweeps, one component per lane.
template <class T, class B, bool PACKED>
__device__ __noinline__ void phase_sweep_lanes(const SolveArgs<T, B>& S, const T* in, int64_t in_stride,
                                const int* run) {
  const int lane = threadIdx.x & 31, r = lane - 5 * (lane / 5);
  SweepLane<T, PACKED> L, next;
  int st = 0;
  int64_t it = first_item();
  sweep_lane_load<T, B, PACKED>(S, st, it, r, run, L);
  while (st < S.plan.n) {
    const int64_t items = (int64_t)row_chunks<true>(S.plan.r1[st] - S.plan.r0[st]) * S.nslot;
    int st2 = st;
    int64_t it2 = it + item_stride();
    if (it2 >= items) {
      st2 = st + 1;
      it2 = first_item();
    }
    if (st2 < S.plan.n) sweep_lane_load<T, B, PACKED>(S, st2, it2, r, run, next);
    sweep_lane_row<T, B, PACKED>(S, st, r, in, in_stride, L);
    L = next;
    st = st2;
    it = it2;
  }
}

// Z = M^{-1} in for every slot whose run flag is set; Y and Z hold marks before, and Z may be
// incomplete on return.
template <class T, class B, bool PACKED>
__device__ __forceinline__ void phase_precond(const SolveArgs<T, B>& S, const T* in, int64_t in_stride,
                                              const int* run) {
  if (S.ilu) phase_sweep_lanes<T, B, PACKED>(S, in, in_stride, run);
  else phase_jacobi<T, B, PACKED>(S, in, in_stride, run);
}

// W = A Z (Z waited for), or (RESIDUAL) W = b - A X (spmv_row / spmv_packed_row).
template <class T, class B, bool PACKED, bool RESIDUAL>
__device__ __noinline__ void phase_spmv(const SolveArgs<T, B>& S, const int* run) {
  const int nc = S.m.nc;
  int* err = S.bar.error;
  if (!RESIDUAL && S.lane_spmv) {
    const int lane = threadIdx.x & 31, r = lane - 5 * (lane / 5);
    const int64_t items = (int64_t)row_chunks<true>(nc) * S.nslot;
    for (int64_t it = first_item(); it < items; it += item_stride()) {
      const RowItem q = row_item<true>(it, 0, nc, S.nslot, run);
      if (q.i < 0) continue;
      int j[5];
      j[0] = q.i;
#pragma unroll
      for (int s = 0; s < 4; ++s) j[1 + s] = S.m.adj[s * nc + q.i];
      LaneBlock<T, PACKED> blk[5];
#pragma unroll
      for (int s = 0; s < 5; ++s) {
        if constexpr (PACKED) blk[s].load(S.A16.of(q.k), 5, s, q.i, r);
        else blk[s].load(S.A.of(q.k), 5, s, q.i, r);
      }
      const T* x = S.Z.of(q.k);
      T acc = T(0);
#pragma unroll
      for (int s = 0; s < 5; ++s) {
        if (!PACKED && j[s] < 0) continue;  // packed: the block is zero and adds exactly 0
        T y[5];
        wait_gather5(x, j[s] >= 0 ? j[s] : q.i, y, err);
#pragma unroll
        for (int c = 0; c < 5; ++c)
          acc = fma_t(blk[s].entry(c, r), PACKED ? y[c] * blk[s].scale() : y[c], acc);
      }
      S.W.of(q.k)[(int64_t)q.i * 5 + r] = acc;
    }
    return;
  }
  const int64_t items = (int64_t)row_chunks<false>(nc) * S.nslot;
  for (int64_t it = first_item(); it < items; it += item_stride()) {
    const RowItem q = row_item<false>(it, 0, nc, S.nslot, run);
    if (q.i < 0) continue;
    if constexpr (RESIDUAL) {
      const T *x = S.X.of(q.k), *b = S.b.of(q.k);
      if constexpr (PACKED) spmv_packed_row<true>(S.m, q.i, S.A16.of(q.k), x, b, S.W.of(q.k));
      else spmv_row<T, true>(S.m, q.i, S.A.of(q.k), x, b, S.W.of(q.k));
    } else {
      const T* x = S.Z.of(q.k);
      T acc[5] = {T(0), T(0), T(0), T(0), T(0)};
      int j[5];
      j[0] = q.i;
#pragma unroll
      for (int s = 0; s < 4; ++s) j[1 + s] = S.m.adj[s * nc + q.i];
#pragma unroll
      for (int s = 0; s < 5; ++s) {
        if (!PACKED && j[s] < 0) continue;
        T a[25], y[5], sc = T(1);
        if constexpr (PACKED) {
          sc = load_packed(S.A16.of(q.k), 5, s, q.i).unpack(a);
        } else {
          load_block(S.A.of(q.k), 5, s, q.i, a);
        }
        wait_gather5(x, j[s] >= 0 ? j[s] : q.i, y, err);
        if constexpr (PACKED) {
#pragma unroll
          for (int c = 0; c < 5; ++c) y[c] *= sc;
        }
#pragma unroll
        for (int r = 0; r < 5; ++r)
#pragma unroll
          for (int c = 0; c < 5; ++c) acc[r] = fma_t(a[r * 5 + c], y[c], acc[r]);
      }
      T* w = S.W.of(q.k) + (int64_t)q.i * 5;
#pragma unroll
      for (int r = 0; r < 5; ++r) w[r] = acc[r];
    }
  }
}

// The marks of the next preconditioner application, over the vector's 16-byte packs.
template <class T, class B>
__device__ __forceinline__ void set_marks(const SolveArgs<T, B>& S, int k, int vb) {
  typedef Pack16<T> P;
  P mk;
#pragma unroll
  for (int e = 0; e < P::W; ++e) mk.v[e] = Mark<T>::make();
  P* z = reinterpret_cast<P*>(S.Z.of(k));
  P* y = S.ilu ? reinterpret_cast<P*>(S.Y.of(k)) : nullptr;
  const int64_t n = S.ldv / P::W;
  for (int64_t g = (int64_t)vb * 256 + threadIdx.x; g < n; g += (int64_t)kRedBlocks * 256) {
    z[g] = mk;
    if (y) y[g] = mk;
  }
}

// Partial |x|^2 of a vector (norm2_kernel), row 0 of the slot's partials.
template <class T, class B>
__device__ __noinline__ void phase_norm2(const SolveArgs<T, B>& S, const T* x, int64_t stride,
                                            const int* run) {
  typedef typename AccType<T>::type A;
  __shared__ double sh[8];
  for_vblocks(active_vblocks(S.N), S.nslot, run, [&](int k, int vb) {
    const T* v = x + k * stride;
    A sa = A(0);
    for (int64_t idx = (int64_t)vb * 256 + threadIdx.x; idx < S.N; idx += (int64_t)kRedBlocks * 256) {
      const A e = (A)__ldcg(v + idx);
      sa = fma_t(e, e, sa);
    }
    const double s = (double)warp_sum_t<A>(sa);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32) {
      double t = threadIdx.x < 8 ? sh[threadIdx.x] : 0.0;
      t = warp_sum(t);
      if (threadIdx.x == 0) S.red[(int64_t)k * S.sred + vb] = t;
    }
  });
}

// Sum of one row of a slot's partials over the first nvb virtual blocks (reduce_slots_kernel's
// order; the other partials are zero); valid in thread 0.  Every thread of the block calls.
__device__ __noinline__ double reduce_row(const double* __restrict__ row, int nvb) {
  __shared__ double sh[8];
  double x = 0.0;
  for (int b = threadIdx.x; b < nvb; b += 256) x = x + __ldcg(row + b);
  x = warp_sum(x);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x < 32) {
    x = threadIdx.x < 8 ? sh[threadIdx.x] : 0.0;
    x = warp_sum(x);
  }
  return x;
}

// Partial V_k . w (rows k < nv) and |w|^2 (row nv), as gs_dots_kernel; with the second pass
// (reorth) first w -= sum h_k V_k in place, as gs_update_kernel<GS_REORTH>.
constexpr int kDotChunk = 8;  // basis vectors whose accumulators a thread holds at a time
template <class T, class B>
__device__ __noinline__ void phase_dots(const SolveArgs<T, B>& S, int nv, bool reorth,
                                           const int* run, const int* second) {
  typedef typename AccType<T>::type A;
  typedef Pack16<T> P;
  typedef BasisIO<T, B> IO;
  constexpr int W = IO::W, NP = W / P::W;
  __shared__ double sh[kMaxRestart + 1][8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t ng = S.N / W;
  const int tail = (int)(S.N - ng * W);
  for_vblocks(active_vblocks(ng), S.nslot, run, [&](int k, int vb) {
    if (reorth && second[k] != 1) return;
    const B* V = S.V + (int64_t)k * S.sV;
    T* w = S.W.of(k);
    const int64_t g0 = (int64_t)vb * 256 + threadIdx.x;
    if (reorth) {
      const A* c = gs_coef<A>(S.g.dev + (int64_t)k * kGsLd, S.g.devf + (int64_t)k * kGsLd);
      for (int64_t g = g0; g < ng; g += (int64_t)kRedBlocks * 256) {
        A x[W];
#pragma unroll
        for (int p = 0; p < NP; ++p) vec_load_cg<T, A>(w, g * NP + p, x + p * P::W);
        for (int q = 0; q < nv; ++q) {
          A vk[W];
          basis_load_cg<T, B, A>(V + (int64_t)q * S.ldv, g, vk);
          const A cq = __ldcg(c + q);
#pragma unroll
          for (int e = 0; e < W; ++e) x[e] -= cq * vk[e];
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          P o;
#pragma unroll
          for (int e = 0; e < P::W; ++e) o.v[e] = (T)x[p * P::W + e];
          reinterpret_cast<P*>(w)[g * NP + p] = o;
        }
      }
      if (vb == 0 && (int)threadIdx.x < tail) {
        const int64_t i = ng * W + threadIdx.x;
        A x = (A)__ldcg(w + i);
        for (int q = 0; q < nv; ++q)
          x -= __ldcg(c + q) * basis_get_cg<T, B, A>(V + (int64_t)q * S.ldv, i);
        w[i] = (T)x;
      }
    }
    __syncthreads();  // sh of the item before
    for (int k0 = 0; k0 < nv; k0 += kDotChunk) {
      A acc[kDotChunk + 1];
#pragma unroll
      for (int q = 0; q <= kDotChunk; ++q) acc[q] = A(0);
      for (int64_t g = g0; g < ng; g += (int64_t)kRedBlocks * 256) {
        A wv[W];
#pragma unroll
        for (int p = 0; p < NP; ++p) vec_load_cg<T, A>(w, g * NP + p, wv + p * P::W);
        if (k0 == 0)
#pragma unroll
          for (int e = 0; e < W; ++e) acc[kDotChunk] = fma_t(wv[e], wv[e], acc[kDotChunk]);
#pragma unroll
        for (int q = 0; q < kDotChunk; ++q)
          if (k0 + q < nv) {
            A vk[W];
            basis_load_cg<T, B, A>(V + (int64_t)(k0 + q) * S.ldv, g, vk);
#pragma unroll
            for (int e = 0; e < W; ++e) acc[q] += vk[e] * wv[e];
          }
      }
      if (vb == 0 && (int)threadIdx.x < tail) {
        const int64_t i = ng * W + threadIdx.x;
        const A x = (A)__ldcg(w + i);
        if (k0 == 0) acc[kDotChunk] = fma_t(x, x, acc[kDotChunk]);
#pragma unroll
        for (int q = 0; q < kDotChunk; ++q)
          if (k0 + q < nv) acc[q] += basis_get_cg<T, B, A>(V + (int64_t)(k0 + q) * S.ldv, i) * x;
      }
      if (k0 == 0) {
        const A s = warp_sum_t<A>(acc[kDotChunk]);
        if (lane == 0) sh[nv][wid] = (double)s;
      }
      const int pos = warp_sums<kDotChunk, A>(acc);
      if (pos >= 0 && k0 + pos < nv) sh[k0 + pos][wid] = (double)acc[0];
    }
    __syncthreads();
    if ((int)threadIdx.x <= nv) {
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q) s += sh[threadIdx.x][q];
      S.red[(int64_t)k * S.sred + (int64_t)threadIdx.x * kRedBlocks + vb] = s;
    }
  });
}

// V_{j+1} = (w - sum_k c_k V_k) inv of the slots whose pass this is (gs_update_kernel FINAL1:
// second[k] == 0 with the coefficients at off 0; FINAL2: second[k] == 1 at off kGsH2).
template <class T, class B>
__device__ __noinline__ void phase_update(const SolveArgs<T, B>& S, int nv, int want, int off,
                                             const int* run, const int* second,
                                             const typename AccType<T>::type* inv_sh) {
  typedef typename AccType<T>::type A;
  typedef Pack16<T> P;
  typedef BasisIO<T, B> IO;
  constexpr int W = IO::W, NP = W / P::W;
  constexpr bool kCopy = !std::is_same<T, B>::value;
  __shared__ A cs[kMaxRestart];
  const int64_t ng = S.N / W;
  const int tail = (int)(S.N - ng * W);
  for_vblocks(active_vblocks(ng), S.nslot, run, [&](int k, int vb) {
    const A inv = inv_sh[k];
    if (second[k] != want || inv == A(0)) return;
    __syncthreads();
    if ((int)threadIdx.x < nv)
      cs[threadIdx.x] = __ldcg(gs_coef<A>(S.g.dev + (int64_t)k * kGsLd, S.g.devf + (int64_t)k * kGsLd) +
                               off + threadIdx.x);
    __syncthreads();
    const B* V = S.V + (int64_t)k * S.sV;
    B* out = S.V + (int64_t)k * S.sV + (int64_t)nv * S.ldv;
    T* outx = kCopy ? S.Vx.of(k) : nullptr;
    const T* w = S.W.of(k);
    for (int64_t g = (int64_t)vb * 256 + threadIdx.x; g < ng; g += (int64_t)kRedBlocks * 256) {
      A x[W];
#pragma unroll
      for (int p = 0; p < NP; ++p) vec_load_cg<T, A>(w, g * NP + p, x + p * P::W);
#pragma unroll 8
      for (int q = 0; q < nv; ++q) {
        A vk[W];
        basis_load_cg<T, B, A>(V + (int64_t)q * S.ldv, g, vk);
#pragma unroll
        for (int e = 0; e < W; ++e) x[e] -= cs[q] * vk[e];
      }
      A y[W];
#pragma unroll
      for (int e = 0; e < W; ++e) y[e] = (A)(T)(x[e] * inv);
      IO::store(out, g, y);
      if (kCopy) {
#pragma unroll
        for (int p = 0; p < NP; ++p) {
          P o;
#pragma unroll
          for (int e = 0; e < P::W; ++e) o.v[e] = (T)y[p * P::W + e];
          reinterpret_cast<P*>(outx)[g * NP + p] = o;
        }
      }
    }
    if (vb == 0 && (int)threadIdx.x < tail) {
      const int64_t i = ng * W + threadIdx.x;
      A x = (A)__ldcg(w + i);
      for (int q = 0; q < nv; ++q) x -= cs[q] * basis_get_cg<T, B, A>(V + (int64_t)q * S.ldv, i);
      const T y = (T)(x * inv);
      IO::template set<A>(out, i, (A)y);
      if (kCopy) outx[i] = y;
    }
  });
}

// First basis vector of a cycle, V_0 = r / beta (basis_start_kernel).
template <class T, class B>
__device__ __noinline__ void phase_basis_start(const SolveArgs<T, B>& S, const T* r, int64_t stride,
                                                  const int* run) {
  typedef typename AccType<T>::type A;
  constexpr bool kCopy = !std::is_same<T, B>::value;
  for_vblocks(active_vblocks(S.N), S.nslot, run, [&](int k, int vb) {
    const A s = (A)__ldcg(S.g.sc + 8 * k + 3);
    B* V0 = S.V + (int64_t)k * S.sV;
    T* x0 = kCopy ? S.Vx.of(k) : nullptr;
    for (int64_t i = (int64_t)vb * 256 + threadIdx.x; i < S.N; i += (int64_t)kRedBlocks * 256) {
      const T y = (T)((A)__ldcg(r + k * stride + i) * s);
      BasisIO<T, B>::template set<A>(V0, i, (A)y);
      if (kCopy) x0[i] = y;
    }
  });
}

// Rows of the slots' partials into dev (off) and their FP32 copies, one block per row.
template <class T, class B>
__device__ __noinline__ void phase_reduce(const SolveArgs<T, B>& S, int rows, int nvb, int off,
                                             const int* run, const int* second) {
  for (int it = blockIdx.x; it < rows * S.nslot; it += gridDim.x) {
    const int k = it / rows, row = it - k * rows;
    if (run[k] == 0 || (second && second[k] != 1)) continue;
    const double x = reduce_row(S.red + (int64_t)k * S.sred + (int64_t)row * kRedBlocks, nvb);
    if (threadIdx.x == 0) {
      S.g.dev[(int64_t)k * kGsLd + off + row] = x;
      S.g.devf[(int64_t)k * kGsLd + off + row] = (float)x;
    }
  }
}

// |w|^2 - |h|^2 of a slot (gs_decide's sum, in order), the same in every lane of the warp.
__device__ __forceinline__ double decide_norm2(const double* dev, int nv) {
  const int lane = threadIdx.x & 31;
  const double h = lane < nv ? __ldcg(dev + lane) : 0.0;
  const double nw2 = __ldcg(dev + nv);
  double s = 0.0;
  for (int q = 0; q < nv; ++q) {
    const double d = __shfl_sync(0xffffffffu, h, q);
    s = fma(d, d, s);
  }
  return nw2 - s;
}

// y = H^{-1} g of one slot by one warp (gmres_solve_y_kernel): a row's products at once, then
// its subtractions in series.
__device__ __noinline__ void solve_y_warp(const GmresDev& g, int t) {
  __shared__ double prod[kMaxRestart];
  const int lane = threadIdx.x & 31;
  const double* H = g.H + (int64_t)t * kHsize;
  const double* gg = g.g + (int64_t)t * (kMaxRestart + 1);
  const int j = __ldcg(g.jc + t);
  double y = 0.0;  // lane k: y_k
  for (int i = j - 1; i >= 0; --i) {
    if (lane > i && lane < j) prod[lane] = __dmul_rn(__ldcg(H + i * kHld + lane), y);
    __syncwarp();
    double s = __ldcg(gg + i);
    for (int k = i + 1; k < j; ++k) s = __dsub_rn(s, prod[k]);
    const double yi = s / __ldcg(H + i * kHld + i);
    if (lane == i) y = yi;
    __syncwarp();
  }
  if (lane < j) g.y[(int64_t)t * kMaxRestart + lane] = y;
}

template <class T, class B, bool PACKED>
__global__ void __launch_bounds__(256, std::is_same<T, double>::value ? 1 : 2) gmres_solve_kernel(const __grid_constant__ SolveArgs<T, B> args) {
  typedef typename AccType<T>::type A;
  __shared__ A inv_sh[kMaxSlots];
  __shared__ int second_sh[kMaxSlots];
  __shared__ int run_sh[kMaxSlots];  // the flags of the current phases
  // the arguments in shared memory: the phases are functions of their own (inlined into one body
  // they spill 500 to 1400 bytes, and a spilled register comes back from L2 behind every barrier;
  // as functions 68 bytes in FP32 and none in FP64)
  __shared__ __align__(16) unsigned char args_sh[sizeof(SolveArgs<T, B>)];
  for (unsigned q = threadIdx.x; q < sizeof(SolveArgs<T, B>) / 4; q += 256)
    reinterpret_cast<unsigned*>(args_sh)[q] = reinterpret_cast<const unsigned*>(&args)[q];
  __syncthreads();
  const SolveArgs<T, B>& S = *reinterpret_cast<const SolveArgs<T, B>*>(args_sh);
  if (*(volatile int*)S.bar.error) return;
  unsigned target = 0;  // thread 0's barrier count
  const int tid = threadIdx.x, ns = S.nslot;
  const GmresDev& g = S.g;
  const int nvb_n = active_vblocks(S.N), nvb_g = active_vblocks(S.N / BasisIO<T, B>::W);
  const bool lead = blockIdx.x == 0 && tid == 0;
  auto bar = [&] { return grid_barrier(S.bar, target); };
  auto stamp = [&](int cat, int begin) {
    if (!lead || S.prof == nullptr) return;
    const unsigned long long t = global_ns();
    if (begin) {
      S.prof[cat] = t;
    } else {
      S.prof[PROF_NCAT + cat] += t - S.prof[cat];
      S.prof[2 * PROF_NCAT + cat] += 1;
    }
  };
  // takes the flags into run_sh
  auto any = [&](const int32_t* flags) {
    int f = 0;
    __syncthreads();
    for (int k = tid; k < ns; k += 256) {
      const int v = __ldcg(flags + k);
      run_sh[k] = v;
      f |= v;
    }
    return __syncthreads_or(f) != 0;
  };
  // slots dealt to blocks from the last one, which has the least of the other work
  auto slot_block = [&](int k) { return (int)(gridDim.x - 1 - k % gridDim.x); };

  // ---- start: x = 0, beta = |b|, v_0 = b / beta (zero, norm2, gmres_init, basis_start)
  stamp(PROF_ORTHO, 1);
  any(S.act);
  for_vblocks(nvb_n, ns, run_sh, [&](int k, int vb) {
    T* x = S.X.of(k);
    for (int64_t i = (int64_t)vb * 256 + tid; i < S.N; i += (int64_t)kRedBlocks * 256) x[i] = T(0);
    set_marks(S, k, vb);
  });
  phase_norm2(S, S.b.p, S.b.stride, run_sh);
  if (!bar()) return;
  for (int k = 0; k < ns; ++k) {
    if (slot_block(k) != (int)blockIdx.x) continue;
    int lin = 0;
    if (run_sh[k]) {
      const double r2 = reduce_row(S.red + (int64_t)k * S.sred, nvb_n);
      if (tid == 0) {
        g.dev[(int64_t)k * kGsLd + kGsR] = r2;
        lin = gmres_init_slot(g, S.P, k, r2, *S.nan_flag);
      }
    }
    if (tid == 0) {
      g.lin[k] = lin;
      g.cyc[k] = lin;
    }
  }
  if (!bar()) return;
  any(g.lin);
  phase_basis_start(S, S.b.p, S.b.stride, run_sh);
  if (!bar()) return;
  stamp(PROF_ORTHO, 0);

  while (any(g.lin)) {
    for (int j = 0; j < S.P.mr; ++j) {
      if (!any(g.cyc)) break;
      const int nv = j + 1;
      stamp(PROF_PRECOND, 1);
      const T* in;
      int64_t in_stride;
      if constexpr (std::is_same<T, B>::value) {
        in = (const T*)(S.V + (int64_t)j * S.ldv);
        in_stride = S.sV;
      } else {
        in = S.Vx.p;
        in_stride = S.Vx.stride;
      }
      phase_precond<T, B, PACKED>(S, in, in_stride, run_sh);
      stamp(PROF_PRECOND, 0);
      stamp(PROF_SPMV, 1);
      phase_spmv<T, B, PACKED, false>(S, run_sh);
      if (!bar()) return;
      stamp(PROF_SPMV, 0);
      stamp(PROF_ORTHO, 1);
      phase_dots(S, nv, false, run_sh, second_sh);
      if (!bar()) return;
      phase_reduce(S, nv + 1, nvb_g, 0, run_sh, nullptr);
      if (!bar()) return;
      // gs_decide stage 1, by every block, a warp per slot
      int re = 0;
      for (int k = tid >> 5; k < ns; k += 8) {
        if (!run_sh[k]) continue;
        double* dev = g.dev + (int64_t)k * kGsLd;
        const double est = decide_norm2(dev, nv);
        const double nw2 = __ldcg(dev + nv);
        const bool reorth = !(est > kReorthTheta2 * nw2);
        const double hn = reorth ? 0.0 : sqrt(est);
        const double inv = hn > 0.0 ? 1.0 / hn : 0.0;
        re |= reorth;
        if ((tid & 31) == 0) {
          inv_sh[k] = (A)inv;
          second_sh[k] = reorth;
          if (slot_block(k) == (int)blockIdx.x) {
            dev[kGsFlag] = reorth ? 1.0 : 0.0;
            dev[kGsNorm] = hn;
          }
        }
      }
      const bool pass2 = __syncthreads_or(re) != 0;
      if (!pass2) {
        // the rotations run beside the update of the new basis vector
        for (int k = tid >> 5; k < ns; k += 8)
          if (slot_block(k) == (int)blockIdx.x && run_sh[k]) givens_warp(g, S.P, k, j);
      }
      phase_update(S, nv, 0, 0, run_sh, second_sh, inv_sh);
      for_vblocks(nvb_n, ns, run_sh, [&](int k, int vb) { set_marks(S, k, vb); });
      if (!bar()) return;
      if (pass2) {
        phase_dots(S, nv, true, run_sh, second_sh);
        if (!bar()) return;
        phase_reduce(S, nv + 1, nvb_g, kGsH2, run_sh, second_sh);
        if (!bar()) return;
        // gs_decide_kernel
        for (int k = tid >> 5; k < ns; k += 8) {
          if (!run_sh[k] || second_sh[k] != 1) continue;
          double* dev = g.dev + (int64_t)k * kGsLd;
          const double e2 = decide_norm2(dev + kGsH2, nv);
          const double hn = e2 > 0.0 ? sqrt(e2) : 0.0;
          if ((tid & 31) == 0) {
            inv_sh[k] = (A)(hn > 0.0 ? 1.0 / hn : 0.0);
            if (slot_block(k) == (int)blockIdx.x) dev[kGsNorm] = hn;
          }
        }
        __syncthreads();
        for (int k = tid >> 5; k < ns; k += 8)
          if (slot_block(k) == (int)blockIdx.x && run_sh[k]) givens_warp(g, S.P, k, j);
        phase_update(S, nv, 1, kGsH2, run_sh, second_sh, inv_sh);
        if (!bar()) return;
        if (lead) ++g.counters[2];
      }
      if (lead) ++g.counters[0];
      stamp(PROF_ORTHO, 0);
    }
    // ---- end of a cycle: x += M^{-1} V y, r = b - A x, restart or stop
    stamp(PROF_ORTHO, 1);
    any(g.lin);
    for (int k = 0; k < ns; ++k)
      if (tid < 32 && slot_block(k) == (int)blockIdx.x && run_sh[k]) solve_y_warp(g, k);
    if (!bar()) return;
    for_vblocks(nvb_n, ns, run_sh, [&](int k, int vb) {
      __shared__ A ys[kMaxRestart];
      const int nv = __ldcg(g.jc + k);
      __syncthreads();
      if (tid < nv) ys[tid] = (A)__ldcg(g.y + (int64_t)k * kMaxRestart + tid);
      __syncthreads();
      const B* V = S.V + (int64_t)k * S.sV;
      T* w = S.W.of(k);
      for (int64_t i = (int64_t)vb * 256 + tid; i < S.N; i += (int64_t)kRedBlocks * 256) {
        A x = A(0);
#pragma unroll 8
        for (int q = 0; q < nv; ++q) x += ys[q] * basis_get_cg<T, B, A>(V + (int64_t)q * S.ldv, i);
        w[i] = (T)x;
      }
    });
    if (!bar()) return;
    stamp(PROF_ORTHO, 0);
    stamp(PROF_PRECOND, 1);
    phase_precond<T, B, PACKED>(S, S.W.p, S.W.stride, run_sh);
    if (!bar()) return;
    stamp(PROF_PRECOND, 0);
    stamp(PROF_SPMV, 1);
    for_vblocks(nvb_n, ns, run_sh, [&](int k, int vb) {
      T* x = S.X.of(k);
      const T* z = S.Z.of(k);
      for (int64_t i = (int64_t)vb * 256 + tid; i < S.N; i += (int64_t)kRedBlocks * 256)
        x[i] = __ldcg(x + i) + __ldcg(z + i);
    });
    if (!bar()) return;
    phase_spmv<T, B, PACKED, true>(S, run_sh);
    if (!bar()) return;
    stamp(PROF_SPMV, 0);
    stamp(PROF_ORTHO, 1);
    phase_norm2(S, S.W.p, S.W.stride, run_sh);
    if (!bar()) return;
    for (int k = 0; k < ns; ++k) {
      if (slot_block(k) != (int)blockIdx.x || !run_sh[k]) continue;
      const double r2 = reduce_row(S.red + (int64_t)k * S.sred, nvb_n);
      if (tid == 0) {
        g.dev[(int64_t)k * kGsLd + kGsR] = r2;
        const int lin = gmres_restart_slot(g, S.P, k, r2, *S.guard);
        g.lin[k] = lin;
        g.cyc[k] = lin;
      }
      __syncthreads();
    }
    if (!bar()) return;
    any(g.lin);
    phase_basis_start(S, S.W.p, S.W.stride, run_sh);
    for_vblocks(nvb_n, ns, run_sh, [&](int k, int vb) { set_marks(S, k, vb); });
    if (lead) ++g.counters[1];
    if (!bar()) return;
    stamp(PROF_ORTHO, 0);
  }
}

}  // namespace bes
