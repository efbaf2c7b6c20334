// Batched H-matrix-vector product over all leaves (sm_100a).
//
// Restates HMatrix<T>::gemv (h_matrix.cpp:792-857) with its leaf products
// (ScalarArray::gemm, scalar_array.cpp:413-443; RkMatrix::gemv, rk_matrix.cpp:156-206) and the
// reorderVector / restoreVectorOrder permutations of the C wrapper (h_matrix.cpp:75-141,
// c_wrapping.hpp:233-252), as a few launches over device-resident schedules (gemv_plan.h):
//
//   gather   xz[i][q] = x[perm[i] + q ld]           client -> cluster order, row-major
//   'N': z-phase  z = B^T x_J, one task per group of Rk leaves with one column range (chunks for
//                 long ones, summed afterwards)
//        y-phase  partial rows of sum (F x | A z), the output blocks' matrices streamed
//   'T': column pass  every column of every output block's matrix times the block's x rows: the
//                 full leaves' share of y and the z' = A^T x parts of the Rk leaves
//        z'-sum   the parts of leaves over several blocks
//        group pass  partial rows of sum B z' per output block, over the B^T groups
//   final    y = beta y + alpha sum of a row's parts, in client order
//
// Every task streams its units (contiguous pieces of the leaf arena and of the xz buffer)
// through per-warp shared-memory pipelines filled by TMA bulk copies (cp.async.bulk, completion
// on an mbarrier), on a persistent grid cut into ranges of about equal bytes.  Sums run in a
// fixed order, so repeated products are bitwise identical.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include "gemv_plan.h"
#include "kernels.h"

namespace hmatb200 {
size_t warp_stream_smem_bytes(int elem_bytes);
namespace {

// ---------------------------------------------------------------------------------
// TMA bulk copy + mbarrier helpers
__device__ inline uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Programmatic dependent launch.  The kernels after the gather in a product are launched with
// programmatic stream serialization (launch_pdl) and start with pdl_wait(), which returns once
// the kernel before them on the stream has completed and its writes are visible (for a kernel
// launched normally it returns at once).  No kernel triggers its dependents early: their launch
// then overlaps only the end of the kernel before them (100,000-point cylinder, FP32, graph
// replay: 0.250 -> 0.247 ms).  Triggering at the start of every kernel let the next grid be
// scheduled beside the persistent kernels and took the product to 0.285 ms.
__device__ inline void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ inline void mbar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ inline void mbar_fence_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ inline void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ inline void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// L2 policies of the streamed copies: a leaf piece is read once per product (evict first), the
// x / z rows by every unit over their columns (evict last), so that the stream of pieces does
// not push the vector rows out of L2 and the units read them from DRAM again (100,000-point
// cylinder, 16 right-hand sides: FP32 product 0.248 -> 0.2435 ms, FP64 0.750 -> 0.743 ms).
__device__ inline uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ inline uint64_t policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ inline void bulk_g2s_hint(void* dst, const void* src, uint32_t bytes, uint64_t* bar, uint64_t pol) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(pol)
      : "memory");
}
// A leaf piece, and the X rows of a unit.
__device__ inline void bulk_piece(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  bulk_g2s_hint(dst, src, bytes, bar, policy_evict_first());
}
__device__ inline void bulk_xrows(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  bulk_g2s_hint(dst, src, bytes, bar, policy_evict_last());
}
__device__ inline bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait for a barrier phase: false once `limit` polls went by without it completing.
// A negative limit gives up at once (a test mode of the status path: the caller still drains
// its copies with a positive limit before it stops).
__device__ inline bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, long long limit) {
  if (limit < 0) return false;
  long long spins = 0;
  while (!mbar_try_wait(bar, parity))
    if (++spins > limit) return false;
  return true;
}

// A warp whose wait gave up: sets the status flag, then waits (bounded) for the copies of
// the units it has issued and not consumed (u .. last_issued, one stage each) to land, so
// that no bulk copy is still writing its shared memory when it exits.
__device__ inline long long drain_limit(const GemvStatus* st) {
  return st->wait_limit > 0 && st->wait_limit < kGemvDrainLimit ? st->wait_limit : kGemvDrainLimit;
}
__device__ inline void warp_give_up(GemvStatus* st, uint64_t* bars, int nstages, int u_begin, int u, int last_issued) {
  atomicCAS(&st->failed, 0, 1);
  const long long lim = drain_limit(st);
  for (int v = u; v <= last_issued; ++v)
    mbar_wait_bounded(&bars[(v - u_begin) % nstages], (uint32_t)(((v - u_begin) / nstages) & 1), lim);
}

__device__ inline uint32_t round16(uint64_t b) { return (uint32_t)((b + 15) & ~15ull); }

__device__ inline float shfl_xor(float v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ inline double shfl_xor(double v, int m) { return __shfl_xor_sync(0xffffffffu, v, m); }
__device__ inline cfloat shfl_xor(cfloat v, int m) {
  return cfloat{__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m)};
}
__device__ inline cdouble shfl_xor(cdouble v, int m) {
  return cdouble{__shfl_xor_sync(0xffffffffu, v.x, m), __shfl_xor_sync(0xffffffffu, v.y, m)};
}

// Loads Q consecutive elements from shared memory (vectorised when aligned).
template <typename T, int Q>
__device__ inline void lds_vec(const T* p, T (&out)[Q]) {
  constexpr int bytes = Q * (int)sizeof(T);
  if constexpr (bytes % 16 == 0) {
    const uint4* s = reinterpret_cast<const uint4*>(p);
    uint4* d = reinterpret_cast<uint4*>(out);
#pragma unroll
    for (int c = 0; c < bytes / 16; ++c) d[c] = s[c];
  } else if constexpr (bytes % 8 == 0) {
    const uint2* s = reinterpret_cast<const uint2*>(p);
    uint2* d = reinterpret_cast<uint2*>(out);
#pragma unroll
    for (int c = 0; c < bytes / 8; ++c) d[c] = s[c];
  } else {
#pragma unroll
    for (int c = 0; c < Q; ++c) out[c] = p[c];
  }
}

template <typename T>
constexpr int rs_of(int R) {
  return R * (int)sizeof(T) >= 16 ? R : (16 / (int)sizeof(T));
}

// ---------------------------------------------------------------------------------
// x (client order, column-major with leading dimension ldx; right-hand sides q0 .. q0 + R - 1
// of r) into xz in cluster order (row-major, RS columns, zeros past R).  A CTA takes
// kGatherRows client rows: it reads each column of x along the rows (coalesced), transposes
// through shared memory, and writes each client row's RS values as one contiguous xz row at
// its cluster position iperm[j].  One more CTA clears the kZeroRows zero rows from row `zrow0`
// (the X rows of the y matrices' padding columns).
constexpr int kGatherRows = 64;
template <typename T, int R, int RS>
__global__ void __launch_bounds__(256) gather_kernel(const T* __restrict__ x, int N, int ldx, int q0, int r,
                                                     const int* __restrict__ iperm, T* __restrict__ xz, int zrow0) {
  __shared__ T tile[RS][kGatherRows + 1];
  const int nblk = (N + kGatherRows - 1) / kGatherRows;
  if ((int)blockIdx.x >= nblk) {
    for (int e = threadIdx.x; e < kZeroRows * RS; e += blockDim.x) xz[(size_t)zrow0 * RS + e] = zero<T>();
    return;
  }
  const int j0 = blockIdx.x * kGatherRows;
  for (int e = threadIdx.x; e < RS * kGatherRows; e += blockDim.x) {
    const int q = e / kGatherRows, jl = e % kGatherRows, j = j0 + jl;
    T v = zero<T>();
    if (j < N && q < R && q0 + q < r) v = x[(size_t)j + (size_t)(q0 + q) * ldx];
    tile[q][jl] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < RS * kGatherRows; e += blockDim.x) {
    const int jl = e / RS, q = e % RS, j = j0 + jl;
    if (j < N) xz[(size_t)iperm[j] * RS + q] = tile[q][jl];
  }
}
inline unsigned gather_grid(int N) { return (unsigned)((N + kGatherRows - 1) / kGatherRows + 1); }

// Checks a unit's copies into a warp-level stage before they are issued: 16-byte sizes and
// addresses (the bulk-copy rule), the piece below the X rows, the X rows inside the stage, and
// runs that cover exactly its columns.  A unit that fails is not copied: the stage's barrier
// gets a plain arrival (so nothing waits for it), and the status block records code 2 and the
// unit's index.
template <typename T, int RS>
__device__ inline bool unit_copies_ok(const GemvUnit& U, const T* arena, const T* xz, int stage_bytes, int xoff) {
  const uint64_t pbytes = round16((uint64_t)U.pel * sizeof(T));
  const uint64_t xbytes = (uint64_t)U.c * RS * sizeof(T);
  if (U.c <= 0 || U.pel <= 0 || (reinterpret_cast<uintptr_t>(arena + U.poff) & 15) != 0) return false;
  if (xoff < (int)pbytes || xoff % 16 != 0 || (uint64_t)xoff + xbytes > (uint64_t)stage_bytes) return false;
  if (((size_t)RS * sizeof(T)) % 16 != 0) return false;
  if (U.nruns < 0 || U.nruns > kUnitRuns) return false;
  if (U.nruns > 0) {
    int rows = 0;
    for (int r = 0; r < kUnitRuns; ++r)
      if (r < U.nruns) rows += U.run_len[r];
    if (rows != U.c) return false;
  }
  return true;
}
__device__ inline void record_bad_unit(GemvStatus* st, int u) {
  atomicExch(&st->failed, 2);
  atomicExch(&st->pad, u);
}

// The X rows of a unit into a pipeline stage: one bulk copy, or one per run.
template <typename T, int RS>
__device__ inline void issue_x(unsigned char* dst, const T* xz, const GemvUnit& U, uint64_t* bar) {
  if (U.nruns == 0) {
    bulk_xrows(dst, xz + (size_t)U.xrow * RS, (uint32_t)U.c * RS * (uint32_t)sizeof(T), bar);
    return;
  }
  uint32_t off = 0;
#pragma unroll
  for (int r = 0; r < kUnitRuns; ++r) {  // constant indices: the descriptor stays in registers
    if (r < U.nruns) {
      const uint32_t b = (uint32_t)U.run_len[r] * RS * (uint32_t)sizeof(T);
      bulk_xrows(dst + off, xz + (size_t)U.run_row[r] * RS, b, bar);
      off += b;
    }
  }
}

// ---------------------------------------------------------------------------------
// The descriptors of the next unit and the next task a warp-level kernel issues, prefetched one
// issue ahead.  LANES = true spreads each over the warp's lanes, one 32-bit word a lane, and
// gathers it with shuffles when it is used (every lane calls get()), instead of holding it whole
// in every lane's registers through the unit's sums.  The FP64 y-phase kernel then keeps its
// accumulators without spilling (100,000-point cylinder, 16 right-hand sides: y-phase 0.393 ->
// 0.340 ms) and the FP32 one with up to 8 tiles schedules better (0.128 -> 0.1245 ms); the
// column-slice z kernels keep the whole copy (the FP64 one is slower with the shuffles, 0.349 ->
// 0.362 ms), and so does the 16-tile FP32 kernel (it spills more with them).
constexpr int kUnitWords = (int)(sizeof(GemvUnit) / 4);
constexpr int kTaskWords = (int)(sizeof(GemvTask) / 4);
static_assert(sizeof(GemvUnit) % 4 == 0 && kUnitWords <= 32, "unit descriptor words");
static_assert(sizeof(GemvTask) % 4 == 0 && kTaskWords <= 32, "task descriptor words");
template <typename D, int W>
__device__ __forceinline__ D from_lanes(uint32_t w) {
  D d;
  uint32_t* p = reinterpret_cast<uint32_t*>(&d);
#pragma unroll
  for (int i = 0; i < W; ++i) p[i] = __shfl_sync(0xffffffffu, w, i);
  return d;
}
template <bool LANES>
struct NextUnit {  // lane 0 holds the descriptor
  GemvUnit d;
  __device__ void load(const GemvUnit* units, int v, int lane) {
    if (lane == 0) d = units[v];
  }
  __device__ GemvUnit get() const { return d; }
};
template <>
struct NextUnit<true> {  // lane l < kUnitWords holds word l
  uint32_t w = 0;
  __device__ void load(const GemvUnit* units, int v, int lane) {
    w = lane < kUnitWords ? __ldg(reinterpret_cast<const uint32_t*>(units + v) + lane) : 0u;
  }
  __device__ GemvUnit get() const { return from_lanes<GemvUnit, kUnitWords>(w); }
};
template <bool LANES>
struct NextTask {  // every lane holds the descriptor
  GemvTask d;
  __device__ void load(const GemvTask* tasks, int t, int /*lane*/) { d = tasks[t]; }
  __device__ GemvTask get() const { return d; }
};
template <>
struct NextTask<true> {  // lane l < kTaskWords holds word l
  uint32_t w = 0;
  __device__ void load(const GemvTask* tasks, int t, int lane) {
    w = lane < kTaskWords ? __ldg(reinterpret_cast<const uint32_t*>(tasks + t) + lane) : 0u;
  }
  __device__ GemvTask get() const { return from_lanes<GemvTask, kTaskWords>(w); }
};

// ---------------------------------------------------------------------------------
// Warp-level streamed tasks (the 'N' products).  Every warp owns a contiguous range of whole
// tasks and runs its own two-stage TMA pipeline: lane 0 copies the unit descriptor into the
// stage and issues the unit's bulk copies (P piece; X rows at the unit's byte offset o0 in the
// stage, right after the piece), completion on the stage's
// mbarrier, so warps never wait for one another.  Lane maps (output rows O of the task):
//   MODE 2 (O <= 32): the warp is a window of floor(32 / O) column slices x O rows, lane =
//          slice * O + row; P is read as one contiguous run per step (no bank conflicts);
//          the slices are summed through shared memory at the end of the task.
//   MODE 1 (O <= 16 * A2): two column slices (half-warps) x 16 rows, A2 rows per lane
//          (row, row + 16, ...); slices summed with one shuffle.
//   MODE 0 (O <= 32 * A2): lanes over rows, A2 rows per lane, one slice.
// Row groups above O are skipped warp-uniformly.  Every lane keeps all R right-hand sides
// of its rows; float sums use the paired FMA (fma.rn.f32x2: two IEEE fmaf per
// instruction).  Summation orders are fixed, so repeated products are bitwise identical.
constexpr int kWarpCTA = 4;
constexpr int kWarpStages = 2;
__host__ __device__ constexpr int warp_stage_bytes(int elem_bytes) { return warp_piece_bytes(elem_bytes) + kWarpXBytes; }

// R accumulators of one output row, and one X row as the FMAs consume it.
template <typename T, int R, bool PAIR = std::is_same<T, float>::value && (R % 2 == 0)>
struct RowOps {
  using XV = T[R];
  using AV = T[R];
  __device__ static void load(const T* p, XV& x) { lds_vec<T, R>(p, x); }
  __device__ static void zero_(AV& a) {
#pragma unroll
    for (int q = 0; q < R; ++q) a[q] = zero<T>();
  }
  __device__ static void fma(T p, const XV& x, AV& a) {
#pragma unroll
    for (int q = 0; q < R; ++q) a[q] = fmadd(p, x[q], a[q]);
  }
  __device__ static T get(const AV& a, int q) { return a[q]; }
};
template <int R>
struct RowOps<float, R, true> {
  static constexpr int N = R / 2;
  using XV = unsigned long long[N];
  using AV = unsigned long long[N];
  __device__ static void load(const float* p, XV& x) {
    if constexpr (R % 4 == 0) {
      const ulonglong2* s = reinterpret_cast<const ulonglong2*>(p);
#pragma unroll
      for (int c = 0; c < R / 4; ++c) {
        const ulonglong2 v = s[c];
        x[2 * c] = v.x;
        x[2 * c + 1] = v.y;
      }
    } else {
      const unsigned long long* s = reinterpret_cast<const unsigned long long*>(p);
#pragma unroll
      for (int c = 0; c < N; ++c) x[c] = s[c];
    }
  }
  __device__ static void zero_(AV& a) {
#pragma unroll
    for (int i = 0; i < N; ++i) a[i] = 0ull;  // the bits of (+0.0f, +0.0f)
  }
  __device__ static void fma(float p, const XV& x, AV& a) {
    unsigned long long pp;
    asm("mov.b64 %0, {%1, %1};" : "=l"(pp) : "f"(p));
#pragma unroll
    for (int i = 0; i < N; ++i) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(a[i]) : "l"(pp), "l"(x[i]));
  }
  __device__ static float get(const AV& a, int q) {
    float lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a[q / 2]));
    return (q & 1) ? hi : lo;
  }
};

// One unit of a warp task: lane's rows row0 + a * stride (a < NA) of the columns
// j = js, js + SL, ... < c, all R right-hand sides.
// O is the column stride of the piece.  With `active` >= 0 only the first `active` row
// groups are computed (a guarded loop).
// UNROLL: columns a loop iteration takes (4 for the lanes-over-rows maps, 1 for the
// column-slice windows: FP64 y-phase 0.345 -> 0.331 ms, z-phase 0.334 -> 0.333 ms against 2 for
// both on the 100,000-point cylinder, 16 right-hand sides).
template <typename T, int R, int RS, int NA, int A2, int UNROLL>
__device__ __forceinline__ void rows_loop(const T* P, const T* X, int c, int js, int SL, int O, int row0, int stride,
                                          typename RowOps<T, R>::AV (&acc)[A2], int active = -1) {
  using Ops = RowOps<T, R>;
#pragma unroll UNROLL
  for (int j = js; j < c; j += SL) {
    typename Ops::XV xv;
    Ops::load(X + (size_t)j * RS, xv);
    const T* pc = P + (size_t)j * O + row0;
#pragma unroll
    for (int a = 0; a < NA; ++a)
      if (active < 0 || a < active) Ops::fma(pc[a * stride], xv, acc[a]);
  }
}

// Blocks per SM the register budget allows: more accumulator bytes, fewer resident warps.
template <typename T, int R, int A2>
constexpr int warp_min_blocks() {
  return A2 * R * (int)sizeof(T) <= 256 ? 4 : 2;
}

template <typename T, int R, int RS, int MODE, int A2>
__global__ void __launch_bounds__(kWarpCTA * 32, (warp_min_blocks<T, R, A2>()))
    warp_stream_kernel(const GemvTask* __restrict__ tasks, const int* __restrict__ warp_begin,
                       const GemvUnit* __restrict__ units, const T* __restrict__ arena, T* xz, GemvStatus* err) {
  using Ops = RowOps<T, R>;
  constexpr int OL = MODE == 0 ? 32 : 16;
  // MODE 2: right-hand sides per round of the slice sums (a power of two)
  constexpr int QC0 = warp_piece_bytes((int)sizeof(T)) / (32 * A2 * (int)sizeof(T));
  constexpr int QC1 = QC0 >= 16 ? 16 : (QC0 >= 8 ? 8 : (QC0 >= 4 ? 4 : (QC0 >= 2 ? 2 : 1)));
  constexpr int QC2 = QC1 < R ? QC1 : R, QC = R % QC2 == 0 ? QC2 : 4;
  static_assert(QC >= 1 && (R % QC) == 0, "reduction chunk");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* wbase = smem_raw + (size_t)warp * kWarpStages * warp_stage_bytes((int)sizeof(T));
  // per stage: the unit's column count and X offset (what the consumers read), then the barriers
  int2* uslot =
      reinterpret_cast<int2*>(smem_raw + (size_t)kWarpCTA * kWarpStages * warp_stage_bytes((int)sizeof(T))) + warp * kWarpStages;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + (size_t)kWarpCTA * kWarpStages *
                                                               (warp_stage_bytes((int)sizeof(T)) + sizeof(int2))) +
                   warp * kWarpStages;
  const int gw = blockIdx.x * kWarpCTA + warp;
  const int t0 = warp_begin[gw], t1 = warp_begin[gw + 1];
  if (t0 >= t1) return;
  const int u_begin = tasks[t0].first_unit;
  const int u_end = tasks[t1 - 1].first_unit + tasks[t1 - 1].nunits;
  const long long wlim = err->wait_limit;

  if (lane == 0) {
    for (int s = 0; s < kWarpStages; ++s) mbar_init(&bars[s], 1);
    mbar_fence_init();
  }
  __syncwarp();
  // lane 0: descriptor into the stage, then the unit's two bulk copies.  The descriptor of
  // the next unit to issue is loaded one issue ahead, off the critical path.
  constexpr bool kLanes = MODE != 2;
  NextUnit<kLanes> nxt;
  int last_issued = u_begin - 1;  // lane 0: the last unit whose copies were issued
  auto issue = [&](int u, const GemvUnit& U) {
    const int s = (u - u_begin) % kWarpStages;
    last_issued = u;
    uslot[s] = make_int2(U.c, U.o0);
    const uint32_t pbytes = round16((uint64_t)U.pel * sizeof(T));
    const uint32_t xbytes = (uint32_t)U.c * RS * (uint32_t)sizeof(T);
    unsigned char* st = wbase + (size_t)s * warp_stage_bytes((int)sizeof(T));
    if (!unit_copies_ok<T, RS>(U, arena, xz, warp_stage_bytes((int)sizeof(T)), U.o0)) {
      record_bad_unit(err, u);
      mbar_arrive(&bars[s]);
      return;
    }
    mbar_expect_tx(&bars[s], pbytes + xbytes);
    bulk_piece(st, arena + U.poff, pbytes, &bars[s]);
    issue_x<T, RS>(st + U.o0, xz, U, &bars[s]);
  };
  auto issue_next = [&](int v) {  // nxt holds units[v]; kLanes: every lane calls it, else lane 0
    const GemvUnit U = nxt.get();
    if (lane == 0) issue(v, U);
    if (v + 1 < u_end) nxt.load(units, v + 1, lane);
  };
  if (lane == 0)
    for (int v = u_begin; v < u_end && v < u_begin + kWarpStages; ++v) issue(v, units[v]);
  if (u_begin + kWarpStages < u_end) nxt.load(units, u_begin + kWarpStages, lane);

  int u = u_begin;
  NextTask<kLanes> task_next;
  task_next.load(tasks, t0, lane);
  for (int t = t0; t < t1; ++t) {
    const GemvTask task = task_next.get();
    if (t + 1 < t1) task_next.load(tasks, t + 1, lane);
    const int O = task.O;
    int row0, js, SL, Og = O;
    float inv = 1.f;
    if constexpr (MODE == 2) {
      // window: Og = ceil(O / A2) lanes per column, SL = floor(32 / Og) columns per step;
      // exact for lane < 32 and Og <= 32 (the quotients are at least 1/64 from integers)
      Og = (O + A2 - 1) / A2;
      inv = __frcp_rn((float)Og);
      SL = (int)(32.5f * inv);
      js = (int)(((float)lane + 0.5f) * inv);
      row0 = lane - js * Og;
    } else if constexpr (MODE == 1) {
      SL = 2;
      row0 = lane & 15;
      js = lane >> 4;
    } else {
      SL = 1;
      row0 = lane;
      js = 0;
    }
    // row groups holding rows of this task (warp-uniform)
    const int na = MODE == 2 ? A2 : min(A2, (O + OL - 1) / OL);
    typename Ops::AV acc[A2];
#pragma unroll
    for (int a = 0; a < A2; ++a) Ops::zero_(acc[a]);

    int s = 0;
    for (int kk = 0; kk < task.nunits; ++kk, ++u) {
      s = (u - u_begin) % kWarpStages;
      const uint32_t parity = (uint32_t)(((u - u_begin) / kWarpStages) & 1);
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bars[s], parity, wlim))) {
        // a copy did not land in time: flag it, let the copies in flight land, stop the warp
        if (lane == 0) warp_give_up(err, bars, kWarpStages, u_begin, u, last_issued);
        return;
      }
      const int c = uslot[s].x;
      const T* P = reinterpret_cast<const T*>(wbase + (size_t)s * warp_stage_bytes((int)sizeof(T)));
      const T* X = reinterpret_cast<const T*>(wbase + (size_t)s * warp_stage_bytes((int)sizeof(T)) + uslot[s].y);
      // Rows of a lane past O read the next column (or, in the last column, the first
      // elements of the X rows of the same stage); they are never written.
      if constexpr (MODE == 2) {
        if (js < SL) rows_loop<T, R, RS, A2, A2, 1>(P, X, c, js, SL, O, row0, Og, acc);
      } else {
        rows_loop<T, R, RS, A2, A2, 4>(P, X, c, js, SL, O, row0, OL, acc, na);
      }
      __syncwarp();  // every lane is done with stage s
      // the last unit's stage stays free until the epilogue has used it as scratch
      if ((kLanes || lane == 0) && kk + 1 < task.nunits && u + kWarpStages < u_end) issue_next(u + kWarpStages);
    }

    // ---- epilogue: the task's rows go to xz[out_row + l], zero-padded to RS ----
    T* out = xz + (size_t)task.out_row * RS;
    if constexpr (MODE == 2) {
      // slices summed in slice order through the stage just consumed, QC right-hand sides
      // per round: lane's partial of (its row a, q) at sc[(lane * A2 + a) * QC + q - q0]
      T* sc = reinterpret_cast<T*>(wbase + (size_t)s * warp_stage_bytes((int)sizeof(T)));
      if (task.nunits > 0) {
#pragma unroll
        for (int qc0 = 0; qc0 < R; qc0 += QC) {
          if (js < SL)
#pragma unroll
            for (int a = 0; a < A2; ++a)
#pragma unroll
              for (int qq = 0; qq < QC; ++qq) sc[(lane * A2 + a) * QC + qq] = Ops::get(acc[a], qc0 + qq);
          __syncwarp();
          for (int e = lane; e < O * QC; e += 32) {
            const int row = e / QC, qq = e % QC;
            const int a = (int)(((float)row + 0.5f) * inv);  // row < 128, Og <= 32: exact
            const int l = row - a * Og;
            T v = sc[(l * A2 + a) * QC + qq];
            for (int k = 1; k < SL; ++k) v = v + sc[((k * Og + l) * A2 + a) * QC + qq];
            out[(size_t)row * RS + qc0 + qq] = v;
          }
          __syncwarp();
        }
      } else {
        for (int e = lane; e < O * R; e += 32) out[(size_t)(e / R) * RS + e % R] = zero<T>();
      }
      if constexpr (RS > R)
        for (int e = lane; e < O * (RS - R); e += 32) out[(size_t)(e / (RS - R)) * RS + R + e % (RS - R)] = zero<T>();
    } else {
#pragma unroll
      for (int a = 0; a < A2; ++a) {
        if (a * OL < O) {
          const int l = row0 + a * OL;
          T* row = out + (size_t)l * RS;
#pragma unroll
          for (int q = 0; q < R; ++q) {
            T v = Ops::get(acc[a], q);
            if constexpr (MODE == 1) v = v + shfl_xor(v, 16);
            // MODE 1: half-warp js writes half js of the right-hand sides
            const bool mine = MODE == 0 || (js == 0 ? q < (R + 1) / 2 : q >= (R + 1) / 2);
            if (l < O && mine) row[q] = v;
          }
          if (l < O && js == 0)
#pragma unroll
            for (int q = R; q < RS; ++q) row[q] = zero<T>();
        }
      }
    }
    if (task.nunits > 0 && (kLanes || lane == 0) && (u - 1) + kWarpStages < u_end) {
      // the scratch writes (generic proxy) are ordered before the copy that reuses the stage
      if (lane == 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      issue_next(u - 1 + kWarpStages);
    }
  }
}

// Warp-level streamed tasks on the tensor cores (FP32 'N' products).  Same per-warp TMA
// pipeline as warp_stream_kernel; the product of a unit is a sequence of warp MMAs
// (mma.sync m16n8k8, TF32 operands, FP32 accumulators) computing out^T = X^T P^T: the
// right-hand sides are the 16 rows of the MMA (A = X^T, one fragment per 8-column step for
// the whole task), the output rows its 8 columns (B = P^T, one fragment per 8-row tile), so an
// output of O rows takes ceil(O / 8) tiles.  FP32 accuracy is kept with the three-term split
// a = a_hi + a_lo (a_hi = a truncated to TF32): X P ~ X_lo P_hi + X_hi P_lo + X_hi P_hi, the
// lo x lo term (2^-20 relative at most) dropped, and every 8-column step goes to fresh
// fragments that are added to the running FP32 sums with round-to-nearest adds (the tensor
// core's own sums are not rounded to nearest).  Operands are read from the stage in fragment
// order (g = lane / 4, t = lane % 4): A holds X[k0 + t (+4)][g (+8)], B holds
// P[k0 + t (+4)][row 8 tile + g]; rows at or past O are computed and never written.  Only the
// last step of a unit whose width is not a multiple of 8 masks its columns (TAIL).
// a_hi = a with its low 13 mantissa bits cleared (a TF32 value), a_lo = a - a_hi (exact in
// FP32; the MMA reads its leading 11 bits).
__device__ __forceinline__ void tf32_split(float v, uint32_t& hi, uint32_t& lo) {
  hi = __float_as_uint(v) & 0xffffe000u;
  lo = __float_as_uint(v - __uint_as_float(hi));
}
// Not volatile: independent tiles' MMA chains may be interleaved by the scheduler.
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// One 8-column step k0 of a unit: the A fragment (X^T) once, then the NT 8-row tiles of the
// output (NT a compile-time count, so that the tiles' MMA chains are independent straight-line
// code the scheduler interleaves).  TAIL masks the columns at or past c (both operands: the
// stage past a short piece holds stale data).
template <int RS, int NT, int NTILE, bool TAIL>
__device__ __forceinline__ void mma_kstep(const float* P, const float* X, int k0, int c, int O, int g, int tg,
                                          float (&acc)[NTILE][4]) {
  const int ka = k0 + tg, kb = k0 + tg + 4;
  const bool va = !TAIL || ka < c, vb = !TAIL || kb < c;
  // right-hand sides g and g + 8 of the xz rows (RS columns; the rest are zeros)
  const bool q0 = g < RS, q1 = g + 8 < RS;
  uint32_t ah[4], al[4];
  tf32_split((va && q0) ? X[ka * RS + g] : 0.f, ah[0], al[0]);
  tf32_split((va && q1) ? X[ka * RS + g + 8] : 0.f, ah[1], al[1]);
  tf32_split((vb && q0) ? X[kb * RS + g] : 0.f, ah[2], al[2]);
  tf32_split((vb && q1) ? X[kb * RS + g + 8] : 0.f, ah[3], al[3]);
  const float* pa = P + ka * O + g;
  const float* pb = P + kb * O + g;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    uint32_t bh0, bl0, bh1, bl1;
    tf32_split(va ? pa[t * 8] : 0.f, bh0, bl0);
    tf32_split(vb ? pb[t * 8] : 0.f, bh1, bl1);
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    mma_tf32(d, al, bh0, bh1);
    mma_tf32(d, ah, bl0, bl1);
    mma_tf32(d, ah, bh0, bh1);
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[t][e] += d[e];
  }
}

// All steps of one unit with NT output tiles.
template <int RS, int NT, int NTILE>
__device__ __forceinline__ void mma_unit(const float* P, const float* X, int c, int O, int g, int tg,
                                         float (&acc)[NTILE][4]) {
  int k0 = 0;
  if constexpr (NT <= 4) {
    // two steps per iteration: their MMA chains are independent and overlap (wider tasks
    // have enough independent tiles in one step, and the registers go to their sums; with
    // two steps for 5-7 tiles the y-phase took 0.1213 -> 0.1235 ms, and with them for 4 tiles
    // the z-phase 0.1145 -> 0.111 ms, on the 100,000-point cylinder)
#pragma unroll 2
    for (; k0 + 8 <= c; k0 += 8) mma_kstep<RS, NT, NTILE, false>(P, X, k0, c, O, g, tg, acc);
  } else {
#pragma unroll 1
    for (; k0 + 8 <= c; k0 += 8) mma_kstep<RS, NT, NTILE, false>(P, X, k0, c, O, g, tg, acc);
  }
  if (k0 < c) mma_kstep<RS, NT, NTILE, true>(P, X, k0, c, O, g, tg, acc);
}
// The unit with the task's tile count (1 .. NTILE) as a compile-time constant.
template <typename T, int RS, int NTILE, int NT = 1>
__device__ __forceinline__ void mma_unit_dispatch(int ntn, const T* P, const T* X, int c, int O, int g, int tg,
                                                  T (&acc)[NTILE][4]) {
  if constexpr (NT < NTILE) {
    if (ntn == NT) {
      mma_unit<RS, NT, NTILE>(P, X, c, O, g, tg, acc);
      return;
    }
    mma_unit_dispatch<T, RS, NTILE, NT + 1>(ntn, P, X, c, O, g, tg, acc);
  } else {
    mma_unit<RS, NTILE, NTILE>(P, X, c, O, g, tg, acc);
  }
}

// CTAs an SM the tensor-core kernel is compiled for: four, the number its shared memory allows
// (two stages of warp_stage_bytes(4) for each of its four warps), so every tile count gets the
// registers of four CTAs.
constexpr int kMmaMinBlocks = 4;

template <typename T, int R, int RS, int NTILE>
__global__ void __launch_bounds__(kWarpCTA * 32, kMmaMinBlocks)
    mma_stream_kernel(const GemvTask* __restrict__ tasks, const int* __restrict__ warp_begin,
                      const GemvUnit* __restrict__ units, const T* __restrict__ arena, T* xz, GemvStatus* err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, tg = lane & 3;
  unsigned char* wbase = smem_raw + (size_t)warp * kWarpStages * warp_stage_bytes((int)sizeof(T));
  // per stage: the unit's column count and X offset (what the consumers read), then the barriers
  int2* uslot =
      reinterpret_cast<int2*>(smem_raw + (size_t)kWarpCTA * kWarpStages * warp_stage_bytes((int)sizeof(T))) + warp * kWarpStages;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + (size_t)kWarpCTA * kWarpStages *
                                                               (warp_stage_bytes((int)sizeof(T)) + sizeof(int2))) +
                   warp * kWarpStages;
  const int gw = blockIdx.x * kWarpCTA + warp;
  const int t0 = warp_begin[gw], t1 = warp_begin[gw + 1];
  if (t0 >= t1) return;
  const int u_begin = tasks[t0].first_unit;
  const int u_end = tasks[t1 - 1].first_unit + tasks[t1 - 1].nunits;
  const long long wlim = err->wait_limit;

  if (lane == 0) {
    for (int s = 0; s < kWarpStages; ++s) mbar_init(&bars[s], 1);
    mbar_fence_init();
  }
  __syncwarp();
  constexpr bool kLanes = NTILE <= 8;  // descriptors spread over the lanes (NextUnit)
  NextUnit<kLanes> nxt;
  int last_issued = u_begin - 1;  // lane 0: the last unit whose copies were issued
  auto issue = [&](int u, const GemvUnit& U) {
    const int s = (u - u_begin) % kWarpStages;
    last_issued = u;
    uslot[s] = make_int2(U.c, U.o0);
    const uint32_t pbytes = round16((uint64_t)U.pel * sizeof(T));
    const uint32_t xbytes = (uint32_t)U.c * RS * (uint32_t)sizeof(T);
    unsigned char* st = wbase + (size_t)s * warp_stage_bytes((int)sizeof(T));
    if (!unit_copies_ok<T, RS>(U, arena, xz, warp_stage_bytes((int)sizeof(T)), U.o0)) {
      record_bad_unit(err, u);
      mbar_arrive(&bars[s]);
      return;
    }
    mbar_expect_tx(&bars[s], pbytes + xbytes);
    bulk_piece(st, arena + U.poff, pbytes, &bars[s]);
    issue_x<T, RS>(st + U.o0, xz, U, &bars[s]);
  };
  auto issue_next = [&](int v) {  // nxt holds units[v]; kLanes: every lane calls it, else lane 0
    const GemvUnit U = nxt.get();
    if (lane == 0) issue(v, U);
    if (v + 1 < u_end) nxt.load(units, v + 1, lane);
  };
  if (lane == 0)
    for (int v = u_begin; v < u_end && v < u_begin + kWarpStages; ++v) issue(v, units[v]);
  if (u_begin + kWarpStages < u_end) nxt.load(units, u_begin + kWarpStages, lane);

  int u = u_begin;
  NextTask<kLanes> task_next;
  task_next.load(tasks, t0, lane);
  for (int t = t0; t < t1; ++t) {
    const GemvTask task = task_next.get();
    if (t + 1 < t1) task_next.load(tasks, t + 1, lane);
    const int O = task.O;
    const int ntn = (O + 7) >> 3;  // 8-row tiles holding rows of this task (warp-uniform)
    T acc[NTILE][4];
#pragma unroll
    for (int i = 0; i < NTILE; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][e] = zero<T>();

    for (int kk = 0; kk < task.nunits; ++kk, ++u) {
      const int s = (u - u_begin) % kWarpStages;
      const uint32_t parity = (uint32_t)(((u - u_begin) / kWarpStages) & 1);
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bars[s], parity, wlim))) {
        if (lane == 0) warp_give_up(err, bars, kWarpStages, u_begin, u, last_issued);
        return;
      }
      const int c = uslot[s].x;
      const T* P = reinterpret_cast<const T*>(wbase + (size_t)s * warp_stage_bytes((int)sizeof(T)));
      const T* X = reinterpret_cast<const T*>(wbase + (size_t)s * warp_stage_bytes((int)sizeof(T)) + uslot[s].y);
      mma_unit_dispatch<T, RS, NTILE>(ntn, P, X, c, O, g, tg, acc);
      __syncwarp();  // every lane is done with stage s
      if ((kLanes || lane == 0) && u + kWarpStages < u_end) issue_next(u + kWarpStages);
    }

    // ---- epilogue: accumulator (rhs g (+8), rows 8 i + 2 t (+1)); right-hand sides past R
    // hold exact zeros (their X columns were zeros), which pads the row to RS ----
    T* out = xz + (size_t)task.out_row * RS;
#pragma unroll
    for (int i = 0; i < NTILE; ++i) {
      if (i < ntn) {
        const int r0 = i * 8 + 2 * tg, r1 = r0 + 1;
        if (g < RS) {
          if (r0 < O) out[(size_t)r0 * RS + g] = acc[i][0];
          if (r1 < O) out[(size_t)r1 * RS + g] = acc[i][1];
        }
        if (g + 8 < RS) {
          if (r0 < O) out[(size_t)r0 * RS + g + 8] = acc[i][2];
          if (r1 < O) out[(size_t)r1 * RS + g + 8] = acc[i][3];
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------
// Transposed products ('T' / 'C'), every type: out[col] += sum_i op(P[i, col]) X[i] for
// column-major pieces P.  A warp holds CL x CP columns, lane = slice * CL + cl: column cl + CL a
// (a < CP) in its registers for all R right-hand sides, rows slice, slice + SL, ... of the piece.
// Each X row it loads serves CP columns, and each P scalar R multiply-adds (FP32, 16 right-hand
// sides: 32 paired FMAs per 4 scalars of P and 4 loads of X a lane); the slices are joined by a
// shuffle exchange that leaves each lane a share of the sums.  At 16 right-hand sides latency bounds
// it: 122 to 128 registers leave 13 warps an SM, issue slots half and the FMA pipe a quarter busy.
//
// Products that ran a CTA per task, with a block barrier per unit and one column a lane, took
// (device time, before -> now): cylinder of 50,001 points, FP32, 16 right-hand sides 753 -> 192 us
// (1.9 TB/s); of 60,000 points, FP64, 11 right-hand sides 1,948 -> 384 us (2.4 TB/s); 12 covariance
// matrices, FP32, one right-hand side 906 -> 159 us (3.9 TB/s); Helmholtz cylinder of 50,000
// points, complex FP32, four 1,794 -> 300 us (3.6 TB/s).  FP32 stays on CUDA cores: its sums are
// chains of a few FMAs a slice, more accurate than the split TF32 products of the 'N' kernels.

// acc[a] += sum over this lane's rows of P[i, cols[a]] X[i], a in [A0, A0 + NA).
template <typename T, int R, int CP, int A0, int NA, int SL>
__device__ __forceinline__ void trans_rows(const T* P, int O, int c, int cl, int CL, const T* X, int xs, int sl,
                                           bool conj, typename RowOps<T, R>::AV (&acc)[CP]) {
  using Ops = RowOps<T, R>;
  const T* p[NA];
#pragma unroll
  for (int a = 0; a < NA; ++a) p[a] = P + (size_t)min(cl + CL * a, c - 1) * O;  // past the piece: not written
#pragma unroll 2
  for (int i = sl; i < O; i += SL) {
    typename Ops::XV xv;
    Ops::load(X + (size_t)i * xs, xv);
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      T v = p[a][i];
      if constexpr (Traits<T>::is_complex) {
        if (conj) v = conjg(v);
      }
      Ops::fma(v, xv, acc[A0 + a]);
    }
  }
}
// The number of columns groups (na of CP from group a0) as a compile-time constant.
template <typename T, int R, int CP, int SL, int A0 = 0, int NA = 1>
__device__ __forceinline__ void trans_dispatch(int a0, int na, const T* P, int O, int c, int cl, int CL, const T* X,
                                               int xs, int sl, bool conj, typename RowOps<T, R>::AV (&acc)[CP]) {
  if (a0 == A0 && na == NA) {
    trans_rows<T, R, CP, A0, NA, SL>(P, O, c, cl, CL, X, xs, sl, conj, acc);
    return;
  }
  if constexpr (A0 + NA < CP) {
    trans_dispatch<T, R, CP, SL, A0, NA + 1>(a0, na, P, O, c, cl, CL, X, xs, sl, conj, acc);
  } else if constexpr (A0 + 1 < CP) {
    trans_dispatch<T, R, CP, SL, A0 + 1, 1>(a0, na, P, O, c, cl, CL, X, xs, sl, conj, acc);
  }
}

// Sums v over the lanes that differ in the slice bits (M = 16 down to CL), in exchanges that
// halve what each lane keeps: afterwards the lane holds the sums of values off .. off + (what is
// left) - 1; `mine` is false on lanes holding a copy of another lane's.
__host__ __device__ constexpr int trans_left(int V, int CL) {
  for (int m = 16; m >= CL; m >>= 1)
    if (V % 2 == 0) V /= 2;
  return V;
}
template <typename T, int CL, int N, int V, int M>
__device__ __forceinline__ void slice_sum(T (&v)[N], int lane, int& off, bool& mine) {
  if constexpr (M >= CL) {
    if constexpr (V % 2 == 0) {
      constexpr int H = V / 2;
      const bool hi = (lane & M) != 0;
#pragma unroll
      for (int i = 0; i < H; ++i) {
        const T send = hi ? v[i] : v[i + H];
        const T keep = hi ? v[i + H] : v[i];
        v[i] = keep + shfl_xor(send, M);
      }
      off += hi ? H : 0;
      slice_sum<T, CL, N, H, M / 2>(v, lane, off, mine);
    } else {
#pragma unroll
      for (int i = 0; i < V; ++i) v[i] = v[i] + shfl_xor(v[i], M);
      mine = mine && (lane & M) == 0;
      slice_sum<T, CL, N, V, M / 2>(v, lane, off, mine);
    }
  }
}
template <typename T, int Q>
__device__ inline void stg_vec(T* p, const T* v) {
  constexpr int bytes = Q * (int)sizeof(T);
  if constexpr (bytes % 16 == 0) {
#pragma unroll
    for (int c = 0; c < bytes / 16; ++c) reinterpret_cast<uint4*>(p)[c] = reinterpret_cast<const uint4*>(v)[c];
  } else {
#pragma unroll
    for (int c = 0; c < Q; ++c) p[c] = v[c];
  }
}

constexpr int kTransWarps = 4;
constexpr int kTransStages = 2;
__device__ inline GemvTransUnit load_unit(const GemvTransUnit* p) {
  const int4 w = __ldg(reinterpret_cast<const int4*>(p));
  GemvTransUnit u;
  memcpy(&u, &w, sizeof(u));
  return u;
}

// Row stride (scalars) of the x rows the column pass keeps in shared memory: padded by 16 bytes
// where the slices' rows would otherwise share banks.
template <typename T, int RS>
__host__ __device__ constexpr int trans_xstride() {
  return (RS * (int)sizeof(T)) % 64 == 0 ? RS + 16 / (int)sizeof(T) : RS;
}

// Column pass: a task is a part of an output block's matrix (O rows, the block's x rows at
// out_row), a unit up to 64 whole columns of it; column j of a unit is written to the xz row
// colmap[unit.xrow + j].  The four warps of a CTA share the block's x rows (staged once a task)
// and take its units in turn, each through its own two-stage ring.
template <typename T, int R, int RS>
__global__ void __launch_bounds__(kTransWarps * 32, (trans_ctas_per_sm((int)sizeof(T))))
    trans_columns_kernel(const GemvTask* __restrict__ tasks, const int* __restrict__ cta_begin,
                         const GemvTransUnit* __restrict__ units, const int* __restrict__ colmap,
                         const T* __restrict__ arena, T* xz, int conj, int stage_bytes, int xrows, GemvStatus* err) {
  using Ops = RowOps<T, R>;
  constexpr int CL = trans_column_lanes((int)sizeof(T), R), CW = trans_cols((int)sizeof(T)), CP = CW / CL, SL = 32 / CL;
  constexpr int XS = trans_xstride<T, RS>();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cl = lane % CL, sl = lane / CL;
  T* X = reinterpret_cast<T*>(smem_raw);
  unsigned char* wbase = smem_raw + (size_t)xrows * XS * sizeof(T) + (size_t)warp * kTransStages * stage_bytes;
  unsigned char* tail = smem_raw + (size_t)xrows * XS * sizeof(T) + (size_t)kTransWarps * kTransStages * stage_bytes;
  int2* uslot = reinterpret_cast<int2*>(tail) + warp * kTransStages;  // a unit's columns, offset of its map
  uint64_t* bars = reinterpret_cast<uint64_t*>(tail + kTransWarps * kTransStages * sizeof(int2)) + warp * kTransStages;
  const int t0 = cta_begin[blockIdx.x], t1 = cta_begin[blockIdx.x + 1];
  if (t0 >= t1) return;
  const int u_begin = tasks[t0].first_unit + warp;
  const int u_end = tasks[t1 - 1].first_unit + tasks[t1 - 1].nunits;
  const long long wlim = err->wait_limit;
  if (lane == 0) {
    for (int s = 0; s < kTransStages; ++s) mbar_init(&bars[s], 1);
    mbar_fence_init();
  }
  __syncwarp();
  GemvTransUnit nxt{};  // lane 0: the next unit to issue, loaded one issue ahead
  int issued = 0;       // lane 0: units issued so far (unit i of the warp is u_begin + i kTransWarps)
  auto issue = [&](const GemvTransUnit& U, int v) {
    const int s = issued % kTransStages;
    ++issued;
    const uint32_t pbytes = round16((uint64_t)U.rows * U.cols * sizeof(T)), mbytes = round16((uint64_t)U.cols * sizeof(int));
    unsigned char* st = wbase + (size_t)s * stage_bytes;
    if (U.cols == 0 || U.rows == 0 || pbytes + mbytes > (uint32_t)stage_bytes ||
        (reinterpret_cast<uintptr_t>(arena + U.poff) & 15) != 0 || (U.x & 3) != 0) {
      record_bad_unit(err, v);
      uslot[s] = make_int2(0, 0);
      mbar_arrive(&bars[s]);
      return;
    }
    uslot[s] = make_int2(U.cols, (int)pbytes);
    mbar_expect_tx(&bars[s], pbytes + mbytes);
    bulk_piece(st, arena + U.poff, pbytes, &bars[s]);
    bulk_piece(st + pbytes, colmap + U.x, mbytes, &bars[s]);
  };
  if (lane == 0)
    for (int k = 0, v = u_begin; k < kTransStages && v < u_end; ++k, v += kTransWarps) issue(load_unit(units + v), v);
  int vnext = u_begin + kTransStages * kTransWarps;  // the next unit to issue
  if (lane == 0 && vnext < u_end) nxt = load_unit(units + vnext);

  bool dead = false;  // a wait gave up: the warp only keeps the CTA's barriers company
  int u = u_begin, done = 0;
  for (int t = t0; t < t1; ++t) {
    const GemvTask task = tasks[t];
    const int O = task.O;
    __syncthreads();  // the previous task's x rows are read
    {
      constexpr int V = 16 / (int)sizeof(T);  // scalars a 16-byte chunk
      constexpr int RC = RS / V;              // chunks a row
      const uint4* src = reinterpret_cast<const uint4*>(xz + (size_t)task.out_row * RS);
      for (int e = tid; e < O * RC; e += kTransWarps * 32)
        *reinterpret_cast<uint4*>(X + (size_t)(e / RC) * XS + (size_t)(e % RC) * V) = src[e];
    }
    __syncthreads();
    const int task_end = task.first_unit + task.nunits;
    for (; u < task_end; u += kTransWarps, ++done) {
      if (dead) continue;
      const int s = done % kTransStages;
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bars[s], (uint32_t)((done / kTransStages) & 1), wlim))) {
        if (lane == 0) {
          atomicCAS(&err->failed, 0, 1);
          for (int v = done; v < issued; ++v)
            mbar_wait_bounded(&bars[v % kTransStages], (uint32_t)((v / kTransStages) & 1), drain_limit(err));
        }
        __syncwarp();
        dead = true;
        continue;
      }
      const int c = uslot[s].x;
      const T* P = reinterpret_cast<const T*>(wbase + (size_t)s * stage_bytes);
      const int* map = reinterpret_cast<const int*>(wbase + (size_t)s * stage_bytes + uslot[s].y);
      for (int c0 = 0; c0 < c; c0 += CW) {
        typename Ops::AV acc[CP];
#pragma unroll
        for (int a = 0; a < CP; ++a) Ops::zero_(acc[a]);
        const int left = c - c0;
        trans_dispatch<T, R, CP, SL>(0, min(CP, (left + CL - 1) / CL), P + (size_t)c0 * O, O, left, cl, CL, X, XS, sl,
                                     conj != 0, acc);
        constexpr int V = CP * R, VF = trans_left(V, CL);
        T v[V];
#pragma unroll
        for (int a = 0; a < CP; ++a)
#pragma unroll
          for (int q = 0; q < R; ++q) v[a * R + q] = Ops::get(acc[a], q);
        int off = 0;
        bool mine = true;
        slice_sum<T, CL, V, V, 16>(v, lane, off, mine);
        const int col = cl + CL * (off / R);
        if (mine && col < left) stg_vec<T, VF>(xz + (size_t)map[c0 + col] * RS + off % R, v);
      }
      __syncwarp();  // every lane is done with stage s
      if (vnext < u_end) {
        if (lane == 0) {
          issue(nxt, vnext);
          if (vnext + kTransWarps < u_end) nxt = load_unit(units + vnext + kTransWarps);
        }
        vnext += kTransWarps;
      }
    }
  }
}

// Group pass: a task is up to CL x CP columns (rows of y) of an output block, a unit the task's
// columns of one B^T group (all of them, or some of the CL-wide groups from column o0 of a tall
// one) with the group's z' rows; the warp keeps the task's sums in registers and writes them as
// partial rows.  The piece starts `shift` scalars after a 16-byte boundary.
template <typename T, int R, int RS>
__global__ void __launch_bounds__(kTransWarps * 32, (trans_ctas_per_sm((int)sizeof(T))))
    trans_groups_kernel(const GemvTask* __restrict__ tasks, const int* __restrict__ warp_begin,
                        const GemvTransUnit* __restrict__ units, const T* __restrict__ arena, T* xz, int conj,
                        int stage_bytes, GemvStatus* err) {
  using Ops = RowOps<T, R>;
  constexpr int CL = trans_lanes((int)sizeof(T)), CP = trans_cols((int)sizeof(T)) / CL, SL = 32 / CL;
  constexpr int kAlign = 16 / (int)sizeof(T);  // scalars of a 16-byte step
  extern __shared__ __align__(128) unsigned char smem_raw[];
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int cl = lane % CL, sl = lane / CL;
  unsigned char* wbase = smem_raw + (size_t)warp * kTransStages * stage_bytes;
  unsigned char* tail = smem_raw + (size_t)kTransWarps * kTransStages * stage_bytes;
  // a unit's rows, columns, first column group, and piece shift << 20 | X offset in 16-byte steps
  int4* uslot = reinterpret_cast<int4*>(tail) + warp * kTransStages;
  uint64_t* bars = reinterpret_cast<uint64_t*>(tail + kTransWarps * kTransStages * sizeof(int4)) + warp * kTransStages;
  const int gw = blockIdx.x * kTransWarps + warp;
  const int t0 = warp_begin[gw], t1 = warp_begin[gw + 1];
  if (t0 >= t1) return;
  const int u_begin = tasks[t0].first_unit;
  const int u_end = tasks[t1 - 1].first_unit + tasks[t1 - 1].nunits;
  const long long wlim = err->wait_limit;
  if (lane == 0) {
    for (int s = 0; s < kTransStages; ++s) mbar_init(&bars[s], 1);
    mbar_fence_init();
  }
  __syncwarp();
  GemvTransUnit nxt{};  // lane 0: the next unit to issue, loaded one issue ahead
  int last_issued = u_begin - 1;
  auto issue = [&](const GemvTransUnit& U, int v) {
    const int s = (v - u_begin) % kTransStages;
    last_issued = v;
    const int shift = (int)(U.poff % kAlign);  // the copy starts at the 16-byte boundary below
    const uint32_t pbytes = round16((uint64_t)(U.rows * U.cols + shift) * sizeof(T));
    const uint32_t xbytes = (uint32_t)U.rows * RS * (uint32_t)sizeof(T);
    unsigned char* st = wbase + (size_t)s * stage_bytes;
    const T* src = arena + (U.poff - shift);
    if (U.rows == 0 || U.cols == 0 || U.o0 % CL != 0 || U.o0 + U.cols > CL * CP ||
        pbytes + xbytes > (uint32_t)stage_bytes || (reinterpret_cast<uintptr_t>(src) & 15) != 0) {
      record_bad_unit(err, v);
      uslot[s] = make_int4(0, 1, 0, 0);
      mbar_arrive(&bars[s]);
      return;
    }
    uslot[s] = make_int4(U.rows, U.cols, U.o0 / CL, (shift << 20) | (int)(pbytes >> 4));
    mbar_expect_tx(&bars[s], pbytes + xbytes);
    bulk_piece(st, src, pbytes, &bars[s]);
    bulk_xrows(st + pbytes, xz + (size_t)U.x * RS, xbytes, &bars[s]);
  };
  if (lane == 0) {
    for (int v = u_begin; v < u_end && v < u_begin + kTransStages; ++v) issue(load_unit(units + v), v);
    if (u_begin + kTransStages < u_end) nxt = load_unit(units + u_begin + kTransStages);
  }

  int u = u_begin;
  for (int t = t0; t < t1; ++t) {
    const GemvTask task = tasks[t];
    typename Ops::AV acc[CP];
#pragma unroll
    for (int a = 0; a < CP; ++a) Ops::zero_(acc[a]);
    for (int kk = 0; kk < task.nunits; ++kk, ++u) {
      const int s = (u - u_begin) % kTransStages;
      const uint32_t parity = (uint32_t)(((u - u_begin) / kTransStages) & 1);
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bars[s], parity, wlim))) {
        if (lane == 0) warp_give_up(err, bars, kTransStages, u_begin, u, last_issued);
        return;
      }
      const int4 w = uslot[s];
      const T* P = reinterpret_cast<const T*>(wbase + (size_t)s * stage_bytes) + (w.w >> 20);
      const T* X = reinterpret_cast<const T*>(wbase + (size_t)s * stage_bytes + (size_t)((w.w & 0xfffff) << 4));
      trans_dispatch<T, R, CP, SL>(w.z, (w.y + CL - 1) / CL, P, w.x, w.y, cl, CL, X, RS, sl, conj != 0, acc);
      __syncwarp();  // every lane is done with stage s
      if (lane == 0 && u + kTransStages < u_end) {
        issue(nxt, u + kTransStages);
        if (u + kTransStages + 1 < u_end) nxt = load_unit(units + u + kTransStages + 1);
      }
    }
    constexpr int V = CP * R, VF = trans_left(V, CL);
    T v[V];
#pragma unroll
    for (int a = 0; a < CP; ++a)
#pragma unroll
      for (int q = 0; q < R; ++q) v[a * R + q] = Ops::get(acc[a], q);
    int off = 0;
    bool mine = true;
    slice_sum<T, CL, V, V, 16>(v, lane, off, mine);
    const int col = cl + CL * (off / R);
    if (mine && col < task.O) stg_vec<T, VF>(xz + (size_t)(task.out_row + col) * RS + off % R, v);
  }
}

// ---------------------------------------------------------------------------------
// FP32 'N' product on the 5th-generation tensor cores (tcgen05.mma, accumulators in tensor
// memory), one task at a time per CTA of 128 threads; thread t owns output row t.
//
// A unit out(O x 16) += P (O x c) X (c x 16), c <= kTcCols, is D = A B^T with A = P
// (M = 128, K = c) and B = X^T (N = 16, K = c): TF32 operands in shared memory, K-major
// without swizzle (8-row x 16-byte core matrices, 128 B between the two 4-column halves of a
// k-step, 256 B between 8-row groups).  FP32 accuracy as in the warp-level kernel: the split
// P X ~ P_lo X_hi + P_hi X_lo + P_hi X_hi, each 8-column step into its own accumulator
// (tensor-memory columns 16 s) and the steps added in order to the running sums in registers
// with FP32 round-to-nearest adds (the tensor core's own sums are not rounded to nearest).
// Thread 0 streams the pieces through a ring of kTcStages stages (cp.async.bulk + mbarrier),
// issues the MMAs and commits them to an mbarrier; all threads split the raw piece into the
// hi / lo tiles and read the accumulators back (tcgen05.ld, one 32-lane quarter per warp).
// Tile rows at or past O are not written: they hold what earlier units left and only reach
// output rows that are never stored.  Every wait is bounded and sets `err` when it gives up.
constexpr int kTcThreads = 128;
constexpr int kTcStages = 4;
constexpr int kTcSteps = kTcCols / 8;
constexpr int kTcTileA = 128 * 8 * 4;  // one k-step of A: 4 KB
constexpr int kTcTileB = 16 * 8 * 4;   // one k-step of B: 512 B
constexpr int kTcStage = kTcPieceBytes + kTcXBytes;
constexpr int kTcTmemCols = 16 * kTcSteps;  // a power of two >= 32
constexpr uint32_t kTcIdesc = (1u << 4)     // D: F32
                              | (2u << 7)   // A: TF32
                              | (2u << 10)  // B: TF32
                              | (2u << 17)  // N = 16
                              | (8u << 24); // M = 128

__device__ __forceinline__ uint32_t tc_kmaj(int r, int k) {
  return (uint32_t)((r >> 3) * 256 + (k >> 2) * 128 + (r & 7) * 16 + (k & 3) * 4);
}
__device__ __forceinline__ uint64_t tc_desc(const void* p) {
  const uint32_t a = smem_u32(p);
  return (uint64_t)((a >> 4) & 0x3fff) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) |
         ((uint64_t)1 << 46);
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(kTcIdesc), "r"(accumulate));
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&f)[16]) {
  uint32_t v[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
        "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]);
}
__device__ __forceinline__ float4 tc_hi(float4 v, float4& lo) {
  float4 h;
  h.x = __uint_as_float(__float_as_uint(v.x) & 0xffffe000u);
  h.y = __uint_as_float(__float_as_uint(v.y) & 0xffffe000u);
  h.z = __uint_as_float(__float_as_uint(v.z) & 0xffffe000u);
  h.w = __uint_as_float(__float_as_uint(v.w) & 0xffffe000u);
  lo = make_float4(v.x - h.x, v.y - h.y, v.z - h.z, v.w - h.w);
  return h;
}

template <int RS>
__global__ void __launch_bounds__(kTcThreads, 1)
    umma_stream_kernel(const GemvTask* __restrict__ tasks, const int* __restrict__ cta_begin,
                       const GemvUnit* __restrict__ units, const float* __restrict__ arena, float* xz, GemvStatus* err) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* ring = smem_raw;
  unsigned char* tAh = ring + kTcStages * kTcStage;
  unsigned char* tAl = tAh + kTcSteps * kTcTileA;
  unsigned char* tBh = tAl + kTcSteps * kTcTileA;
  unsigned char* tBl = tBh + kTcSteps * kTcTileB;
  uint64_t* full = reinterpret_cast<uint64_t*>(tBl + kTcSteps * kTcTileB);
  uint64_t* mmab = full + kTcStages;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mmab + 1);
  GemvUnit* uslot = reinterpret_cast<GemvUnit*>(tslot + 4);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int t0 = cta_begin[blockIdx.x], t1 = cta_begin[blockIdx.x + 1];
  if (t0 >= t1) return;
  const int u_begin = tasks[t0].first_unit;
  const int u_end = tasks[t1 - 1].first_unit + tasks[t1 - 1].nunits;
  const long long wlim = err->wait_limit;
  if (tid == 0) {
    for (int s = 0; s < kTcStages; ++s) mbar_init(&full[s], 1);
    mbar_init(mmab, 1);
    mbar_fence_init();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                 "r"(kTcTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tslot;
  const uint32_t tlane = tmem + ((uint32_t)(warp * 32) << 16);

  int last_issued = u_begin - 1;  // thread 0: the last unit whose copies were issued
  auto issue = [&](int v) {
    const GemvUnit U = units[v];
    const int s = (v - u_begin) % kTcStages;
    last_issued = v;
    uslot[s] = U;
    const uint32_t pbytes = round16((uint64_t)U.pel * sizeof(float));
    const uint32_t xbytes = (uint32_t)U.c * RS * (uint32_t)sizeof(float);
    unsigned char* st = ring + (size_t)s * kTcStage;
    mbar_expect_tx(&full[s], pbytes + xbytes);
    bulk_piece(st, arena + U.poff, pbytes, &full[s]);
    issue_x<float, RS>(st + kTcPieceBytes, xz, U, &full[s]);
  };
  if (tid == 0)
    for (int v = u_begin; v < u_end && v < u_begin + kTcStages; ++v) issue(v);

  uint32_t mma_parity = 0;
  int u = u_begin;
  // a wait that gives up stops the CTA (CTA-uniform): `pending` is the first unit whose
  // copies are not consumed, `mma_pending` whether a commit is not waited for
  bool failed = false, mma_pending = false;
  int pending = u_begin;
  for (int t = t0; t < t1 && !failed; ++t) {
    const GemvTask task = tasks[t];
    const int O = task.O;
    float acc[16];
#pragma unroll
    for (int n = 0; n < 16; ++n) acc[n] = 0.f;
    for (int kk = 0; kk < task.nunits; ++kk, ++u) {
      const int s = (u - u_begin) % kTcStages;
      if (__syncthreads_or(!mbar_wait_bounded(&full[s], (uint32_t)(((u - u_begin) / kTcStages) & 1), wlim))) {
        failed = true;
        pending = u;
        break;
      }
      const int c = uslot[s].c;
      const float* P = reinterpret_cast<const float*>(ring + (size_t)s * kTcStage);
      const float* X = reinterpret_cast<const float*>(ring + (size_t)s * kTcStage + kTcPieceBytes);
      // A tiles: (row i, 4-column quad q), rows < O, columns past c as zeros
      for (int it = tid; it < O * (kTcCols / 4); it += kTcThreads) {
        const int i = it % O, q = it / O, k0 = 4 * q;
        float4 v;
        v.x = k0 < c ? P[(size_t)k0 * O + i] : 0.f;
        v.y = k0 + 1 < c ? P[(size_t)(k0 + 1) * O + i] : 0.f;
        v.z = k0 + 2 < c ? P[(size_t)(k0 + 2) * O + i] : 0.f;
        v.w = k0 + 3 < c ? P[(size_t)(k0 + 3) * O + i] : 0.f;
        float4 lo;
        const float4 hi = tc_hi(v, lo);
        const uint32_t off = (uint32_t)(q >> 1) * kTcTileA + tc_kmaj(i, (q & 1) * 4);
        *reinterpret_cast<float4*>(tAh + off) = hi;
        *reinterpret_cast<float4*>(tAl + off) = lo;
      }
      // B tiles: (right-hand side n, quad q), exactly one item a thread
      {
        const int n = tid & 15, q = tid >> 4, k0 = 4 * q;
        float4 v;
        v.x = (n < RS && k0 < c) ? X[(size_t)k0 * RS + n] : 0.f;
        v.y = (n < RS && k0 + 1 < c) ? X[(size_t)(k0 + 1) * RS + n] : 0.f;
        v.z = (n < RS && k0 + 2 < c) ? X[(size_t)(k0 + 2) * RS + n] : 0.f;
        v.w = (n < RS && k0 + 3 < c) ? X[(size_t)(k0 + 3) * RS + n] : 0.f;
        float4 lo;
        const float4 hi = tc_hi(v, lo);
        const uint32_t off = (uint32_t)(q >> 1) * kTcTileB + tc_kmaj(n, (q & 1) * 4);
        *reinterpret_cast<float4*>(tBh + off) = hi;
        *reinterpret_cast<float4*>(tBl + off) = lo;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncthreads();  // tiles written, stage s read
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int nsteps = (c + 7) >> 3;
      if (tid == 0) {
        for (int st = 0; st < nsteps; ++st) {
          const uint64_t ah = tc_desc(tAh + st * kTcTileA), al = tc_desc(tAl + st * kTcTileA);
          const uint64_t bh = tc_desc(tBh + st * kTcTileB), bl = tc_desc(tBl + st * kTcTileB);
          const uint32_t d = tmem + 16 * st;
          tc_mma(d, al, bh, 0);
          tc_mma(d, ah, bl, 1);
          tc_mma(d, ah, bh, 1);
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(mmab))
                     : "memory");
        if (u + kTcStages < u_end) issue(u + kTcStages);
      }
      if (__syncthreads_or(!mbar_wait_bounded(mmab, mma_parity, wlim))) {
        failed = mma_pending = true;
        pending = u + 1;
        break;
      }
      mma_parity ^= 1u;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      for (int st = 0; st < nsteps; ++st) {
        float f[16];
        tc_ld16(tlane + 16 * st, f);
#pragma unroll
        for (int n = 0; n < 16; ++n) acc[n] = __fadd_rn(acc[n], f[n]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    if (failed) break;
    if (tid < O) {
      float* out = xz + (size_t)(task.out_row + tid) * RS;
      if constexpr (RS % 4 == 0) {
#pragma unroll
        for (int n = 0; n < RS; n += 4)
          *reinterpret_cast<float4*>(out + n) = make_float4(acc[n], acc[n + 1], acc[n + 2], acc[n + 3]);
      } else {
#pragma unroll
        for (int n = 0; n < RS; ++n) out[n] = acc[n];
      }
    }
  }
  if (failed && tid == 0) {
    // flag the product, then let the MMAs and copies in flight finish before the tensor
    // memory is freed and the CTA exits
    atomicExch(&err->failed, 1);
    if (mma_pending) mbar_wait_bounded(mmab, mma_parity, drain_limit(err));
    for (int v = pending; v <= last_issued; ++v)
      mbar_wait_bounded(&full[(v - u_begin) % kTcStages], (uint32_t)(((v - u_begin) / kTcStages) & 1),
                        drain_limit(err));
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcTmemCols));
}

template <int RS>
void launch_umma_t(const GemvLaunch& L, const GemvUnit* units, const float* arena, float* xz, GemvStatus* err,
                   cudaStream_t s) {
  auto kern = umma_stream_kernel<RS>;
  const size_t smem = (size_t)kTcStages * kTcStage + 2 * kTcSteps * (kTcTileA + kTcTileB) + (kTcStages + 1) * 8 +
                      16 + kTcStages * sizeof(GemvUnit);
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr = true;
  }
  kern<<<L.ncta, kTcThreads, smem, s>>>(L.tasks, L.cta_begin, units, arena, xz, err);
}

// y in client order from the partial rows of the 'N' y tasks:
// y[i, q0 + q] = alpha * sum_p xz[pos + p * O, q] + beta * y[i, q0 + q].  A CTA takes 128
// client rows: the partial rows are read along q (contiguous), transposed through shared
// memory, and y is written along i (contiguous in each column of y).
constexpr int kFinalRows = 128;
template <typename T, int R, int RS>
__global__ void __launch_bounds__(256) yfinal_kernel(const int2* __restrict__ rows, int n, const T* __restrict__ xz,
                                                     T* __restrict__ y, int ldy, int q0, int r, T alpha, T beta) {
  __shared__ T tile[R][kFinalRows + 1];
  __shared__ int2 rd[kFinalRows];
  pdl_wait();
  const int i0 = blockIdx.x * kFinalRows;
  // the rows' part descriptors first, so that the loads of the partial rows below do not wait
  // on them one by one
  for (int il = threadIdx.x; il < kFinalRows; il += blockDim.x) rd[il] = i0 + il < n ? rows[i0 + il] : int2{0, 0};
  __syncthreads();
#pragma unroll 4
  for (int e = threadIdx.x; e < kFinalRows * R; e += blockDim.x) {
    const int il = e / R, q = e % R;
    const int2 d = rd[il];
    const int O = d.y & 255, np = d.y >> 8;
    T v = zero<T>();
    for (int p = 0; p < np; ++p) v = v + xz[((size_t)d.x + (size_t)p * O) * RS + q];
    tile[q][il] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < kFinalRows * R; e += blockDim.x) {
    const int q = e / kFinalRows, il = e % kFinalRows, i = i0 + il;
    if (i < n && q0 + q < r) {
      T* yp = y + (size_t)i + (size_t)(q0 + q) * ldy;
      T outv = alpha * tile[q][il];
      if (!is_zero_val(beta)) outv = fmadd(beta, *yp, outv);
      *yp = outv;
    }
  }
}

// Sums partial slots: xz[final + l] = sum_p xz[part + p k + l].  A warp per sum (kZredWarps sums
// a CTA), lanes over 16-byte chunks of the k x RS slot (a row of RS scalars is a multiple of 16
// bytes), the parts added in part order; the first `nwide` sums take a CTA each, its warps an
// eighth of the parts, joined in warp order (long groups and leaves have hundreds of parts, and
// one warp's loads are a chain).  FP64 and complex z kernels that summed their chunks themselves,
// the last chunk's warp adding all parts, took 331 us for the 50,000-point Helmholtz cylinder
// (complex FP32, four right-hand sides; 280 us with this pass) and 35 us for the 8,000-point
// cylinder (FP64, one; 31 us), one product alone; products queued one after the other 22.3 -> 20.4 us
// for the small one and nothing beyond noise for the large one.
constexpr int kZredWarps = 8;
constexpr int kZredBatch = 8;  // parts loaded before they are added (loads in flight together)
template <typename T, int RS>
__device__ __forceinline__ void zred_parts(const T* part, int k, int c, int p0, int p1, T (&s)[sizeof(T) >= 16 ? 1 : 16 / sizeof(T)]) {
  constexpr int V = sizeof(T) >= 16 ? 1 : 16 / (int)sizeof(T);  // scalars a 16-byte chunk
#pragma unroll
  for (int e = 0; e < V; ++e) s[e] = zero<T>();
  for (int b = p0; b < p1; b += kZredBatch) {
    uint4 raw[kZredBatch];
#pragma unroll
    for (int i = 0; i < kZredBatch; ++i)
      if (b + i < p1) raw[i] = *reinterpret_cast<const uint4*>(part + ((size_t)(b + i) * k * RS + (size_t)c * V));
#pragma unroll
    for (int i = 0; i < kZredBatch; ++i)
      if (b + i < p1) {
        const T* v = reinterpret_cast<const T*>(&raw[i]);
#pragma unroll
        for (int e = 0; e < V; ++e) s[e] = s[e] + v[e];
      }
  }
}
// The sum so far, of the rounds before this one.
template <typename T, int V>
__device__ __forceinline__ void zred_add(const T* fin, T (&s)[V]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(fin);
  const T* v = reinterpret_cast<const T*>(&raw);
#pragma unroll
  for (int e = 0; e < V; ++e) s[e] = v[e] + s[e];
}
template <typename T, int RS>
__global__ void __launch_bounds__(kZredWarps * 32) zred_kernel(const GemvZred* __restrict__ zr, int n, int nwide, T* xz) {
  constexpr int V = sizeof(T) >= 16 ? 1 : 16 / (int)sizeof(T);
  static_assert((RS * sizeof(T)) % 16 == 0, "xz rows are 16-byte multiples");
  __shared__ uint4 s_part[kZredWarps][32];
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if ((int)blockIdx.x < nwide) {
    const GemvZred d = zr[blockIdx.x];
    const int nchunk = d.k * RS / V;
    const T* part = xz + (size_t)d.part_row * RS;
    T* fin = xz + (size_t)d.final_row * RS;
    const int p0 = (int)((long long)d.nparts * warp / kZredWarps), p1 = (int)((long long)d.nparts * (warp + 1) / kZredWarps);
    for (int c0 = 0; c0 < nchunk; c0 += 32) {
      const int c = c0 + lane;
      T s[V];
      if (c < nchunk) {
        zred_parts<T, RS>(part, d.k, c, p0, p1, s);
        s_part[warp][lane] = *reinterpret_cast<const uint4*>(s);
      }
      __syncthreads();
      if (warp == 0 && c < nchunk) {
        for (int w = 1; w < kZredWarps; ++w) {
          const uint4 raw = s_part[w][lane];
          const T* v = reinterpret_cast<const T*>(&raw);
#pragma unroll
          for (int e = 0; e < V; ++e) s[e] = s[e] + v[e];
        }
        if (d.add) zred_add<T, V>(fin + (size_t)c * V, s);
        *reinterpret_cast<uint4*>(fin + (size_t)c * V) = *reinterpret_cast<const uint4*>(s);
      }
      __syncthreads();
    }
    return;
  }
  const int w = nwide + ((int)blockIdx.x - nwide) * kZredWarps + warp;
  if (w >= n) return;
  const GemvZred d = zr[w];
  const int nchunk = d.k * RS / V;
  const T* part = xz + (size_t)d.part_row * RS;
  T* fin = xz + (size_t)d.final_row * RS;
  for (int c = lane; c < nchunk; c += 32) {
    T s[V];
    zred_parts<T, RS>(part, d.k, c, 0, d.nparts, s);
    if (d.add) zred_add<T, V>(fin + (size_t)c * V, s);
    *reinterpret_cast<uint4*>(fin + (size_t)c * V) = *reinterpret_cast<const uint4*>(s);
  }
}
inline unsigned zred_grid(int n, int nwide) { return (unsigned)(nwide + (n - nwide + kZredWarps - 1) / kZredWarps); }

// A launch with programmatic stream serialization (see pdl_wait): the kernel must begin with
// pdl_wait() before it reads what the kernel before it wrote.
template <typename... KArgs, typename... Args>
void launch_pdl(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, args...);  // errors surface through cudaGetLastError, as for <<<>>>
}

// ---------------------------------------------------------------------------------
template <typename T, int R, int RS, int MODE, int A2>
void launch_warp_t(const GemvLaunch& L, const GemvUnit* units, const T* arena, T* xz, GemvStatus* err, cudaStream_t s) {
  auto kern = warp_stream_kernel<T, R, RS, MODE, A2>;
  const size_t smem = warp_stream_smem_bytes((int)sizeof(T));
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr = true;
  }
  launch_pdl(kern, dim3(L.ncta), dim3(kWarpCTA * 32), smem, s, L.tasks, L.cta_begin, units, arena, xz, err);
}

template <typename T, int R, int RS, int NTILE>
void launch_mma_t(const GemvLaunch& L, const GemvUnit* units, const T* arena, T* xz, GemvStatus* err,
                  cudaStream_t s) {
  auto kern = mma_stream_kernel<T, R, RS, NTILE>;
  const size_t smem = warp_stream_smem_bytes((int)sizeof(T));
  static bool attr = false;
  if (!attr) {
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    attr = true;
  }
  launch_pdl(kern, dim3(L.ncta), dim3(kWarpCTA * 32), smem, s, L.tasks, L.cta_begin, units, arena, xz, err);
}

// The 'N' launches.
template <typename T, int R, int RS>
void launch_stream(const GemvLaunch& L, const GemvUnit* units, const T* arena, T* xz, GemvStatus* err, cudaStream_t s) {
  if (L.ntasks <= 0) return;
  if constexpr (std::is_same<T, float>::value) {
    if (L.map == 4) {
      launch_umma_t<RS>(L, units, arena, xz, err, s);
      return;
    }
    // One right-hand side: CUDA cores, since the tensor-core tiles compute 16 rows of which one is
    // wanted and the splitting is paid all the same (12 covariance matrices, 610 MB: 170 -> 141 us,
    // 3.6 -> 4.3 TB/s; 20,000-point cube 124 -> 103 us), with half the error (FP32 against FP64 on
    // the same leaves 3.1e-7 -> 1.6e-7).  At four the tiles are still faster (95 against 101 us).
    if constexpr (R == 1) {
      if (L.rpt <= 4)
        launch_warp_t<T, R, RS, 2, 2>(L, units, arena, xz, err, s);
      else if (L.rpt <= 8)
        launch_warp_t<T, R, RS, 0, 2>(L, units, arena, xz, err, s);
      else
        launch_warp_t<T, R, RS, 0, 4>(L, units, arena, xz, err, s);
      return;
    }
    switch (L.rpt) {  // map 3: rpt = 8-row tiles of the launch's tallest task (exact up to 8)
      case 1: launch_mma_t<T, R, RS, 1>(L, units, arena, xz, err, s); break;
      case 2: launch_mma_t<T, R, RS, 2>(L, units, arena, xz, err, s); break;
      case 3: launch_mma_t<T, R, RS, 3>(L, units, arena, xz, err, s); break;
      case 4: launch_mma_t<T, R, RS, 4>(L, units, arena, xz, err, s); break;
      case 5: launch_mma_t<T, R, RS, 5>(L, units, arena, xz, err, s); break;
      case 6: launch_mma_t<T, R, RS, 6>(L, units, arena, xz, err, s); break;
      case 7: launch_mma_t<T, R, RS, 7>(L, units, arena, xz, err, s); break;
      case 8: launch_mma_t<T, R, RS, 8>(L, units, arena, xz, err, s); break;
      default: launch_mma_t<T, R, RS, 16>(L, units, arena, xz, err, s); break;
    }
  } else {
    if (L.map == 2)
      launch_warp_t<T, R, RS, 2, 2>(L, units, arena, xz, err, s);
    else if (L.map == 5)
      launch_warp_t<T, R, RS, 0, 2>(L, units, arena, xz, err, s);
    else if (L.map == 1)
      launch_warp_t<T, R, RS, 1, 4>(L, units, arena, xz, err, s);
    else
      launch_warp_t<T, R, RS, 0, 4>(L, units, arena, xz, err, s);
  }
}

template <typename F>
void allow_smem(F kern, bool& done) {
  if (done) return;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxCtaSmem);
  done = true;
}

template <typename T, int RS>
void launch_zred(const GemvZred* zred, int n, int nwide, T* xz, cudaStream_t s) {
  if (n > 0)
    launch_pdl(zred_kernel<T, RS>, dim3(zred_grid(n, nwide)), dim3(kZredWarps * 32), 0, s, zred, n, nwide, xz);
}

// The column pass of the transposed products and its sums, round by round: afterwards xz holds the
// z' rows of every Rk leaf and the full leaves' partial rows of y.
template <typename T, int R, int RS>
void run_trans_columns(const GemvSide& side, const T* arena, T* xz, int conj, GemvStatus* err, cudaStream_t s) {
  for (const GemvTransRound& round : side.rounds) {
    const GemvLaunch& L = round.columns;
    if (L.ntasks > 0) {
      auto kern = trans_columns_kernel<T, R, RS>;
      static bool attr = false;
      allow_smem(kern, attr);
      launch_pdl(kern, dim3(L.ncta), dim3(kTransWarps * 32),
                 trans_columns_smem(L.piece_bytes, L.xrows, trans_xstride<T, RS>() * (int)sizeof(T)), s, L.tasks,
                 L.cta_begin, side.tunits, side.colmap, arena, xz, conj, L.piece_bytes, L.xrows, err);
    }
    launch_zred<T, RS>(side.zred + round.zred0, round.nzred, round.nzwide, xz, s);
  }
}

template <typename T, int R, int RS>
void run_trans_groups(const GemvSide& side, const T* arena, T* xz, int conj, GemvStatus* err, cudaStream_t s) {
  for (int c = 0; c < side.ng; ++c) {
    const GemvLaunch& L = side.g[c];
    if (L.ntasks <= 0) continue;
    auto kern = trans_groups_kernel<T, R, RS>;
    static bool attr = false;
    allow_smem(kern, attr);
    launch_pdl(kern, dim3(L.ncta), dim3(kTransWarps * 32),
               trans_groups_smem(L.piece_bytes, L.xrows, RS * (int)sizeof(T)), s, L.tasks, L.cta_begin, side.tunits,
               arena, xz, conj, L.piece_bytes + L.xrows * RS * (int)sizeof(T), err);
  }
}

template <typename T, int R, bool TRANSP>
void run_tile(const GemvPlan& p, int nrhs, int q0, T alpha, T beta, const T* x, T* y, T* xz, int conj, GemvStatus* err,
              cudaStream_t s, const GemvTiming* tm) {
  constexpr int RS = rs_of<T>(R);
  const GemvSide& side = p.side[TRANSP ? 1 : 0];
  const int n_in = TRANSP ? p.n_rows : p.n_cols;
  const int* iperm_in = TRANSP ? p.iperm_rows : p.iperm_cols;
  const int ld_in = n_in, ld_out = TRANSP ? p.n_cols : p.n_rows;
  const T* arena = (const T*)p.arena;
  if (tm) cudaEventRecord(tm->ev[0], s);
  gather_kernel<T, R, RS><<<gather_grid(n_in), 256, 0, s>>>(x, n_in, ld_in, q0, nrhs, iperm_in, xz, p.n_in_max);
  if (tm) cudaEventRecord(tm->ev[1], s);
  if constexpr (TRANSP) {
    run_trans_columns<T, R, RS>(side, arena, xz, conj, err, s);
  } else {
    for (int c = 0; c < side.nz; ++c)
      launch_stream<T, R, RS>(side.z[c], side.units, arena, xz, err, s);
    launch_zred<T, RS>(side.zred, side.nzred, side.nzwide, xz, s);
  }
  if (tm) cudaEventRecord(tm->ev[2], s);
  if constexpr (TRANSP)
    run_trans_groups<T, R, RS>(side, arena, xz, conj, err, s);
  else
    launch_stream<T, R, RS>(side.y, side.units, arena, xz, err, s);
  if (side.nyrows > 0) {
    const unsigned nb = (unsigned)((side.nyrows + kFinalRows - 1) / kFinalRows);
    launch_pdl(yfinal_kernel<T, R, RS>, dim3(nb), dim3(256), 0, s, side.yrows, side.nyrows, xz, y, ld_out, q0, nrhs,
               alpha, beta);
  }
  if (tm) cudaEventRecord(tm->ev[3], s);
}

// Right-hand sides are taken in tiles of 16, 12, 8, 4 or 1 (complex double 4 or 1: its
// accumulators).
template <typename T, bool TRANSP>
void run_all(const GemvPlan& p, int nrhs, T alpha, T beta, const T* x, T* y, T* xz, int conj, GemvStatus* err,
             cudaStream_t s, const GemvTiming* tm) {
  constexpr int maxR = sizeof(T) >= 16 ? 4 : 16;
  int tile;
  for (int q0 = 0; q0 < nrhs; q0 += tile) {
    const int rem = nrhs - q0;
    tile = 1;
    // 9 to 12: a tile of 12 where the work grows with the tile's width (not the FP32 'N' products,
    // whose tensor-core tiles hold 16 anyway): 60,000-point cylinder, FP64, 11 right-hand sides
    // 387 -> 292 us
    constexpr bool has12 = sizeof(T) == 8 || (sizeof(T) == 4 && TRANSP);
    if (has12 && rem > 8 && rem <= 12) {
      tile = 12;
      run_tile<T, (has12 ? 12 : 4), TRANSP>(p, nrhs, q0, alpha, beta, x, y, xz, conj, err, s, tm);
    } else if (maxR == 16 && rem > 8) {
      tile = 16;
      run_tile<T, (maxR >= 16 ? 16 : 4), TRANSP>(p, nrhs, q0, alpha, beta, x, y, xz, conj, err, s, tm);
    } else if (maxR == 16 && rem > 4) {
      tile = 8;
      run_tile<T, (maxR >= 16 ? 8 : 4), TRANSP>(p, nrhs, q0, alpha, beta, x, y, xz, conj, err, s, tm);
    } else if (rem > 1) {
      tile = 4;
      run_tile<T, 4, TRANSP>(p, nrhs, q0, alpha, beta, x, y, xz, conj, err, s, tm);
    } else {
      run_tile<T, 1, TRANSP>(p, nrhs, q0, alpha, beta, x, y, xz, conj, err, s, tm);
    }
  }
}

// ---------------------------------------------------------------------------------
// Leaf-factor gradients (adjoint of y = H x with respect to the stored leaves), written in
// the canonical layout (full: m x n, Rk: A m x k then B n x k, column-major).
// R is the right-hand-side tile (compile time): columns past the caller's count hold exact
// zeros in xs and rs (the gather pads them), so they add nothing.
//
// An outer product out(m x n) = sum_q a[., q] b[., q]^T per full leaf, and two per Rk leaf (dA, dB),
// each taken by one warp on its own: a lane holds two rows of `a` in registers and walks the
// columns, whose row of `b` all lanes load alike, so that an entry costs R multiply-adds and its
// store and no warp waits for another.  Bound by the stores: on the 20,000-point cube (402 MB of
// FP32 gradients, one right-hand side) the adjoint call takes 314 us with it, 422 us with a CTA per
// leaf and a warp per column, 396 us with a CTA per product and its columns staged in shared
// memory (two block barriers for 6 KB of output); 30,000-point cylinder, 16 right-hand sides, the
// leaf gradients alone 1,822 -> 239 us.  Entries that are written and not added to are stored with
// an evict-first hint: the gradients are not read again here, and the vector rows and leaves of the
// passes around them stay in L2 (cube: adjoint 311 -> 296 us; 50,000-point cylinder, FP64, 309 -> 296
// us; 16 right-hand sides 281 us either way).
__device__ __forceinline__ void store_stream(float* p, float v) { __stcs(p, v); }
__device__ __forceinline__ void store_stream(double* p, double v) { __stcs(p, v); }
template <typename T>
__device__ __forceinline__ void store_stream(T* p, T v) { *p = v; }
constexpr int kGradWarps = 8;
constexpr int kGradRows = 2;  // rows a lane
template <typename T, int RS, int R, bool ACC>
__device__ __forceinline__ void grad_outer(const T* __restrict__ a, int m, const T* __restrict__ b, int n, T* out,
                                           int lane) {
  for (int i0 = 0; i0 < m; i0 += 32 * kGradRows) {
    T av[kGradRows][R];
    bool in[kGradRows];
#pragma unroll
    for (int h = 0; h < kGradRows; ++h) {
      const int i = i0 + 32 * h + lane;
      in[h] = i < m;
      lds_vec<T, R>(a + (size_t)(in[h] ? i : 0) * RS, av[h]);
    }
    T* o = out + i0 + lane;
#pragma unroll 4
    for (int j = 0; j < n; ++j) {
      T bv[R];
      lds_vec<T, R>(b + (size_t)j * RS, bv);
#pragma unroll
      for (int h = 0; h < kGradRows; ++h) {
        if (!in[h]) continue;
        T* e = o + (size_t)j * m + 32 * h;
        T acc = ACC ? *e : zero<T>();
#pragma unroll
        for (int q = 0; q < R; ++q) acc = fmadd(av[h][q], bv[q], acc);
        if (ACC)
          *e = acc;
        else
          store_stream(e, acc);
      }
    }
  }
}

// Items: the full leaves, then dA and dB of every Rk leaf.
template <typename T, int RS, int R, bool ACC>
__global__ void __launch_bounds__(kGradWarps * 32) grad_kernel(const GemvFullLeaf* __restrict__ full, int nfull,
                                                               const GemvRkLeaf* __restrict__ rk, int nrk,
                                                               const T* __restrict__ xs, const T* __restrict__ rs,
                                                               T* gfull, T* grk) {
  const int lane = threadIdx.x & 31;
  for (int it = blockIdx.x * kGradWarps + (threadIdx.x >> 5); it < nfull + 2 * nrk; it += gridDim.x * kGradWarps) {
    if (it < nfull) {  // dF = r x^T
      const GemvFullLeaf F = full[it];
      if (gfull)
        grad_outer<T, RS, R, ACC>(rs + (size_t)F.row_off * RS, F.m, xs + (size_t)F.col_off * RS, F.n, gfull + F.goff,
                                  lane);
      continue;
    }
    if (!grk) continue;
    const GemvRkLeaf L = rk[(it - nfull) >> 1];
    T* dA = grk + L.goff;
    if (((it - nfull) & 1) == 0)  // dA = r z^T,  z = B^T x  (rows zrow_n of the x buffer)
      grad_outer<T, RS, R, ACC>(rs + (size_t)L.row_off * RS, L.m, xs + (size_t)L.zrow_n * RS, L.k, dA, lane);
    else  // dB = x w^T,  w = A^T r  (rows zrow_t of the r buffer)
      grad_outer<T, RS, R, ACC>(xs + (size_t)L.col_off * RS, L.n, rs + (size_t)L.zrow_t * RS, L.k,
                                dA + (size_t)L.m * L.k, lane);
  }
}

// x in cluster order (columns) and z = B^T x, in xz.
template <typename T, int R>
void forward_z(const GemvPlan& p, int nrhs, const T* x, T* xz, GemvStatus* err, cudaStream_t s) {
  constexpr int RS = rs_of<T>(R);
  const GemvSide& sn = p.side[0];
  gather_kernel<T, R, RS><<<gather_grid(p.n_cols), 256, 0, s>>>(x, p.n_cols, p.n_cols, 0, nrhs, p.iperm_cols, xz,
                                                                p.n_in_max);
  for (int c = 0; c < sn.nz; ++c)
    launch_stream<T, R, RS>(sn.z[c], sn.units, (const T*)p.arena, xz, err, s);
  launch_zred<T, RS>(sn.zred, sn.nzred, sn.nzwide, xz, s);
}
template <typename T, int R>
void grads_outer(const GemvPlan& p, const T* xz, const T* rz, T* gfull, T* grk, bool accumulate, cudaStream_t s) {
  constexpr int RS = rs_of<T>(R);
  const int items = p.nfull + 2 * p.nrk, need = (items + kGradWarps - 1) / kGradWarps;
  if (items <= 0) return;
  const auto kern = accumulate ? grad_kernel<T, RS, R, true> : grad_kernel<T, RS, R, false>;
  const int grid = std::min(need, persistent_grid(8));
  kern<<<grid, kGradWarps * 32, 0, s>>>(p.full, p.nfull, p.rk, p.nrk, xz, rz, gfull, grk);
}

template <typename T, int R>
void grads_tile(const GemvPlan& p, int nrhs, const T* x, const T* r, T* xz, T* rz, T* gfull, T* grk, bool accumulate,
                GemvStatus* err, cudaStream_t s) {
  constexpr int RS = rs_of<T>(R);
  forward_z<T, R>(p, nrhs, x, xz, err, s);
  // r in cluster order (rows) and w = A^T r
  gather_kernel<T, R, RS><<<gather_grid(p.n_rows), 256, 0, s>>>(r, p.n_rows, p.n_rows, 0, nrhs, p.iperm_rows, rz,
                                                                p.n_in_max);
  run_trans_columns<T, R, RS>(p.side[1], (const T*)p.arena, rz, 0, err, s);
  grads_outer<T, R>(p, xz, rz, gfull, grk, accumulate, s);
}

// The adjoint of y = H x at the output gradient r in one pass: dx = H^T r (the 'T' product,
// whose z' = A^T r stays in rz) and the leaf gradients, which reuse that z' as w; z = B^T x is
// formed once in xz.
template <typename T, int R>
void adjoint_tile(const GemvPlan& p, int nrhs, const T* x, const T* r, T* dx, T* xz, T* rz, T* gfull, T* grk,
                  bool accumulate, GemvStatus* err, cudaStream_t s) {
  run_tile<T, R, true>(p, nrhs, 0, one<T>(), zero<T>(), r, dx, rz, 0, err, s, nullptr);
  forward_z<T, R>(p, nrhs, x, xz, err, s);
  grads_outer<T, R>(p, xz, rz, gfull, grk, accumulate, s);
}

}  // namespace

size_t trans_columns_smem(int stage_bytes, int xrows, int xrow_bytes) {
  return (size_t)xrows * xrow_bytes + (size_t)kTransWarps * kTransStages * (stage_bytes + sizeof(int2) + sizeof(uint64_t));
}
size_t trans_groups_smem(int piece_bytes, int xrows, int xrow_bytes) {
  return (size_t)kTransWarps * kTransStages *
         ((size_t)piece_bytes + (size_t)xrows * xrow_bytes + sizeof(int4) + sizeof(uint64_t));
}
int trans_warps_per_cta() { return kTransWarps; }

int gemv_rhs_stride(int elem_bytes, int R) { return R * elem_bytes >= 16 ? R : 16 / elem_bytes; }

size_t warp_stream_smem_bytes(int elem_bytes) {
  return (size_t)kWarpCTA * kWarpStages * (warp_stage_bytes(elem_bytes) + sizeof(int2) + sizeof(uint64_t));
}
int warp_stream_warps_per_cta() { return kWarpCTA; }
int mma_stream_blocks_per_sm() { return kMmaMinBlocks; }

size_t umma_smem_bytes() {
  return (size_t)kTcStages * kTcStage + 2 * kTcSteps * (kTcTileA + kTcTileB) + (kTcStages + 1) * 8 + 16 +
         kTcStages * sizeof(GemvUnit);
}

int gemv_launch_count(const GemvPlan& p, char trans, int nrhs, int elem_bytes) {
  const GemvSide& side = p.side[(trans == 'N' || trans == 'n') ? 0 : 1];
  int per_tile = 1;  // gather
  for (int c = 0; c < side.nz; ++c) per_tile += side.z[c].ntasks > 0;
  per_tile += side.nzred > 0;
  for (const GemvTransRound& r : side.rounds) per_tile += (r.columns.ntasks > 0) + (r.nzred > 0);
  per_tile += side.y.ntasks > 0;
  for (int c = 0; c < side.ng; ++c) per_tile += side.g[c].ntasks > 0;
  per_tile += side.nyrows > 0;  // final pass
  const int maxR = elem_bytes >= 16 ? 4 : 16;
  return per_tile * ((nrhs + maxR - 1) / maxR);
}

template <typename T>
void launch_leaf_gradients(const GemvPlan& p, int nrhs, const T* x, const T* r, T* xz, T* rz, T* gfull, T* grk,
                           bool accumulate, GemvStatus* err, cudaStream_t s) {
  constexpr bool big = sizeof(T) < 16;
  if (big && nrhs > 8) grads_tile<T, big ? 16 : 4>(p, nrhs, x, r, xz, rz, gfull, grk, accumulate, err, s);
  else if (big && nrhs > 4) grads_tile<T, big ? 8 : 4>(p, nrhs, x, r, xz, rz, gfull, grk, accumulate, err, s);
  else if (nrhs > 1) grads_tile<T, 4>(p, nrhs, x, r, xz, rz, gfull, grk, accumulate, err, s);
  else grads_tile<T, 1>(p, nrhs, x, r, xz, rz, gfull, grk, accumulate, err, s);
}

template <typename T>
void launch_gemv_adjoint(const GemvPlan& p, int nrhs, const T* x, const T* r, T* dx, T* xz, T* rz, T* gfull, T* grk,
                         bool accumulate, GemvStatus* err, cudaStream_t s) {
  constexpr bool big = sizeof(T) < 16;
  if (big && nrhs > 8) adjoint_tile<T, big ? 16 : 4>(p, nrhs, x, r, dx, xz, rz, gfull, grk, accumulate, err, s);
  else if (big && nrhs > 4) adjoint_tile<T, big ? 8 : 4>(p, nrhs, x, r, dx, xz, rz, gfull, grk, accumulate, err, s);
  else if (nrhs > 1) adjoint_tile<T, 4>(p, nrhs, x, r, dx, xz, rz, gfull, grk, accumulate, err, s);
  else adjoint_tile<T, 1>(p, nrhs, x, r, dx, xz, rz, gfull, grk, accumulate, err, s);
}

template <typename T>
void launch_gemv(const GemvPlan& p, char trans, int nrhs, T alpha, T beta, const T* x_client, T* y_client, T* xz,
                 GemvStatus* err, cudaStream_t s, const GemvTiming* tm) {
  if (trans == 'N') run_all<T, false>(p, nrhs, alpha, beta, x_client, y_client, xz, 0, err, s, tm);
  else
    run_all<T, true>(p, nrhs, alpha, beta, x_client, y_client, xz, (trans == 'C' && Traits<T>::is_complex) ? 1 : 0,
                     err, s, tm);
}

#define HB_INST(T)                                                                                            \
  template void launch_gemv<T>(const GemvPlan&, char, int, T, T, const T*, T*, T*, GemvStatus*, cudaStream_t,         \
                               const GemvTiming*);                                                             \
  template void launch_leaf_gradients<T>(const GemvPlan&, int, const T*, const T*, T*, T*, T*, T*, bool, GemvStatus*, \
                                         cudaStream_t);                                                                  \
  template void launch_gemv_adjoint<T>(const GemvPlan&, int, const T*, const T*, T*, T*, T*, T*, T*, bool, GemvStatus*, \
                                       cudaStream_t);
HB_INST(float)
HB_INST(double)
HB_INST(cfloat)
HB_INST(cdouble)
#undef HB_INST

}  // namespace hmatb200
