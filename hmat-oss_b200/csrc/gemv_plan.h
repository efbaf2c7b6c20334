// Device-resident schedule of the batched H-matrix-vector product (built on the host by
// the engine from the leaf list, consumed by gemv.cu).
//
// The leaf arena has two regions (layout in engine.cu): per output block (a leaf of the output
// cluster tree, cut into pieces of at most 128 rows) one column-major matrix holding the block's
// rows of every full leaf F and of every Rk leaf's A over those rows; then the B^T of the Rk
// leaves, those of one column range stacked into column-major groups.
//
// A product is a list of tasks; a task is one output ('N': an output block of y or the z = B^T x
// slots of a group; 'T': the columns of an output block, or a strip of columns of a column block)
// accumulated from a list of units, each one contiguous piece P of the arena times rows X of the
// xz buffer (x in cluster order, row-major, followed by the z rows).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

namespace hmatb200 {

// X rows of a unit come from at most kUnitRuns runs of consecutive xz rows (the columns of a
// block's matrix belong to several leaves, whose x or z rows are not adjacent).
constexpr int kUnitRuns = 4;

struct GemvUnit {
  long long poff;  // element offset of the piece P in the arena (16-byte aligned)
  int xrow;        // first row of the X piece in the xz buffer (nruns == 0)
  int c;           // inner extent (rows of X)
  int o0, ow;      // o0 = byte offset of the X rows in a warp-level pipeline stage (the piece's
                   // capacity; the FP32 tensor-core kernel reads it per unit); ow = output rows
  int pel;         // elements of the piece P (O x c)
  int shift;       // elements between the 16-byte aligned copy start and the piece (0)
  int nruns;       // 0: X rows xrow .. xrow + c - 1; else X rows from the runs below, in order
  int run_row[kUnitRuns];
  unsigned short run_len[kUnitRuns];
};

// A unit of a transposed product, 16 bytes (one load): a column-major piece of `rows` x `cols`
// from element poff, `cols` of its columns from column o0 of the task (group pass; 0 in the column
// pass).  x: the first xz row of its X rows (group pass), or its first entry of the column map.
struct GemvTransUnit {
  long long poff;
  int x;
  unsigned char rows, cols, o0, pad;
};
static_assert(sizeof(GemvTransUnit) == 16, "one 16-byte load");

struct GemvTask {
  int O;           // output rows
  int first_unit;  // units [first_unit, first_unit + nunits) in order
  int nunits;
  int out_row;     // first xz row of the output slot; column pass: first xz row of the x rows
};

// One launch: tasks of one shape class; each CTA (column pass) or warp of a persistent grid takes
// a contiguous range [cta_begin[b], cta_begin[b + 1]) of tasks.
struct GemvLaunch {
  int ntasks = 0;
  int ncta = 0;
  const GemvTask* tasks = nullptr;
  const int* cta_begin = nullptr;  // one range per warp (ncta * 4 + 1 entries); column pass: per CTA
  // 'N' launches: map 3 (FP32) tensor-core tiles, rpt 8-row tiles held; map 2: column-slice
  // window over tasks of at most 32 rows; map 1: half-warp row groups (at most 64 rows); maps 5
  // and 0: lanes over rows (at most 64 / 128); map 4 (FP32 y launches): the tensor-memory
  // kernel, one task at a time per CTA, units of at most kTcCols columns and kTcPieceBytes bytes.
  int rpt = 1;
  int map = 0;
  // 'T' launches: the most bytes of a unit's piece (column pass: with its column map) and the
  // most X rows of a unit (column pass: of a block).
  int piece_bytes = 0;
  int xrows = 0;
};

// Transposed products: a warp takes trans_cols columns at a time, trans_lanes lanes side by side
// (the other lanes split the rows); its accumulators are at most 64 registers at 16 (complex
// double: 4) right-hand sides.
__host__ __device__ constexpr int trans_lanes(int elem_bytes) { return elem_bytes >= 16 ? 4 : 8; }
__host__ __device__ constexpr int trans_cols(int elem_bytes) { return elem_bytes == 4 ? 32 : (elem_bytes == 8 ? 16 : 8); }
// CTAs an SM of a transposed launch.  8-byte types: three, which leaves the kernels at 16 right-hand
// sides their registers (FP64, 60,000-point cylinder, 11 right-hand sides: 382 us against 471 with
// spills at four) and is what their shared memory mostly allows; the others four (three: FP32 at
// one right-hand side 5 to 8% slower).
__host__ __device__ constexpr int trans_ctas_per_sm(int elem_bytes) { return elem_bytes == 8 ? 3 : 4; }
// Most bytes of a unit's piece (a unit holds trans_lanes columns at least, however tall), and the
// shared memory a CTA may use.
constexpr int kTransPieceBytes = 8192;
// Shape of a warp in the column pass: at 16 FP32 right-hand sides two columns on 16 lanes, since
// joining the slices of four columns on 8 lanes takes a third as many instructions as their sums
// (50,001-point cylinder, column pass with the z' sums: 107.6 -> 103.5 us).
__host__ __device__ constexpr int trans_column_lanes(int elem_bytes, int R) {
  return elem_bytes == 4 && R >= 16 ? 16 : trans_lanes(elem_bytes);
}
constexpr int kMaxCtaSmem = 227 * 1024;

// The arena's y region: per output block, the row panels of every leaf covering it side by side
// (full leaves n columns, Rk leaves their A panel of k columns) as one column-major matrix
// whose width is a multiple of kYColAlign (zero columns at the end, their X rows the zero rows
// of the xz buffer, kZeroRows of them after the x part).
constexpr int kYColAlign = 8;
constexpr int kZeroRows = 8;

// Unit capacities of the tensor-memory kernel: columns, piece bytes (128 rows x kTcCols),
// X rows bytes (kTcCols rows of 16 floats).
constexpr int kTcCols = 32;
constexpr int kTcPieceBytes = 128 * kTcCols * 4;
constexpr int kTcXBytes = kTcCols * 16 * 4;

// Per-stage capacities of the warp-level pipeline (bytes): one P piece and its X rows.  FP32
// pieces are 5,088 B: four CTAs of the tensor-core kernel (4 warps, two stages of 5,088 +
// 2,048 B a warp, 57.2 KB a CTA, 1 KB reserved) fill an SM's 228 KB, and the kernel's output
// tiles get the registers of four CTAs.  Against 3,584-B pieces at five CTAs an SM for the
// z-phase (the y-phase's 6 to 8 tiles already ran at four), fewer and larger units took the
// y-phase of the 100,000-point cylinder from 0.148 to 0.132 ms with the z-phase unchanged: per
// unit the kernel pays its barrier wait, descriptor and copy issue, and the larger pieces also
// keep more bytes in flight a warp.
// The FP64 and complex kernels use the same stage (the FP64 y-phase: 0.420 -> 0.403 ms against
// 4,096-byte pieces).
__host__ __device__ constexpr int warp_piece_bytes(int /*elem_bytes*/) { return 5088; }
constexpr int kWarpXBytes = 2048;
// FP32 units of short pieces (the z-phase's k x c blocks of B^T) may split the same stage the
// other way, kWarpXBytesWide bytes of X rows after a piece of the rest.
constexpr int kWarpXBytesWide = 3584;

// A sum of partial slots (a long group's or leaf's z, a strip's y): nparts consecutive slots of k
// rows from part_row are summed into final_row, with add != 0 on top of what stands there.
struct GemvZred {
  int final_row;
  unsigned short k, add;
  int part_row, nparts;
};

// The allocation-free products (noalloc.cu) take a matrix by a bound on its rows; every matrix
// within the bound is planned so that its rows, at the widest tile of right-hand sides, fit the
// array those products use.
constexpr long long kNoAllocBoundBytes = 16LL << 20;
constexpr long long kNoAllocArrayBytes = 40LL << 20;

// A round of the 'T' column pass: consecutive output blocks, then the sums [zred0, zred0 + nzred) of
// its partial slots, the first nzwide of them on a CTA each.  The rounds use the same slots.
struct GemvTransRound {
  GemvLaunch columns;
  int zred0 = 0, nzred = 0, nzwide = 0;
};

struct GemvSide {
  static const int kMaxLaunch = 4;
  int nz = 0;  // 'N': z-phase launches (one per rank class)
  GemvLaunch z[kMaxLaunch];
  int nzred = 0;   // 'N'
  int nzwide = 0;  // 'N': sums at the front of zred that take a CTA each
  const GemvZred* zred = nullptr;
  std::vector<GemvTransRound> rounds;  // 'T'
  const int* colmap = nullptr;  // 'T': destination rows of the column pass
  int ng = 0;                   // 'T': group-pass launches (one per group height class)
  GemvLaunch g[2];
  GemvLaunch y;  // 'N'
  const GemvUnit* units = nullptr;         // 'N'
  const GemvTransUnit* tunits = nullptr;   // 'T'
  // The y launches, the group pass and the column pass (full leaves; with several rounds, the sum of
  // their parts) write partial rows of the output blocks into xz; the final pass reads, per client
  // row i, yrows[i] = {xz row of part 0, nparts << 8 | O}.
  int nyrows = 0;
  const int2* yrows = nullptr;
};

struct GemvFullLeaf {
  int row_off, m, col_off, n;
  long long goff;  // canonical offset (gradients, payload): column-major m x n
};
struct GemvRkLeaf {
  int row_off, m, col_off, n, k, pad;
  long long goff;   // canonical offset: A (m x k) then B (n x k), column-major
  int zrow_n, zrow_t;  // xz rows of z = B^T x ('N') and z' = A^T x ('T' / 'C'), each in its numbering
};

// Status block of the products of one matrix, in device memory.  A kernel whose bounded
// wait for a bulk copy gives up sets `failed` (after waiting, again bounded, for the copies
// it has in flight) and stops; the host reads and clears it.  `wait_limit` bounds each wait
// (polls of a stage barrier); the drain after a give-up uses kGemvDrainLimit.
struct GemvStatus {
  int failed;
  int pad;
  long long wait_limit;
};
constexpr long long kGemvWaitLimit = 1LL << 26;
constexpr long long kGemvDrainLimit = 1LL << 26;

struct GemvTiming {
  cudaEvent_t ev[4];
};

struct GemvPlan {
  int n_rows = 0, n_cols = 0;
  int n_in_max = 0;      // rows of the x part of the xz buffer (kZeroRows zero rows follow it)
  // rows of the xz buffer of an 'N' and of a 'T' / 'C' product (x part, zero rows, z slots,
  // partial slots); the two numberings are independent (rows past the zero rows overlap)
  long long xz_rows[2] = {0, 0};
  const int* iperm_rows = nullptr;  // client -> internal
  const int* iperm_cols = nullptr;
  const void* arena = nullptr;
  int nfull = 0, nrk = 0;
  const GemvFullLeaf* full = nullptr;
  const GemvRkLeaf* rk = nullptr;
  GemvSide side[2];                       // [0] 'N', [1] 'T' / 'C'
};

}  // namespace hmatb200
