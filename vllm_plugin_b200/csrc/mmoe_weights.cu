// Load-time weight transform of the MegaMoE layer as CUDA kernels for sm_100a: the byte shuffles that turn checkpoint-
// order expert weights into the layout the grouped GEMMs read (the reference does them with torch indexing ops,
// backend/weights.py:83-145).
//
//   rows     W13 [gate | up] -> [g0..7, u0..7, g8..15, u8..15, ...] per expert (W2 rows are copied unchanged)
//   scales   int32 words (four UE8M0 bytes each), MN-major [G][K/128][rows]: the same row interleave for W13, then
//            inside every 128-row block the 4x32 transpose (stored position 4c + a holds row 32a + c), which makes each
//            (128 rows, 128 K) block one contiguous 512-byte chunk in the order tcgen05.cp copies into tensor memory
//
// Pure HBM-bound byte movement: every input byte is read once and written once.
#include "mmoe_common.cuh"

namespace mmoe {

namespace {

// source row (in [gate | up] order) of output row r of a matrix with `rows` rows (rows/2 gate + rows/2 up channels)
__device__ __forceinline__ int interleave_src_row(int r, int rows) {
  const int channel = ((r >> 4) << 3) | (r & 7);
  return ((r >> 3) & 1) * (rows >> 1) + channel;
}

// Copies run in pieces that are contiguous on both sides, with a block per piece and five 16-byte loads in flight per thread: 20 KB for
// the two-slice copy, eight rows for the row order, which is 20 KB at hidden 5120 (other widths leave part of the loads idle in the
// last pass).  Blocks that
// walked pieces 148 x 8 apart instead read and wrote too many DRAM pages at a time: 48 experts, rows and both halves 494 -> 446 us
// (transform 210 -> 195, two-slice copy 292 -> 254 us, 6.7 TB/s); with ten loads of 128 threads 450, four of 512 462.
// kAgain: the result is read again soon (the two-slice copy of what the transform has written).
constexpr int kCopyThreads = 256, kCopyLoads = 5;
template <bool kAgain>
__device__ __forceinline__ void copy_run(const uint4* __restrict__ src, uint4* __restrict__ dst, int64_t n) {
  for (int64_t v0 = threadIdx.x; v0 < n; v0 += kCopyLoads * kCopyThreads) {
    uint4 q[kCopyLoads];
#pragma unroll
    for (int u = 0; u < kCopyLoads; ++u)
      if (v0 + kCopyThreads * u < n) q[u] = __ldcs(src + v0 + kCopyThreads * u);
#pragma unroll
    for (int u = 0; u < kCopyLoads; ++u)
      if (v0 + kCopyThreads * u < n) {
        if (kAgain) dst[v0 + kCopyThreads * u] = q[u];
        else __stcs(dst + v0 + kCopyThreads * u, q[u]);
      }
  }
}

// A block per eight output rows, which are neighbours in the input too.
__global__ void __launch_bounds__(kCopyThreads) interleave_rows_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst, int rows, int vec) {
  const int64_t row = 8 * (int64_t)blockIdx.x, g = row / rows;
  const int r = static_cast<int>(row - g * rows);
  copy_run<true>(src + (g * rows + interleave_src_row(r, rows)) * vec, dst + row * vec, 8 * (int64_t)vec);
}

// One warp per 128-word block of a K column: stored position 4c + a holds row 32a + c of the block (after the optional
// gate/up interleave), so lane c gathers rows c, 32 + c, 64 + c, 96 + c -- four coalesced loads per warp (runs of eight
// words when rows are interleaved) -- and stores them as one 16-byte vector.  Two blocks in flight per warp.  HBM-bound;
// 48 experts (35 + 18 MB each way, in two launches): 45 us with one thread per word, 24 us in this form, 22.5 with
// a grid that is not cut off at 148 x 8 blocks.
__global__ void __launch_bounds__(256) scale_layout_kernel(const int32_t* __restrict__ src, int32_t* __restrict__ dst,
                                                           int64_t total_blocks, int rows, int row_stride, int interleave) {
  const int lane = threadIdx.x & 31;
  const int blocks_per_col = rows >> 7;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; b < total_blocks; b += 2 * warps) {
    int4 v[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t bu = b + u * warps;
      if (bu >= total_blocks) break;
      const int64_t col = bu / blocks_per_col;         // g * kwords + w
      const int r0 = static_cast<int>(bu - col * blocks_per_col) * 128 + lane;
      const int32_t* in = src + col * row_stride;
      int r[4];
#pragma unroll
      for (int a = 0; a < 4; ++a) r[a] = interleave ? interleave_src_row(r0 + 32 * a, rows) : r0 + 32 * a;
      v[u] = make_int4(__ldcs(in + r[0]), __ldcs(in + r[1]), __ldcs(in + r[2]), __ldcs(in + r[3]));
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int64_t bu = b + u * warps;
      if (bu >= total_blocks) break;
      const int64_t col = bu / blocks_per_col;
      const int blk = static_cast<int>(bu - col * blocks_per_col);
      __stcs(reinterpret_cast<int4*>(dst + col * row_stride + blk * 128) + lane, v[u]);
    }
  }
}

// Two-slice form of row-major matrices: half h of matrix g goes to dst + h * slice_stride + g * half_vec, contiguous both ways, so
// the copy is cut into pieces of one half each.  (As two strided byte-tensor copies per matrix 48 experts took 1790 us.)
constexpr int kSplitPieceVec = kCopyThreads * kCopyLoads;
__global__ void __launch_bounds__(kCopyThreads) split_halves_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst,
                                                                    int64_t pieces_per_half, int64_t half_vec, int64_t slice_vec) {
  const int64_t piece = (int64_t)gridDim.x - 1 - blockIdx.x;   // from the end: what a transform in front has written last is still in L2
  const int64_t half = piece / pieces_per_half;                // 2 g + h, in source order
  const int64_t v0 = (piece - half * pieces_per_half) * kSplitPieceVec, left = half_vec - v0;
  copy_run<false>(src + half * half_vec + v0, dst + (half & 1) * slice_vec + (half >> 1) * half_vec + v0, left < kSplitPieceVec ? left : kSplitPieceVec);
}

}  // namespace

cudaError_t launch_interleave_rows(const void* src, void* dst, int groups, int rows, int row_bytes, cudaStream_t s) {
  const int64_t eights = (int64_t)groups * rows / 8;             // rows % 16 == 0: checked by the entry point
  if (eights == 0) return cudaSuccess;
  if (eights > INT32_MAX) return cudaErrorInvalidValue;
  return launch_plain(interleave_rows_kernel, dim3(static_cast<unsigned>(eights)), dim3(kCopyThreads), 0, s, static_cast<const uint4*>(src),
                      static_cast<uint4*>(dst), rows, row_bytes / 16);
}

cudaError_t launch_scale_layout(const int32_t* src, int32_t* dst, int groups, int rows, int row_stride, int kwords,
                                int interleave, cudaStream_t s) {
  const int64_t blocks128 = (int64_t)groups * kwords * (rows / 128);     // rows % 128 == 0: checked by the entry point
  if (blocks128 == 0) return cudaSuccess;
  if (blocks128 / 16 >= INT32_MAX) return cudaErrorInvalidValue;
  return launch_plain(scale_layout_kernel, dim3(static_cast<unsigned>(blocks128 / 16 + 1)), dim3(256), 0, s, src, dst, blocks128, rows, row_stride, interleave);
}

cudaError_t launch_split_halves(const void* src, void* dst, int groups, int64_t half_bytes, int64_t slice_stride, cudaStream_t s) {
  const int64_t half_vec = half_bytes / 16, per_half = (half_vec + kSplitPieceVec - 1) / kSplitPieceVec, pieces = 2 * (int64_t)groups * per_half;
  if (pieces == 0) return cudaSuccess;
  if (pieces > INT32_MAX) return cudaErrorInvalidValue;
  return launch_plain(split_halves_kernel, dim3(static_cast<unsigned>(pieces)), dim3(kCopyThreads), 0, s, static_cast<const uint4*>(src),
                      static_cast<uint4*>(dst), per_half, half_vec, slice_stride / 16);
}

}  // namespace mmoe
