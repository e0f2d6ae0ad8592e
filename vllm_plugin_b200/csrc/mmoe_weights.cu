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

// One warp per output row; four 16-byte loads in flight per lane.
__global__ void __launch_bounds__(256) interleave_rows_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst,
                                                              int64_t total_rows, int rows, int vec) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; row < total_rows; row += warps) {
    const int64_t g = row / rows;
    const int r = static_cast<int>(row - g * rows);
    const uint4* s = src + (g * rows + interleave_src_row(r, rows)) * vec;
    uint4* d = dst + row * vec;
    for (int v0 = lane; v0 < vec; v0 += 128) {
      uint4 q[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (v0 + 32 * u < vec) q[u] = __ldcs(s + v0 + 32 * u);
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (v0 + 32 * u < vec) d[v0 + 32 * u] = q[u];
    }
  }
}

// One warp per 128-word block of a K column: stored position 4c + a holds row 32a + c of the block (after the optional
// gate/up interleave), so lane c gathers rows c, 32 + c, 64 + c, 96 + c -- four coalesced loads per warp (runs of eight
// words when rows are interleaved) -- and stores them as one 16-byte vector.  Two blocks in flight per warp.  HBM-bound;
// 48 experts (35 + 18 MB each way, in two launches): 45 us with one thread per word, 24 us in this form.
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

// Two-slice form of row-major matrices: half h of matrix g goes to dst + h * slice_stride + g * half_vec, contiguous both
// ways, so the copy is cut into pieces of 1024 vectors (16 KB) of one half each; a block takes a piece at a time with four
// 16-byte loads in flight per thread.  Pure HBM traffic: 48 experts (2 x 849 MB) take 284 us, 6.0 TB/s; as two strided
// byte-tensor copies per matrix they took 1790 us.
constexpr int kSplitPieceVec = 1024;
__global__ void __launch_bounds__(256) split_halves_kernel(const uint4* __restrict__ src, uint4* __restrict__ dst,
                                                           int num_halves, int64_t half_vec, int64_t slice_vec) {
  const int64_t pieces_per_half = (half_vec + kSplitPieceVec - 1) / kSplitPieceVec;
  const int64_t pieces = num_halves * pieces_per_half;
  for (int64_t i = blockIdx.x; i < pieces; i += gridDim.x) {
    const int64_t piece = pieces - 1 - i;                // from the end: what a transform in front has written last is still in L2
    const int64_t half = piece / pieces_per_half;        // 2 g + h, in source order
    const int64_t v0 = (piece - half * pieces_per_half) * kSplitPieceVec + threadIdx.x;
    const uint4* s = src + half * half_vec;
    uint4* d = dst + (half & 1) * slice_vec + (half >> 1) * half_vec;
    uint4 q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v0 + 256 * u < half_vec) q[u] = __ldcs(s + v0 + 256 * u);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (v0 + 256 * u < half_vec) __stcs(d + v0 + 256 * u, q[u]);
  }
}

}  // namespace

cudaError_t launch_interleave_rows(const void* src, void* dst, int groups, int rows, int row_bytes, cudaStream_t s) {
  const int64_t total = (int64_t)groups * rows;
  if (total == 0) return cudaSuccess;
  const int blocks = static_cast<int>(total / 8 + 1 < 148 * 16 ? total / 8 + 1 : 148 * 16);
  interleave_rows_kernel<<<blocks, 256, 0, s>>>(static_cast<const uint4*>(src), static_cast<uint4*>(dst), total, rows,
                                               row_bytes / 16);
  return cudaGetLastError();
}

cudaError_t launch_scale_layout(const int32_t* src, int32_t* dst, int groups, int rows, int row_stride, int kwords,
                                int interleave, cudaStream_t s) {
  const int64_t blocks128 = (int64_t)groups * kwords * (rows / 128);     // rows % 128 == 0: checked by the entry point
  if (blocks128 == 0) return cudaSuccess;
  const int blocks = static_cast<int>(blocks128 / 16 + 1 < 148 * 8 ? blocks128 / 16 + 1 : 148 * 8);
  scale_layout_kernel<<<blocks, 256, 0, s>>>(src, dst, blocks128, rows, row_stride, interleave);
  return cudaGetLastError();
}

cudaError_t launch_split_halves(const void* src, void* dst, int groups, int64_t half_bytes, int64_t slice_stride, cudaStream_t s) {
  const int64_t half_vec = half_bytes / 16, pieces = 2 * (int64_t)groups * ((half_vec + kSplitPieceVec - 1) / kSplitPieceVec);
  if (pieces == 0) return cudaSuccess;
  split_halves_kernel<<<static_cast<int>(pieces < 148 * 8 ? pieces : 148 * 8), 256, 0, s>>>(
      static_cast<const uint4*>(src), static_cast<uint4*>(dst), 2 * groups, half_vec, slice_stride / 16);
  return cudaGetLastError();
}

}  // namespace mmoe
