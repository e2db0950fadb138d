// dsgl_eval.cu -- link-prediction scores of held-out pairs: score = <row_u, row_v> of one
// embedding table (fp32 or bf16), the dot-product scoring applied to the holdout that
// src/tools/gtrain.cpp:226-385 writes (test edges and sampled non-edges).
//
// A warp takes kPairs pairs at a time.  Lane l owns columns 4l..4l+3 of each 128-column chunk
// t (chunk order t = 0, 1, ...); it sums u[c] * v[c] over its columns in that order with one
// fused multiply-add per column, then the 32 partial sums of a pair are added by an xor
// butterfly (offsets 16, 8, 4, 2, 1).  The order is fixed, so the CPU restatement reproduces
// every score bit for bit.  The butterfly runs for all pairs at once: at each of its first
// steps a lane hands over the half of the sums that its partner goes on with, and addition
// commutes, so each sum has the bits of a butterfly of its own.
//
// What bounds it: HBM, 2 d s bytes a pair (s = 4 or 2), while enough row loads are in flight.
// One pair per warp, its ids loaded first, had too few: 20M pairs of 128 bf16 columns took
// 2,460 us (4.2 TB/s) and take 1,451 (7.1 TB/s, a few rows being in L2); of 128 fp32 columns
// 3,690 -> 2,806; of 200 (6M pairs) 1,683 -> 1,513; of 256 as before (7.2 TB/s).
#include <cuda_runtime.h>

#include <algorithm>

#include "dsgl_device.cuh"

namespace sgns {

namespace {

template <int S, int kPairs, int kChunks, int kBlocks>
__global__ void __launch_bounds__(256, kBlocks)
link_scores_kernel(const void* table, int d, int64_t V, const int32_t* pairs, int64_t n, float* scores, int32_t* bad) {
  typedef typename RowIO<S>::Raw Raw;
  const int lane = lane_id();
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  const int64_t groups = (n + kPairs - 1) / kPairs;
  const int d4 = d >> 2;
  int64_t g = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  // lane k < 2 kPairs holds word k of the group's pairs, read one group ahead; 0 behind the end
  const auto ids_of = [&](int64_t grp) {
    const int64_t at = grp * (2 * kPairs) + lane;
    return lane < 2 * kPairs && at < 2 * n ? pairs[at] : 0;
  };
  int32_t next = ids_of(g);
  for (; g < groups; g += warps) {
    int32_t ids = next;
    next = ids_of(g + warps);
    const bool in_range = ids >= 0 && (int64_t)ids < V;
    const unsigned out = ~__ballot_sync(kFull, in_range);  // words outside the table
    if (!in_range) ids = 0;                                // their pairs score 0 and are reported
    float acc[kPairs];
#pragma unroll
    for (int p = 0; p < kPairs; p++) acc[p] = 0.f;
    int32_t u[kPairs], v[kPairs];
#pragma unroll
    for (int p = 0; p < kPairs; p++) {
      u[p] = __shfl_sync(kFull, ids, 2 * p);
      v[p] = __shfl_sync(kFull, ids, 2 * p + 1);
    }
#pragma unroll 1
    for (int q = lane; q < d4; q += 32 * kChunks) {
      Raw x[kChunks][kPairs], y[kChunks][kPairs];
#pragma unroll
      for (int c = 0; c < kChunks; c++) {
        if (c > 0 && q + 32 * c >= d4) break;
#pragma unroll
        for (int p = 0; p < kPairs; p++) {
          x[c][p] = RowIO<S>::load_raw(table, u[p], d, q + 32 * c);
          y[c][p] = RowIO<S>::load_raw(table, v[p], d, q + 32 * c);
        }
      }
#pragma unroll
      for (int c = 0; c < kChunks; c++) {
        if (c > 0 && q + 32 * c >= d4) break;
#pragma unroll
        for (int p = 0; p < kPairs; p++) {
          const float4 a = RowIO<S>::widen(x[c][p]), b = RowIO<S>::widen(y[c][p]);
          acc[p] = __fmaf_rn(a.x, b.x, acc[p]);
          acc[p] = __fmaf_rn(a.y, b.y, acc[p]);
          acc[p] = __fmaf_rn(a.z, b.z, acc[p]);
          acc[p] = __fmaf_rn(a.w, b.w, acc[p]);
        }
      }
    }
    int o = 16;
#pragma unroll
    for (int half = kPairs / 2; half > 0; half >>= 1, o >>= 1) {
#pragma unroll
      for (int k = 0; k < half; k++) {
        const bool upper = lane & o;
        const float send = upper ? acc[k] : acc[k + half], keep = upper ? acc[k + half] : acc[k];
        acc[k] = __fadd_rn(keep, __shfl_xor_sync(kFull, send, o));
      }
    }
    for (; o > 0; o >>= 1) acc[0] = __fadd_rn(acc[0], __shfl_xor_sync(kFull, acc[0], o));
    // pair p's sum is in lanes p * 32 / kPairs and up
    const int p = lane / (32 / kPairs);
    if (lane % (32 / kPairs) == 0 && g * kPairs + p < n) {
      const bool miss = (out >> (2 * p)) & 3u;
      scores[g * kPairs + p] = miss ? 0.f : acc[0];
      if (miss) atomicExch(bad, 1);
    }
  }
}

}  // namespace

template <int S, int kPairs, int kChunks, int kBlocks>
cudaError_t link_scores_of(const void* table, int d, int64_t V, const int32_t* pairs, int64_t n, float* scores,
                           int32_t* bad, int num_sms, cudaStream_t s) {
  const int64_t blocks = std::min<int64_t>((n + 8 * kPairs - 1) / (8 * kPairs), (int64_t)num_sms * kBlocks);
  link_scores_kernel<S, kPairs, kChunks, kBlocks><<<(unsigned)blocks, 256, 0, s>>>(table, d, V, pairs, n, scores, bad);
  return cudaGetLastError();
}

// Pairs per warp, 128-column chunks in flight and blocks per SM, from a sweep of 1 to 8 pairs
// and 2 to 8 blocks (2.2M rows; 8 warps a block, all blocks resident, so that no wave is left
// half empty).  Random rows want about 64 KB of loads in flight per SM, less for long rows, and
// fall off above.  20M pairs of 256-byte bf16 rows: 2 pairs x 8 blocks 1,760 us, 4 x 4 1,451,
// 4 x 5 2,140, 8 x 3 3,120.  20M pairs of 512-byte fp32 rows: 1 x 8 3,017 us, 2 x 4 2,806, 2 x 6
// 3,050.  6M pairs of 1 KB rows: 2 x 4 a chunk at a time 1,790 us; both chunks of one pair in
// flight 1,750 with 8 blocks, 1,707 with 4.
cudaError_t launch_link_scores(int storage, const void* table, int d, int64_t V, const int32_t* pairs, int64_t n,
                               float* scores, int32_t* bad, int num_sms, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  if (storage == STORE_BF16) return link_scores_of<STORE_BF16, 4, 1, 4>(table, d, V, pairs, n, scores, bad, num_sms, s);
  if (d <= 128) return link_scores_of<STORE_F32, 2, 1, 4>(table, d, V, pairs, n, scores, bad, num_sms, s);
  return link_scores_of<STORE_F32, 1, 2, 4>(table, d, V, pairs, n, scores, bad, num_sms, s);
}

}  // namespace sgns
