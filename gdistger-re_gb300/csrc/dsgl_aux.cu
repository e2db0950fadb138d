// dsgl_aux.cu -- set-up kernels (Wih initialisation, corpus mapping), the explicit-row
// minibatch update, and the SGNS loss with its hand-written adjoint.
#include <cuda_runtime.h>

#include <algorithm>

#include "dsgl_device.cuh"

namespace sgns {

namespace {

// InitNet (dsgl.hpp:451-456): element i of Wih takes LCG state r_{i+1} (r_0 = 1),
// value ((r & 0xFFFF) / 65536 - 0.5) / d.  Each thread owns 64 consecutive elements and
// starts from a jump-ahead; bf16 tables store the fp32 value rounded to nearest even.
__global__ void init_wih_kernel(void* wih, int storage, int64_t n, int32_t d, const LcgJumps* J) {
  const int64_t i0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * 64;
  if (i0 >= n) return;
  uint64_t r = jump_any(1ULL, (uint64_t)i0, J);
  const float fd = (float)d;
  for (int k = 0; k < 64 && i0 + k < n; k++) {
    r = lcg_next(r);
    const float v = __fdiv_rn(__fsub_rn(__fdiv_rn((float)(uint32_t)(r & 0xFFFF), 65536.0f), 0.5f), fd);
    if (storage == STORE_BF16)
      static_cast<__nv_bfloat16*>(wih)[i0 + k] = __float2bfloat16_rn(v);
    else
      static_cast<float*>(wih)[i0 + k] = v;
  }
}

// vertex ids -> sorted rows; -1 separators kept; anything else outside [0, V) flagged
__device__ __forceinline__ int32_t map_id(int32_t t, const int32_t* row_of, int64_t V, bool* bad) {
  if (t == -1) return -1;
  if (t < 0 || (int64_t)t >= V) {
    *bad = true;
    return -1;
  }
  return __ldg(&row_of[t]);
}
// ids may be device memory or pinned host memory mapped into the device's address space
// (then every id crosses the host link once, read in 16-byte pieces when aligned).
__global__ void map_corpus_kernel(const int32_t* ids, const int32_t* row_of, int32_t* rows, int64_t n,
                                  int64_t V, int32_t* bad, bool vec4) {
  bool b = false;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (vec4) {  // ids and rows 16-byte aligned
    const int64_t n4 = n >> 2;
    for (int64_t i = t0; i < n4; i += stride) {
      const int4 v = reinterpret_cast<const int4*>(ids)[i];
      reinterpret_cast<int4*>(rows)[i] = make_int4(map_id(v.x, row_of, V, &b), map_id(v.y, row_of, V, &b),
                                                   map_id(v.z, row_of, V, &b), map_id(v.w, row_of, V, &b));
    }
    for (int64_t i = (n4 << 2) + t0; i < n; i += stride) rows[i] = map_id(ids[i], row_of, V, &b);
  } else {
    for (int64_t i = t0; i < n; i += stride) rows[i] = map_id(ids[i], row_of, V, &b);
  }
  if (b) atomicExch(bad, 1);
}

// ---- explicit-row minibatch update (the step arithmetic of both trainers) ----------
// One block of four warps per minibatch, its rows staged in shared memory.  The sums are those
// of forward_gradient and backward (dsgl_device.cuh), one chain each, so they are spread by
// chain: dot products by (two outputs, input), outputMd by output, updates by input.
// What bounds it: the chains' latency (a dot product is d dependent multiply-adds) at the five
// blocks that 43 KB of rows (64 inputs, d = 128) leave per SM.  20,000 minibatches of 19.6
// inputs, d = 128, rounded write-back: 2,260 us with one warp per minibatch, the sigmoid table
// copied to shared memory per block and a one-thread prefix of the counts; 297 us now
// (60 us of bytes).
constexpr int kMbThreads = 128;
constexpr int kMbOwnPrefix = 1024;  // up to here a block sums the counts before its own itself

// sum over the block of each thread's a and b (int64)
__device__ __forceinline__ void block_sum2(int64_t& a, int64_t& b, int64_t* scratch) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(kFull, a, o);
    b += __shfl_xor_sync(kFull, b, o);
  }
  if (lane_id() == 0) {
    scratch[2 * (threadIdx.x >> 5)] = a;
    scratch[2 * (threadIdx.x >> 5) + 1] = b;
  }
  __syncthreads();
  a = b = 0;
#pragma unroll
  for (int k = 0; k < kMbThreads / 32; k++) {
    a += scratch[2 * k];
    b += scratch[2 * k + 1];
  }
}

// kRound: instead of the updates, write each updated row (row + update) as bf16 bits with
// the trainers' stochastic rounding (RowIO<STORE_BF16>::store4), event keys from sr_seed
// and the minibatch index; d_in / d_out then point to uint16 rows.  in_off null: the block
// sums the counts of the minibatches before it.
template <bool kRound>
__global__ void __launch_bounds__(kMbThreads) minibatch_kernel(int d, int imax, int omax, const int32_t* in_count,
                                                               const int32_t* in_first, const int32_t* out_count,
                                                               const int32_t* out_meta_all, const float* alpha,
                                                               const int64_t* in_off, const int64_t* out_off,
                                                               const float* in_rows, const float* out_rows,
                                                               float* d_in, float* d_out,
                                                               const float* __restrict__ exp_table, int32_t* status,
                                                               uint64_t sr_seed) {
  extern __shared__ __align__(16) float smem[];
  __shared__ int64_t sums[2 * (kMbThreads / 32)];
  const int b = blockIdx.x, lane = lane_id(), warp = threadIdx.x >> 5;
  const int I = in_count[b], first = in_first[b], O = out_count[b];
  if (I < 1 || I > imax || O < 2 || O > omax || first < 0 || first > I) {
    if (threadIdx.x == 0) atomicExch(status, 1);
    return;
  }
  int64_t i_at, o_at;
  if (in_off) {
    i_at = in_off[b], o_at = out_off[b];
  } else {
    i_at = o_at = 0;  // (a negative count adds nothing, as in prefix_offsets_kernel)
    for (int k = threadIdx.x; k < b; k += kMbThreads) {
      i_at += max(in_count[k], 0);
      o_at += max(out_count[k], 0);
    }
    block_sum2(i_at, o_at, sums);
  }
  const int DP = d + 4, d4 = d >> 2;  // rows 4 banks apart
  constexpr int CS = kOMax;
  float* xin = smem;
  float* out = xin + (size_t)imax * DP;
  float* corr = out + (size_t)kOMax * DP;
  const float* gin = in_rows + i_at * d;
  const float* gout = out_rows + o_at * d;
  for (int e = threadIdx.x; e < (I + O) * d4; e += kMbThreads) {
    const int r = e / d4, q = e - r * d4;
    const float4 v = r < I ? reinterpret_cast<const float4*>(gin)[e] : reinterpret_cast<const float4*>(gout)[e - I * d4];
    reinterpret_cast<float4*>(r < I ? xin + r * DP : out + (r - I) * DP)[q] = v;
  }
  __syncthreads();
  // dot products of outputs 2p, 2p + 1 with input j, then their gradients (dsgl.hpp:1243-1272)
  const float al = alpha[b];
  const int cols = (I + 31) & ~31;  // a warp's lanes hold different inputs against the same outputs
  for (int t = threadIdx.x; t < cols * ((O + 1) >> 1); t += kMbThreads) {
    const int p = t / cols, j = t - p * cols;
    if (j >= I) continue;
    const float4* x = reinterpret_cast<const float4*>(xin + j * DP);
    const float4* oa = reinterpret_cast<const float4*>(out + 2 * p * DP);
    const float4* ob = reinterpret_cast<const float4*>(out + (2 * p + 1 < O ? 2 * p + 1 : 2 * p) * DP);
    float f[2] = {0.f, 0.f};
#pragma unroll 4
    for (int k = 0; k < d4; k++) {
      const float4 xv = x[k], u = oa[k], v = ob[k];
      f[0] = __fmaf_rn(u.x, xv.x, f[0]);
      f[1] = __fmaf_rn(v.x, xv.x, f[1]);
      f[0] = __fmaf_rn(u.y, xv.y, f[0]);
      f[1] = __fmaf_rn(v.y, xv.y, f[1]);
      f[0] = __fmaf_rn(u.z, xv.z, f[0]);
      f[1] = __fmaf_rn(v.z, xv.z, f[1]);
      f[0] = __fmaf_rn(u.w, xv.w, f[0]);
      f[1] = __fmaf_rn(v.w, xv.w, f[1]);
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int i = 2 * p + h;
      if (i < O)
        corr[j * CS + i] = step_gradient(f[h], j < first ? (i == 0) : (i == O - 1), exp_table, al, out_meta_all[o_at + i]);
    }
  }
  __syncthreads();
  // event keys of the rounded rows: EV_WALK0 (inputs) and EV_NEG (outputs) of minibatch b, row
  // index within the minibatch -- the trainers' rounding rule and hash
  const uint64_t ev_in = kRound ? sr_event_key(sr_seed, EV_WALK0, 0u, (uint64_t)b) : 0;
  const uint64_t ev_out = kRound ? sr_event_key(sr_seed, EV_NEG, 0u, (uint64_t)b) : 0;
  uint16_t* gin16 = reinterpret_cast<uint16_t*>(d_in) + i_at * d;
  uint16_t* gout16 = reinterpret_cast<uint16_t*>(d_out) + o_at * d;
  for (int q = lane; q < d4; q += 32) {
    // outputMd_i = sum_j g_ij x_j, in input order
    for (int i = warp; i < O; i += kMbThreads / 32) {
      float4 m = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int j = 0; j < I; j++) m = fma4s(corr[j * CS + i], reinterpret_cast<const float4*>(xin + j * DP)[q], m);
      if (kRound)
        RowIO<STORE_BF16>::store4(gout16, i, d, q, add4(reinterpret_cast<const float4*>(out + i * DP)[q], m), ev_out);
      else
        reinterpret_cast<float4*>(d_out + (o_at + i) * d)[q] = m;
    }
    // input j's update = sum_i g_ij o_i, in output order
    for (int j = warp; j < I; j += kMbThreads / 32) {
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
      for (int i = 0; i < O; i++) a = fma4s(corr[j * CS + i], reinterpret_cast<const float4*>(out + i * DP)[q], a);
      if (kRound)
        RowIO<STORE_BF16>::store4(gin16, j, d, q, add4(reinterpret_cast<const float4*>(xin + j * DP)[q], a), ev_in);
      else
        reinterpret_cast<float4*>(d_in + (i_at + j) * d)[q] = a;
    }
  }
}

// each walk start scans forward to its separator (at most kMaxSentence tokens); one
// atomic per warp
__global__ void max_walk_kernel(const int32_t* rows, int64_t n, int32_t* out) {
  int best = 0;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    if (rows[i] == -1 || (i > 0 && rows[i - 1] != -1)) continue;
    int len = 0;
    while (i + len < n && rows[i + len] != -1 && len < kMaxSentence) len++;
    best = len > best ? len : best;
  }
  for (int o = 16; o > 0; o >>= 1) {
    const int t = __shfl_xor_sync(kFull, best, o);
    best = t > best ? t : best;
  }
  if ((threadIdx.x & 31) == 0 && best > 0) atomicMax(out, best);
}

// Exclusive prefixes of two count arrays, one block: each thread sums its run of consecutive
// counts, the runs are scanned, the runs are written.  A negative count (rejected by its own
// minibatch) adds nothing, so no later minibatch's offset points before the start of the
// caller's row arrays.
constexpr int kPrefixThreads = 1024;
__global__ void __launch_bounds__(kPrefixThreads) prefix_offsets_kernel(const int32_t* cnt_a, const int32_t* cnt_b, int n,
                                                                        int64_t* off_a, int64_t* off_b) {
  __shared__ int64_t wa[32], wb[32];
  const int lane = lane_id(), warp = threadIdx.x >> 5;
  const int run = (n + kPrefixThreads - 1) / kPrefixThreads;
  const int lo = min((int64_t)threadIdx.x * run, (int64_t)n), hi = min((int64_t)lo + run, (int64_t)n);
  int64_t a = 0, b = 0;
  for (int i = lo; i < hi; i++) {
    a += max(cnt_a[i], 0);
    b += max(cnt_b[i], 0);
  }
  int64_t ia = a, ib = b;  // inclusive over the warp, then the block
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t u = __shfl_up_sync(kFull, ia, o), v = __shfl_up_sync(kFull, ib, o);
    if (lane >= o) ia += u, ib += v;
  }
  if (lane == 31) wa[warp] = ia, wb[warp] = ib;
  __syncthreads();
  if (warp == 0) {
    int64_t u = wa[lane], v = wb[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t x = __shfl_up_sync(kFull, u, o), y = __shfl_up_sync(kFull, v, o);
      if (lane >= o) u += x, v += y;
    }
    wa[lane] = u, wb[lane] = v;
  }
  __syncthreads();
  a = ia - a + (warp ? wa[warp - 1] : 0);
  b = ib - b + (warp ? wb[warp - 1] : 0);
  for (int i = lo; i < hi; i++) {
    off_a[i] = a;
    off_b[i] = b;
    a += max(cnt_a[i], 0);
    b += max(cnt_b[i], 0);
  }
}

}  // namespace

// bf16 bits -> fp32 (exact), 4 elements per thread; n % 4 == 0 (d is a multiple of 4)
__global__ void widen_bf16_kernel(const uint2* __restrict__ src, float4* __restrict__ dst, int64_t n4) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
    const uint2 u = src[i];
    dst[i] = make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xFFFF0000u), __uint_as_float(u.y << 16),
                         __uint_as_float(u.y & 0xFFFF0000u));
  }
}

// ---- hotness-block sync: rows out of and back into a table (one warp per row) ----------
__global__ void gather_rows_kernel(const void* tab, int storage, int d, const int32_t* rows, int64_t n, float* buf) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const int64_t r = rows[i];
    for (int c = lane; c < d; c += 32)
      buf[i * d + c] = storage == STORE_BF16 ? bf16_bits_to_f32(static_cast<const uint16_t*>(tab)[r * d + c])
                                             : static_cast<const float*>(tab)[r * d + c];
  }
}
// row = buf / divisor (fp32 division, as the reference averages, dsgl.hpp:741-745); bf16
// tables round to nearest even, so every rank stores the same bits
__global__ void scatter_rows_kernel(void* tab, int storage, int d, const int32_t* rows, int64_t n, const float* buf,
                                    float divisor) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
  for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < n; i += warps) {
    const int64_t r = rows[i];
    for (int c = lane; c < d; c += 32) {
      const float v = __fdiv_rn(buf[i * d + c], divisor);
      if (storage == STORE_BF16) {
        const uint32_t u = __float_as_uint(v);
        uint16_t b;
        if ((u & 0x7F800000u) == 0x7F800000u) b = (uint16_t)((u >> 16) | ((u & 0xFFFFu) ? 0x40u : 0u));
        else b = (uint16_t)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16);
        static_cast<uint16_t*>(tab)[r * d + c] = b;
      } else {
        static_cast<float*>(tab)[r * d + c] = v;
      }
    }
  }
}

cudaError_t launch_gather_rows(const void* tab, int storage, int d, const int32_t* rows, int64_t n, float* buf,
                               cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int64_t blocks = std::min<int64_t>((n + 7) / 8, 152 * 16);
  gather_rows_kernel<<<(unsigned)blocks, 256, 0, s>>>(tab, storage, d, rows, n, buf);
  return cudaGetLastError();
}
cudaError_t launch_scatter_rows(void* tab, int storage, int d, const int32_t* rows, int64_t n, const float* buf,
                                float divisor, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  const int64_t blocks = std::min<int64_t>((n + 7) / 8, 152 * 16);
  scatter_rows_kernel<<<(unsigned)blocks, 256, 0, s>>>(tab, storage, d, rows, n, buf, divisor);
  return cudaGetLastError();
}

cudaError_t launch_widen_bf16(const void* src, float* dst, int64_t n, cudaStream_t s) {
  const int64_t n4 = n / 4;
  if (n4 == 0) return cudaSuccess;
  const int64_t blocks = (n4 + 255) / 256;
  widen_bf16_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0, s>>>(static_cast<const uint2*>(src),
                                                                             reinterpret_cast<float4*>(dst), n4);
  return cudaGetLastError();
}

cudaError_t launch_init_wih(void* wih, int storage, int64_t V, int32_t d, const LcgJumps* jumps,
                            cudaStream_t s) {
  const int64_t n = V * d;
  const int64_t threads = (n + 63) / 64;
  init_wih_kernel<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(wih, storage, n, d, jumps);
  return cudaGetLastError();
}

cudaError_t launch_map_corpus(const int32_t* ids, const int32_t* row_of, int32_t* rows, int64_t n,
                              int64_t V, int32_t* bad, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 152 * 32) blocks = 152 * 32;
  const bool vec4 = ((reinterpret_cast<uintptr_t>(ids) | reinterpret_cast<uintptr_t>(rows)) & 15) == 0;
  map_corpus_kernel<<<(unsigned)blocks, 256, 0, s>>>(ids, row_of, rows, n, V, bad, vec4);
  return cudaGetLastError();
}

cudaError_t launch_max_walk(const int32_t* rows, int64_t n, int32_t* out, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 152 * 32) blocks = 152 * 32;
  max_walk_kernel<<<(unsigned)blocks, 256, 0, s>>>(rows, n, out);
  return cudaGetLastError();
}

namespace {
template <bool kRound>
cudaError_t minibatch_launch(int d, int n, int imax, const int32_t* in_count, const int32_t* in_first,
                             const int32_t* out_count, const int32_t* out_meta, const float* alpha,
                             const float* in_rows, const float* out_rows, float* d_in, float* d_out, uint64_t sr_seed,
                             const float* exp_table, int64_t* offsets, int32_t* status, cudaStream_t s) {
  if (n == 0) return cudaSuccess;
  // small calls: a launch saved is worth the counts being read by every block
  int64_t* in_off = n <= kMbOwnPrefix ? nullptr : offsets;
  int64_t* out_off = n <= kMbOwnPrefix ? nullptr : offsets + n;
  if (in_off) prefix_offsets_kernel<<<1, kPrefixThreads, 0, s>>>(in_count, out_count, n, in_off, out_off);
  const size_t smem = sizeof(float) * ((size_t)(imax + kOMax) * (d + 4) + (size_t)imax * kOMax);
  cudaError_t e = cudaFuncSetAttribute(minibatch_kernel<kRound>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  minibatch_kernel<kRound><<<n, kMbThreads, smem, s>>>(d, imax, kOMax, in_count, in_first, out_count, out_meta, alpha,
                                                       in_off, out_off, in_rows, out_rows, d_in, d_out, exp_table,
                                                       status, sr_seed);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_minibatch_bf16(int d, int n, int imax, const int32_t* in_count, const int32_t* in_first,
                                  const int32_t* out_count, const int32_t* out_meta, const float* alpha,
                                  const float* in_rows, const float* out_rows, uint16_t* new_in, uint16_t* new_out,
                                  uint64_t sr_seed, const float* exp_table, int64_t* offsets, int32_t* status,
                                  cudaStream_t s) {
  return minibatch_launch<true>(d, n, imax, in_count, in_first, out_count, out_meta, alpha, in_rows, out_rows,
                                reinterpret_cast<float*>(new_in), reinterpret_cast<float*>(new_out), sr_seed, exp_table,
                                offsets, status, s);
}

cudaError_t launch_minibatch(int d, int n, int imax, int omax, const int32_t* in_count,
                             const int32_t* in_first, const int32_t* out_count, const int32_t* out_meta,
                             const float* alpha, const float* in_rows, const float* out_rows, float* d_in,
                             float* d_out, const float* exp_table, int64_t* offsets, int32_t* status,
                             cudaStream_t s) {
  (void)omax;
  return minibatch_launch<false>(d, n, imax, in_count, in_first, out_count, out_meta, alpha, in_rows, out_rows, d_in,
                                 d_out, 0, exp_table, offsets, status, s);
}

}  // namespace sgns
