// dsgl_device.cuh -- device building blocks shared by the DSGL engines: storage row
// access (fp32 / bf16 with stochastic rounding), LCG jump-ahead, warp-parallel walk fill,
// negative draws, and the step arithmetic (forward + gradient, both backward products).
//
// Arithmetic contract: every dot product and both backward products are sequential in
// the reduction index, one fused multiply-add per term (the order of the reference's
// loops, dsgl.hpp:1226-1229, 1282-1285, 1301-1304); every other float expression is an
// explicit _rn intrinsic so no contraction can change it.  With one worker the engines
// therefore reproduce the CPU oracle bit for bit.
#pragma once
#include <cuda_bf16.h>
#include <cstdint>

#include "sgns_internal.h"

namespace sgns {

constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}
// index of the n-th (0-based) set bit of x; x has more than n bits set
__device__ __forceinline__ int nth_set_bit(unsigned x, int n) {
  for (int i = 0; i < n; i++) x &= x - 1;
  return __ffs(x) - 1;
}

// Stochastic rounding of two floats to a bf16 pair in one instruction (sm_100a and later):
// lo gets rbits[15:0] and lands in the low half, hi gets rbits[31:16].  For every non-NaN
// input the result equals truncating (bits(x) + r16) to its upper 16 bits; NaN becomes
// 0x7FFF.
__device__ __forceinline__ uint32_t cvt_rs_bf16x2(float lo, float hi, uint32_t rbits) {
  uint32_t d;
  asm("cvt.rs.bf16x2.f32 %0, %1, %2, %3;" : "=r"(d) : "f"(hi), "f"(lo), "r"(rbits));
  return d;
}

// ---- storage rows ------------------------------------------------------------------
// A row of d elements; column chunk q holds columns 4q..4q+3 (d % 4 == 0).
template <int S> struct RowIO;

template <> struct RowIO<STORE_F32> {
  static constexpr int kBytes = 4;
  typedef float4 Raw;  // a chunk as loaded, before widening to fp32
  __device__ static __forceinline__ Raw load_raw(const void* base, int64_t row, int d, int q) {
    return reinterpret_cast<const float4*>(static_cast<const float*>(base) + row * d)[q];
  }
  __device__ static __forceinline__ Raw load_l2(const void* base, int64_t row, int d, int q) {  // past the L1
    return __ldcg(reinterpret_cast<const float4*>(static_cast<const float*>(base) + row * d) + q);
  }
  __device__ static __forceinline__ float4 widen(Raw r) { return r; }
  __device__ static __forceinline__ float4 load4(const void* base, int64_t row, int d, int q) {
    return reinterpret_cast<const float4*>(static_cast<const float*>(base) + row * d)[q];
  }
  __device__ static __forceinline__ float4 store4(void* base, int64_t row, int d, int q, float4 v,
                                                  uint64_t) {
    reinterpret_cast<float4*>(static_cast<float*>(base) + row * d)[q] = v;
    return v;
  }
};

template <> struct RowIO<STORE_BF16> {
  static constexpr int kBytes = 2;
  typedef uint2 Raw;
  __device__ static __forceinline__ Raw load_raw(const void* base, int64_t row, int d, int q) {
    return reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(base) + row * d)[q];
  }
  __device__ static __forceinline__ Raw load_l2(const void* base, int64_t row, int d, int q) {  // past the L1
    return __ldcg(reinterpret_cast<const uint2*>(static_cast<const uint16_t*>(base) + row * d) + q);
  }
  __device__ static __forceinline__ float4 widen(Raw u) {
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xFFFF0000u),
                       __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xFFFF0000u));
  }
  __device__ static __forceinline__ float4 load4(const void* base, int64_t row, int d, int q) {
    return widen(load_raw(base, row, d, q));
  }
  // Stores with stochastic rounding; returns the values actually stored (as fp32).
  // Column 4q+j takes random bits [16j, 16j+16) of sr_bits4.
  __device__ static __forceinline__ float4 store4(void* base, int64_t row, int d, int q, float4 v,
                                                  uint64_t ev) {
    const uint64_t bits = sr_bits4(ev, (uint32_t)row, (uint32_t)q);
    const uint2 u = make_uint2(cvt_rs_bf16x2(v.x, v.y, (uint32_t)bits),
                               cvt_rs_bf16x2(v.z, v.w, (uint32_t)(bits >> 32)));
    reinterpret_cast<uint2*>(static_cast<uint16_t*>(base) + row * d)[q] = u;
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xFFFF0000u),
                       __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xFFFF0000u));
  }
};

__device__ __forceinline__ float4 add4(float4 a, float4 b) {
  return make_float4(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z),
                     __fadd_rn(a.w, b.w));
}
__device__ __forceinline__ float4 fma4s(float s, float4 x, float4 acc) {
  return make_float4(__fmaf_rn(s, x.x, acc.x), __fmaf_rn(s, x.y, acc.y), __fmaf_rn(s, x.z, acc.z),
                     __fmaf_rn(s, x.w, acc.w));
}

// ---- LCG jumps ---------------------------------------------------------------------
struct SmallJumps {
  uint64_t mul[33], add[33];
};
__device__ __forceinline__ uint64_t jump_small(uint64_t r, int k, const SmallJumps& j) {
  return j.mul[k] * r + j.add[k];
}
__device__ __forceinline__ uint64_t jump_any(uint64_t r, uint64_t n, const LcgJumps* J) {
  for (int i = 0; n; i++, n >>= 1)
    if (n & 1) r = __ldg(&J->pow2_mul[i]) * r + __ldg(&J->pow2_add[i]);
  return r;
}

// ---- learning rate (dsgl.hpp:886-897) ----------------------------------------------
__device__ __forceinline__ float alpha_update(const TrainParams& p, unsigned long long wca_now) {
  float a = __fmul_rn(p.start_alpha,
                      __fsub_rn(1.0f, __fdiv_rn(__ull2float_rn(wca_now), p.alpha_denom)));
  float floor_a = __fmul_rn(p.start_alpha, 0.0001f);
  return a < floor_a ? floor_a : a;
}

// ---- walk fill with subsampling (dsgl.hpp:909-933), one warp ------------------------
// Reads tokens from cur until a -1, the slice end (whose last token is consumed and
// dropped, as the reference does) or kMaxSentence kept tokens.  Kept rows go to sen[].
// Returns the kept length; cur, word_count and rng advance exactly as the reference's.
// cap: capacity of sen (>= the longest walk of the corpus, checked by the host); a
// longer walk sets the kernel status to SGNS_EINVAL and is truncated.
__device__ __forceinline__ int fill_walk(const TrainParams& p, const SmallJumps& sj, int* sen,
                                         int64_t& cur, int64_t end, uint64_t& word_count,
                                         uint64_t& rng, int cap) {
  const int lane = lane_id();
  int L = 0;
  while (true) {
    const int64_t q = cur + lane;
    const bool in_range = q < end;
    const int tok = in_range ? __ldg(&p.corpus[q]) : -1;
    const unsigned stop = __ballot_sync(kFull, in_range && (tok == -1 || q == end - 1));
    const int first_stop = stop ? __ffs(stop) - 1 : 32;
    const bool valid = lane < first_stop;
    bool keep = valid;
    if (p.sample_on && valid) {
      uint64_t st = jump_small(rng, lane + 1, sj);
      float u = __fdiv_rn((float)(uint32_t)(st & 0xFFFF), 65536.0f);
      keep = !(__ldg(&p.ran[tok]) < u);
    }
    const unsigned keep_mask = __ballot_sync(kFull, keep);
    const int nk = __popc(keep_mask);
    int consumed, draws;
    bool done;
    if (L + nk >= kMaxSentence) {
      const int cap_lane = nth_set_bit(keep_mask, kMaxSentence - L - 1);
      if (keep && lane <= cap_lane) {
        const int at = L + __popc(keep_mask & lanemask_lt());
        if (at < cap) sen[at] = tok;
      }
      L = kMaxSentence;
      consumed = cap_lane + 1;
      draws = p.sample_on ? cap_lane + 1 : 0;
      done = true;
    } else {
      if (keep) {
        const int at = L + __popc(keep_mask & lanemask_lt());
        if (at < cap) sen[at] = tok;
      }
      L += nk;
      if (first_stop < 32) {
        consumed = first_stop + 1;
        draws = p.sample_on ? first_stop : 0;
        done = true;
      } else {
        consumed = 32;
        draws = p.sample_on ? 32 : 0;
        done = false;
      }
    }
    cur += consumed;
    word_count += (uint64_t)consumed;
    rng = jump_small(rng, draws, sj);
    if (done) break;
  }
  if (L > cap) {
    if (lane == 0) atomicExch(&p.ctr->status, 1);
    L = cap;
  }
  __syncwarp();
  return L;
}

// ---- one group of negatives and the output list (dsgl.hpp:1136-1159) ---------------
// Draw k of the group starting at LCG state gstate is made by lane k: its state and
// the table entry it indexes (a global load that may be issued a step ahead).
struct NegDraw {
  uint64_t st;
  int raw;
};
__device__ __forceinline__ NegDraw neg_draw_issue(const TrainParams& p, const SmallJumps& sj, uint64_t gstate) {
  NegDraw n;
  n.st = 0;
  n.raw = 0;
  if (lane_id() < p.K) {
    n.st = jump_small(gstate, lane_id() + 1, sj);
    n.raw = __ldg(&p.table[fast_mod(n.st >> 16, p.div_table)]);
  }
  return n;
}
// Equal draws merge (meta = multiplicity, first occurrence keeps its place); draws equal
// to t1 are dropped.  Writes out_id/out_meta[0..O) and returns O.  The reference orders
// the outputs t1, negatives, t2; they are stored t1, t2, negatives, so that target 2 sits
// at a fixed index (a run-time index into register arrays would put them in local
// memory).  Every sum whose order matters walks them in the reference's order.
// t2_meta: multiplicity of target 2 (0 in single-window steps, where t2 is a placeholder
// whose coefficients are zero and whose row is not written)
__device__ __forceinline__ int select_outputs(const TrainParams& p, NegDraw nd, int t1, int t2, int* out_id,
                                              int* out_meta, int t2_meta = 1) {
  const int lane = lane_id();
  const bool valid = lane < p.K;
  int s = -2 - lane;
  if (valid) s = nd.raw ? nd.raw : (int)(fast_mod(nd.st, p.div_vm1) + 1);
  const unsigned same = __match_any_sync(kFull, s);
  const bool leader = (__ffs(same) - 1) == lane;
  const unsigned distinct = __ballot_sync(kFull, valid && leader && s != t1);
  const int O = __popc(distinct) + 2;
  if (valid && leader && s != t1) {
    int idx = 2 + __popc(distinct & lanemask_lt());
    out_id[idx] = s;
    out_meta[idx] = __popc(same);
  }
  if (lane == 0) {
    out_id[0] = t1;
    out_meta[0] = 1;
    out_id[1] = t2;
    out_meta[1] = t2_meta;
  }
  __syncwarp();
  return O;
}

// Same output list from K stored draws words[0..K) (the reference's neg_words group);
// also returns, for each output i in 1..O-2, the index k of its first draw in kidx.
__device__ __forceinline__ int select_outputs_stored(int K, const int* words, int t1, int t2,
                                                     int* out_id, int* out_meta, int* kidx, int t2_meta = 1) {
  const int lane = lane_id();
  const bool valid = lane < K;
  const int s = valid ? words[lane] : -2 - lane;
  const unsigned same = __match_any_sync(kFull, s);
  const bool leader = (__ffs(same) - 1) == lane;
  const unsigned distinct = __ballot_sync(kFull, valid && leader && s != t1);
  const int O = __popc(distinct) + 2;
  if (valid && leader && s != t1) {
    int idx = 1 + __popc(distinct & lanemask_lt());
    out_id[idx] = s;
    out_meta[idx] = __popc(same);
    kidx[idx] = lane;
  }
  if (lane == 0) {
    out_id[0] = t1;
    out_meta[0] = 1;
    out_id[O - 1] = t2;
    out_meta[O - 1] = t2_meta;
  }
  __syncwarp();
  return O;
}

// ---- window input list (dsgl.hpp:1100-1132) ------------------------------------------
// Appends the positions c = pos - w + i, i in [b, 2w+1-b), i != w, 0 <= c < len in
// increasing order; slot_of(c) gives the row index stored in in_row.  Returns the count.
// kEveryLane: slot_of is called by all 32 lanes (it may be a warp shuffle) with any c,
// valid or not, and must be safe for every c; otherwise only for valid positions.
template <bool kEveryLane = false, class SlotOf>
__device__ __forceinline__ int window_inputs(int pos, int len, int w, int b, int base, int* in_row,
                                             SlotOf slot_of) {
  const int lane = lane_id();
  int n = 0;
  for (int i0 = 0; i0 < 2 * w + 1; i0 += 32) {
    const int i = i0 + lane;
    const int c = pos - w + i;
    const bool ok = i >= b && i < 2 * w + 1 - b && i != w && c >= 0 && c < len;
    const unsigned m = __ballot_sync(kFull, ok);
    if (kEveryLane) {
      const int sl = slot_of(c);
      if (ok) in_row[base + n + __popc(m & lanemask_lt())] = sl;
    } else {
      if (ok) in_row[base + n + __popc(m & lanemask_lt())] = slot_of(c);
    }
    n += __popc(m);
  }
  return n;
}

// ---- step arithmetic ---------------------------------------------------------------
// Packed fp32x2 arithmetic (Blackwell FFMA2/FADD2): each half is an ordinary IEEE
// operation, so pairing two independent sums changes no result.
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 fadd2(float2 a, float2 b) { return __fadd2_rn(a, b); }

// Output-row layout of one step for at most OM outputs (OM = K + 2):
//   normal rows:      out[i * DP + c]                          (backward, table updates)
//   interleaved rows: outI[(p * d + c) * 2 + b] = out_{2p+b}[c]   (forward; a float4
//                     holds the pair (2p, 2p+1) for two consecutive columns)
//   gradients:        corrP[j * CS + i] = {g_ij, g_ij}          (duplicated pairs)
template <int OM>
struct StepShape {
  static constexpr int OMP = (OM + 1) & ~1;  // outputs rounded up to pairs
  static constexpr int NPAIR = OMP / 2;
  static constexpr int CS = OMP + 2;        // corrP row stride in pairs (16-byte rows)
};

// Rows 2p and 2p+1, columns 4q..4q+3, read back from the interleaved layout.
__device__ __forceinline__ void out_chunk_pair(const float* outI, int d, int p, int q, float4& r0, float4& r1) {
  const float4* src = reinterpret_cast<const float4*>(outI + ((size_t)p * d + 4 * q) * 2);
  const float4 a = src[0], b = src[1];
  r0 = make_float4(a.x, a.z, b.x, b.z);
  r1 = make_float4(a.y, a.w, b.y, b.w);
}

// Forward: lane j computes f_ij for every output i, sequentially over k (pairs of
// outputs share one FFMA2), then the reference gradient g = (label - sigma_table(f)) *
// alpha * meta (dsgl.hpp:1243-1272).  Optional fp32 per-lane loss.
template <int OM, class InPtr>
__device__ __forceinline__ void forward_gradient(int I, int first, int O, int d, InPtr in_ptr,
                                                 const float* outI, const int* out_meta,
                                                 const float* exp_table, float alpha, float2* corrP,
                                                 bool want_loss, float& loss) {
  typedef StepShape<OM> SS;
  const int lane = lane_id();
  const int d4 = d >> 2;
  for (int j0 = 0; j0 < I; j0 += 32) {
    const int j = j0 + lane;
    const float4* x = reinterpret_cast<const float4*>(in_ptr(j < I ? j : I - 1));
    float2 f[SS::NPAIR];
#pragma unroll
    for (int q = 0; q < SS::NPAIR; q++) f[q] = make_float2(0.f, 0.f);
    for (int k4 = 0; k4 < d4; k4++) {
      const float4 xv = x[k4];
      const float2 x0 = make_float2(xv.x, xv.x), x1 = make_float2(xv.y, xv.y);
      const float2 x2 = make_float2(xv.z, xv.z), x3 = make_float2(xv.w, xv.w);
#pragma unroll
      for (int q = 0; q < SS::NPAIR; q++) {
        if (2 * q < O) {
          const float4* op = reinterpret_cast<const float4*>(outI + ((size_t)q * d + 4 * k4) * 2);
          const float4 a = op[0], b = op[1];
          f[q] = ffma2(make_float2(a.x, a.y), x0, f[q]);
          f[q] = ffma2(make_float2(a.z, a.w), x1, f[q]);
          f[q] = ffma2(make_float2(b.x, b.y), x2, f[q]);
          f[q] = ffma2(make_float2(b.z, b.w), x3, f[q]);
        }
      }
    }
    if (j < I) {
#pragma unroll
      for (int i = 0; i < OM; i++) {
        if (i < O) {
          const int label = j < first ? (i == 0) : (i == O - 1);
          const float fi = (i & 1) ? f[i >> 1].y : f[i >> 1].x;
          float g;
          if (fi > (float)kMaxExp) {
            g = __fmul_rn((float)(label - 1), alpha);
          } else if (fi < -(float)kMaxExp) {
            g = __fmul_rn((float)label, alpha);
          } else {
            const int idx =
                __float2int_rz(__fmul_rn(__fadd_rn(fi, (float)kMaxExp), (float)kTableScale));
            g = __fmul_rn(__fsub_rn((float)label, exp_table[idx]), alpha);
          }
          const float gm = __fmul_rn(g, (float)out_meta[i]);
          corrP[j * SS::CS + i] = make_float2(gm, gm);
          if (want_loss) {  // meta * softplus(-(2 label - 1) f) = -meta log sigma(+-f)
            const float z = label ? -fi : fi;
            loss += (float)out_meta[i] * (fmaxf(z, 0.f) + log1pf(__expf(-fabsf(z))));
          }
        }
      }
    }
  }
  __syncwarp();
}

// ---- the persistent engine's rows and step arithmetic ---------------------------------
// The persistent kernels keep a step's rows in shared memory in quarters: when d % 16 == 0,
// a row is four quarters of d / 4 columns, each followed by 4 words of padding, else d
// columns and 4 words.  Shared memory returns 128 bytes per cycle to the registers of an SM
// whatever the lanes' addresses, and that, not FMA issue, bounded these kernels, so the
// layout serves the forward's register tiles: lanes that hold the four quarters of a row
// and two neighbouring rows read 8 distinct 16-byte bank groups (the row stride is 4 groups
// modulo 8).
struct RowShape {
  int stride;  // words from row to row
  int q4;      // 4-column chunks per quarter (d % 16 == 0), else d / 4: one range
};
__host__ __device__ __forceinline__ RowShape row_shape(int d) {
  return (d & 15) == 0 ? RowShape{d + 16, d >> 4} : RowShape{d + 4, d >> 2};
}
// word offset of chunk q's 4 columns in a row
__device__ __forceinline__ int chunk_at(int q, const RowShape& R) { return 4 * (q + q / R.q4); }

// The reference's gradient of one dot product (dsgl.hpp:1243-1272), without branches: past
// +-6 the sigmoid is 1 or 0, and label - 1, label - 0 are exact.
__device__ __forceinline__ float step_gradient(float f, int label, const float* exp_table, float alpha, int meta) {
  const int idx = __float2int_rz(__fmul_rn(__fadd_rn(f, (float)kMaxExp), (float)kTableScale));
  float sig = exp_table[min(max(idx, 0), kExpTableSize)];
  sig = f > (float)kMaxExp ? 1.f : f < -(float)kMaxExp ? 0.f : sig;
  return __fmul_rn(__fmul_rn(__fsub_rn((float)label, sig), alpha), (float)meta);
}
__device__ __forceinline__ float step_loss(float f, int label, int meta) {
  const float z = label ? -f : f;
  return (float)meta * (fmaxf(z, 0.f) + log1pf(__expf(-fabsf(z))));
}

// Forward of one warp's step: every dot product is eight sequential partial sums -- the even
// and the odd k of each quarter of [0, d), each pair advanced by one FFMA2 on
// {o[k], o[k+1]} x {x[k], x[k+1]} -- combined as s_m = even_m + odd_m,
// f = (s_0 + s_1) + (s_2 + s_3) when d % 16 == 0; when not, [0, d) is one range and
// f = even + odd.  The oracle's window policy uses the same order.
// Register tiles: with quarters, lane = m + 4 og + 8 ig holds quarter m of TI inputs
// (j0 + ig + 4 t) against the outputs of parity og, so a chunk of TI + TO rows read feeds
// TI TO products (against 8 reads for 7 with one lane per input and the outputs broadcast);
// the quarters' sums meet by shuffles, (s_0 + s_1) first, each lane keeping a part.  One
// range: lane = og + 2 ig, two inputs each.
// corr[j * CS + i] = g_ij, CS = OM rounded up to 4.
template <int OM, int DFIX, class InPtr>
__device__ __forceinline__ void forward_tiled(int I, int first, int O, int d_rt, InPtr in_ptr, const float* out_rows,
                                              const int* out_meta, const float* exp_table, float alpha, float* corr,
                                              bool want_loss, float& loss) {
  constexpr int CS = (OM + 3) & ~3, TO = (OM + 1) / 2;
  const int d = DFIX ? DFIX : d_rt;
  const RowShape R = row_shape(d);
  const int lane = lane_id();
  auto finish = [&](int j, int i, float f) {
    if (j < I && i < O) {
      const int label = j < first ? (i == 0) : (i == 1);  // outputs t1, t2, negatives
      corr[j * CS + i] = step_gradient(f, label, exp_table, alpha, out_meta[i]);
      if (want_loss) loss += step_loss(f, label, out_meta[i]);
    }
  };
  if ((d & 15) == 0) {
    constexpr int TI = 4;
    const int m = lane & 3, og = (lane >> 2) & 1, ig = lane >> 3;
    const int q4 = R.q4, at = 4 * m * (q4 + 1);  // the quarter's first word
    // output rows og, og + 2, ..; one past OM is read as the first (an unused sum)
    const float* o0 = out_rows + og * R.stride + at;
    const int last = 2 * (TO - 1) + og < OM ? 2 * (TO - 1) * R.stride : 0;
    for (int j0 = 0; j0 < I; j0 += 4 * TI) {
      const float4* x[TI];
#pragma unroll
      for (int t = 0; t < TI; t++) {
        const int j = j0 + ig + 4 * t;
        x[t] = reinterpret_cast<const float4*>(in_ptr(j < I ? j : I - 1) + at);
      }
      float2 f[TI][TO];
#pragma unroll
      for (int t = 0; t < TI; t++)
#pragma unroll
        for (int u = 0; u < TO; u++) f[t][u] = make_float2(0.f, 0.f);
#pragma unroll 2
      for (int k4 = 0; k4 < q4; k4++) {
        float4 xv[TI], ov[TO];  // rows past O hold stale data: unused sums
#pragma unroll
        for (int t = 0; t < TI; t++) xv[t] = x[t][k4];
#pragma unroll
        for (int u = 0; u < TO; u++)
          ov[u] = reinterpret_cast<const float4*>(o0 + (u < TO - 1 ? 2 * u * R.stride : last))[k4];
#pragma unroll
        for (int t = 0; t < TI; t++)
#pragma unroll
          for (int u = 0; u < TO; u++)
            f[t][u] = ffma2(make_float2(ov[u].x, ov[u].y), make_float2(xv[t].x, xv[t].y), f[t][u]);
#pragma unroll
        for (int t = 0; t < TI; t++)
#pragma unroll
          for (int u = 0; u < TO; u++)
            f[t][u] = ffma2(make_float2(ov[u].z, ov[u].w), make_float2(xv[t].z, xv[t].w), f[t][u]);
      }
      // quarters (0, 1) and (2, 3) meet: lanes of even m keep inputs t = 0, 1, of odd m 2, 3;
      // then the two halves: m < 2 keeps the first of its two inputs, m >= 2 the second
      float s[2][TO];
#pragma unroll
      for (int t = 0; t < 2; t++)
#pragma unroll
        for (int u = 0; u < TO; u++) {
          const float a = __fadd_rn(f[t][u].x, f[t][u].y), b = __fadd_rn(f[t + 2][u].x, f[t + 2][u].y);
          const float got = __shfl_xor_sync(kFull, (m & 1) ? a : b, 1);
          s[t][u] = __fadd_rn((m & 1) ? b : a, got);
        }
      const int j = j0 + ig + 4 * (2 * (m & 1) + (m >> 1));
#pragma unroll
      for (int u = 0; u < TO; u++) {
        const float got = __shfl_xor_sync(kFull, (m & 2) ? s[0][u] : s[1][u], 2);
        finish(j, 2 * u + og, __fadd_rn((m & 2) ? s[1][u] : s[0][u], got));
      }
    }
  } else {
    constexpr int TI = 2;
    const int og = lane & 1, ig = lane >> 1;
    const float* o0 = out_rows + og * R.stride;
    const int last = 2 * (TO - 1) + og < OM ? 2 * (TO - 1) * R.stride : 0;
    for (int j0 = 0; j0 < I; j0 += 16 * TI) {
      const float4* x[TI];
#pragma unroll
      for (int t = 0; t < TI; t++) {
        const int j = j0 + ig + 16 * t;
        x[t] = reinterpret_cast<const float4*>(in_ptr(j < I ? j : I - 1));
      }
      float2 f[TI][TO];
#pragma unroll
      for (int t = 0; t < TI; t++)
#pragma unroll
        for (int u = 0; u < TO; u++) f[t][u] = make_float2(0.f, 0.f);
#pragma unroll 2
      for (int k4 = 0; k4 < R.q4; k4++) {
        float4 xv[TI], ov[TO];
#pragma unroll
        for (int t = 0; t < TI; t++) xv[t] = x[t][k4];
#pragma unroll
        for (int u = 0; u < TO; u++)
          ov[u] = reinterpret_cast<const float4*>(o0 + (u < TO - 1 ? 2 * u * R.stride : last))[k4];
#pragma unroll
        for (int t = 0; t < TI; t++)
#pragma unroll
          for (int u = 0; u < TO; u++) {
            f[t][u] = ffma2(make_float2(ov[u].x, ov[u].y), make_float2(xv[t].x, xv[t].y), f[t][u]);
            f[t][u] = ffma2(make_float2(ov[u].z, ov[u].w), make_float2(xv[t].z, xv[t].w), f[t][u]);
          }
      }
#pragma unroll
      for (int t = 0; t < TI; t++)
#pragma unroll
        for (int u = 0; u < TO; u++)
          // the sum's three empty partners of the eight-sum form
          finish(j0 + ig + 16 * t, 2 * u + og, __fadd_rn(__fadd_rn(__fadd_rn(f[t][u].x, f[t][u].y), 0.f), 0.f));
    }
  }
  __syncwarp();
}

// Backward.  Lane owns column chunks q = lane + 32 t (t < DCH, q < d/4), as two pairs.
//   md[i][t]  = sum_j corr[i][j] * in_j[q]     (outputMd, dsgl.hpp:1290), sequential j
//   in_j[q]  += sum_i corr[i][j] * out_i[q]     (inputM then buffer +=, dsgl.hpp:1309-1333),
//               sequential i, inputs applied in order j = 0..I-1.
// md is complete before any input row changes, as the reference's two GEMMs read the
// same pre-update inputM.  apply_in(j, q, a) consumes input j's update of chunk q.
// out_pair(p, q, r0, r1): rows 2p and 2p+1 of the step's outputs, columns 4q..4q+3.
template <int OM, int DCH, class InPtr, class OutPair, class ApplyIn>
__device__ __forceinline__ void backward(int I, int O, int d, InPtr in_ptr, OutPair out_pair,
                                         const float2* corrP, float4 (&md)[OM][DCH], ApplyIn apply_in) {
  typedef StepShape<OM> SS;
  const int lane = lane_id();
  const int d4 = d >> 2;
  float2 mlo[OM][DCH], mhi[OM][DCH];
#pragma unroll
  for (int i = 0; i < OM; i++)
#pragma unroll
    for (int t = 0; t < DCH; t++) mlo[i][t] = mhi[i][t] = make_float2(0.f, 0.f);
  // the next input's row address is fetched one iteration ahead, off the dependency chain
  const float4* x_next = I > 0 ? reinterpret_cast<const float4*>(in_ptr(0)) : nullptr;
  for (int j = 0; j < I; j++) {
    const float4* x = x_next;
    x_next = reinterpret_cast<const float4*>(in_ptr(j + 1 < I ? j + 1 : j));
    const float4* cj = reinterpret_cast<const float4*>(corrP + j * SS::CS);
    float2 c[SS::OMP];
#pragma unroll
    for (int q = 0; q < SS::NPAIR; q++) {
      const float4 v = cj[q];
      c[2 * q] = make_float2(v.x, v.y);
      c[2 * q + 1] = make_float2(v.z, v.w);
    }
#pragma unroll
    for (int t = 0; t < DCH; t++) {
      const int q = lane + 32 * t;
      if (q < d4) {
        const float4 xv = x[q];
        const float2 xl = make_float2(xv.x, xv.y), xh = make_float2(xv.z, xv.w);
#pragma unroll
        for (int i = 0; i < OM; i++)
          if (i < O) {
            mlo[i][t] = ffma2(c[i], xl, mlo[i][t]);
            mhi[i][t] = ffma2(c[i], xh, mhi[i][t]);
          }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < OM; i++)
#pragma unroll
    for (int t = 0; t < DCH; t++) md[i][t] = make_float4(mlo[i][t].x, mlo[i][t].y, mhi[i][t].x, mhi[i][t].y);
  float2 olo[SS::OMP][DCH], ohi[SS::OMP][DCH];
#pragma unroll
  for (int pp = 0; pp < SS::NPAIR; pp++)
#pragma unroll
    for (int t = 0; t < DCH; t++) {
      const int q = lane + 32 * t;
      float4 r0 = make_float4(0.f, 0.f, 0.f, 0.f), r1 = r0;
      if (2 * pp < O && q < d4) out_pair(pp, q, r0, r1);
      olo[2 * pp][t] = make_float2(r0.x, r0.y);
      ohi[2 * pp][t] = make_float2(r0.z, r0.w);
      olo[2 * pp + 1][t] = make_float2(r1.x, r1.y);
      ohi[2 * pp + 1][t] = make_float2(r1.z, r1.w);
    }
  // four inputs per iteration: eight independent chains; updates applied in input order
  for (int j0 = 0; j0 < I; j0 += 4) {
    float2 c[4][SS::OMP];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int j = j0 + u < I ? j0 + u : I - 1;
      const float4* cj = reinterpret_cast<const float4*>(corrP + j * SS::CS);
#pragma unroll
      for (int q = 0; q < SS::NPAIR; q++) {
        const float4 v = cj[q];
        c[u][2 * q] = make_float2(v.x, v.y);
        c[u][2 * q + 1] = make_float2(v.z, v.w);
      }
    }
#pragma unroll
    for (int t = 0; t < DCH; t++) {
      const int q = lane + 32 * t;
      if (q < d4) {
        float2 al[4], ah[4];
#pragma unroll
        for (int u = 0; u < 4; u++) al[u] = ah[u] = make_float2(0.f, 0.f);
#pragma unroll
        for (int i = 0; i < OM; i++) {
          if (i < O) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
              al[u] = ffma2(c[u][i], olo[i][t], al[u]);
              ah[u] = ffma2(c[u][i], ohi[i][t], ah[u]);
            }
          }
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (j0 + u < I) apply_in(j0 + u, q, make_float4(al[u].x, al[u].y, ah[u].x, ah[u].y));
      }
    }
  }
  __syncwarp();
}

// Backward of the persistent kernels.  A lane owns NC pairs of columns of every row: one pair
// (2 columns), a chunk of 4, or two chunks `step` words apart.
//   m_i  = sum_j g_ij x_j     (outputMd, dsgl.hpp:1290), sequential in j
//   x_j += sum_i g_ij o_i     (dsgl.hpp:1309-1333), in the reference's order t1, negatives, t2
//                             (stored rows 0, 2 .. O-1, 1)
// outputMd is summed over rows no input has changed yet: in one pass when no two inputs share
// a row (an input's row is read for outputMd, then updated), else before any update.
template <int NC>
__device__ __forceinline__ void load_cols(const float* p, int step, float2 (&v)[NC]) {
  if constexpr (NC == 1) {
    v[0] = *reinterpret_cast<const float2*>(p);
  } else {
#pragma unroll
    for (int k = 0; k < NC / 2; k++) {
      const float4 t = *reinterpret_cast<const float4*>(p + k * step);
      v[2 * k] = make_float2(t.x, t.y), v[2 * k + 1] = make_float2(t.z, t.w);
    }
  }
}
template <int NC>
__device__ __forceinline__ void store_cols(float* p, int step, const float2 (&v)[NC]) {
  if constexpr (NC == 1) {
    *reinterpret_cast<float2*>(p) = v[0];
  } else {
#pragma unroll
    for (int k = 0; k < NC / 2; k++)
      *reinterpret_cast<float4*>(p + k * step) = make_float4(v[2 * k].x, v[2 * k].y, v[2 * k + 1].x, v[2 * k + 1].y);
  }
}
// gradients of input j for N outputs from i0 (a multiple of 2; of 4 when N > 2)
template <int OM, int N>
__device__ __forceinline__ void load_coef(const float* corr, int j, int i0, float (&c)[N]) {
  constexpr int CS = (OM + 3) & ~3;
  const float* cj = corr + j * CS + i0;
  if constexpr (N % 4 == 2) {  // i0 may be 2 past a multiple of 4
#pragma unroll
    for (int k = 0; k < N / 2; k++) {
      const float2 v = reinterpret_cast<const float2*>(cj)[k];
      c[2 * k] = v.x, c[2 * k + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < (N + 3) / 4; k++) {
      const float4 v = reinterpret_cast<const float4*>(cj)[k];
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int t = 0; t < 4; t++)
        if (4 * k + t < N) c[4 * k + t] = e[t];
    }
  }
}
template <int N, int NC>
__device__ __forceinline__ void accumulate_out(const float (&c)[N], const float2 (&x)[NC], float2 (&m)[N][NC]) {
#pragma unroll
  for (int i = 0; i < N; i++)
#pragma unroll
    for (int t = 0; t < NC; t++) m[i][t] = ffma2(make_float2(c[i], c[i]), x[t], m[i][t]);
}
// an input's addend, sum_i g_ij o_i in the reference's order.  kAll: O == OM
template <int OM, int NC, bool kAll>
__device__ __forceinline__ void input_addend(const float (&c)[OM], const float2 (&o)[OM][NC], int O, float2 (&a)[NC]) {
#pragma unroll
  for (int t = 0; t < NC; t++) a[t] = ffma2(make_float2(c[0], c[0]), o[0][t], make_float2(0.f, 0.f));
#pragma unroll
  for (int i = 2; i < OM; i++)
    if (kAll || i < O) {
#pragma unroll
      for (int t = 0; t < NC; t++) a[t] = ffma2(make_float2(c[i], c[i]), o[i][t], a[t]);
    }
#pragma unroll
  for (int t = 0; t < NC; t++) a[t] = ffma2(make_float2(c[1], c[1]), o[1][t], a[t]);
}
template <int OM, int NC, bool kAll>
__device__ __forceinline__ void update_input(const float (&c)[OM], const float2 (&o)[OM][NC], int O, float2 (&x)[NC]) {
  float2 a[NC];
  input_addend<OM, NC, kAll>(c, o, O, a);
#pragma unroll
  for (int t = 0; t < NC; t++) x[t] = fadd2(x[t], a[t]);
}
// outputMd of N outputs from i0 over all inputs; x: the rows at the lane's columns
template <int OM, int N, int NC>
__device__ __forceinline__ void step_out_md(int I, const float* x, int step, const int* in_off, const float* corr, int i0,
                                            float2 (&m)[N][NC]) {
  int j = 0;
  for (; j + 4 <= I; j += 4) {
    const int4 off = *reinterpret_cast<const int4*>(in_off + j);
    float2 xv[4][NC];
    float c[4][N];
    load_cols<NC>(x + off.x, step, xv[0]);
    load_cols<NC>(x + off.y, step, xv[1]);
    load_cols<NC>(x + off.z, step, xv[2]);
    load_cols<NC>(x + off.w, step, xv[3]);
#pragma unroll
    for (int u = 0; u < 4; u++) load_coef<OM, N>(corr, j + u, i0, c[u]);
#pragma unroll
    for (int u = 0; u < 4; u++) accumulate_out<N, NC>(c[u], xv[u], m);
  }
  for (; j < I; j++) {
    float2 xv[NC];
    float c[N];
    load_cols<NC>(x + in_off[j], step, xv);
    load_coef<OM, N>(corr, j, i0, c);
    accumulate_out<N, NC>(c, xv, m);
  }
}
// updates of inputs [j0, j1), in order
template <int OM, int NC, bool kAll>
__device__ __forceinline__ void step_update(int j0, int j1, int O, bool distinct, float* x, int step, const int* in_off,
                                            const float* corr, const float2 (&o)[OM][NC]) {
  int j = j0;
  if (__builtin_expect(distinct, 1)) {
    for (; j + 2 <= j1; j += 2) {
      float *xa = x + in_off[j], *xb = x + in_off[j + 1];
      float2 va[NC], vb[NC];
      float ca[OM], cb[OM];
      load_cols<NC>(xa, step, va);
      load_cols<NC>(xb, step, vb);
      load_coef<OM, OM>(corr, j, 0, ca);
      load_coef<OM, OM>(corr, j + 1, 0, cb);
      update_input<OM, NC, kAll>(ca, o, O, va);
      update_input<OM, NC, kAll>(cb, o, O, vb);
      store_cols<NC>(xa, step, va);
      store_cols<NC>(xb, step, vb);
    }
  }
  for (; j < j1; j++) {
    float* xa = x + in_off[j];
    float2 va[NC];
    float ca[OM];
    load_cols<NC>(xa, step, va);
    load_coef<OM, OM>(corr, j, 0, ca);
    update_input<OM, NC, kAll>(ca, o, O, va);
    store_cols<NC>(xa, step, va);
  }
}
// both products over all inputs, for steps without shared rows
template <int OM, int NC, bool kAll>
__device__ __forceinline__ void step_merged(int I, int O, float* x, int step, const int* in_off, const float* corr,
                                            const float2 (&o)[OM][NC], float2 (&m)[OM][NC]) {
  int j = 0;
  for (; j + 2 <= I; j += 2) {
    const int2 off = *reinterpret_cast<const int2*>(in_off + j);
    float2 va[NC], vb[NC];
    float ca[OM], cb[OM];
    load_cols<NC>(x + off.x, step, va);
    load_cols<NC>(x + off.y, step, vb);
    load_coef<OM, OM>(corr, j, 0, ca);
    load_coef<OM, OM>(corr, j + 1, 0, cb);
    accumulate_out<OM, NC>(ca, va, m);
    update_input<OM, NC, kAll>(ca, o, O, va);
    store_cols<NC>(x + off.x, step, va);
    accumulate_out<OM, NC>(cb, vb, m);
    update_input<OM, NC, kAll>(cb, o, O, vb);
    store_cols<NC>(x + off.y, step, vb);
  }
  if (j < I) {
    float* xa = x + in_off[j];
    float2 va[NC];
    float ca[OM];
    load_cols<NC>(xa, step, va);
    load_coef<OM, OM>(corr, j, 0, ca);
    accumulate_out<OM, NC>(ca, va, m);
    update_input<OM, NC, kAll>(ca, o, O, va);
    store_cols<NC>(xa, step, va);
  }
}

// Stores the step's output rows from registers in the interleaved layout (see StepShape).
template <int OM, int DCH>
__device__ __forceinline__ void store_out_interleaved(const float4 (&v)[OM][DCH], int O, int d, float* outI) {
  typedef StepShape<OM> SS;
  const int lane = lane_id(), d4 = d >> 2;
#pragma unroll
  for (int t = 0; t < DCH; t++) {
    const int q = lane + 32 * t;
    if (q < d4) {
#pragma unroll
      for (int p = 0; p < SS::NPAIR; p++) {
        if (2 * p < O) {
          const float4 a = v[2 * p][t];
          const float4 b = (2 * p + 1 < OM && 2 * p + 1 < O) ? v[(2 * p + 1) < OM ? 2 * p + 1 : 0][t]
                                                            : make_float4(0.f, 0.f, 0.f, 0.f);
          float4* dst = reinterpret_cast<float4*>(outI + ((size_t)p * d + 4 * q) * 2);
          dst[0] = make_float4(a.x, b.x, a.y, b.y);
          dst[1] = make_float4(a.z, b.z, a.w, b.w);
        }
      }
    }
  }
}

// trainers: buffered input row += update
template <class InPtr>
struct AddToInput {
  InPtr in_ptr;
  __device__ __forceinline__ void operator()(int j, int q, float4 a) const {
    float4* x = reinterpret_cast<float4*>(const_cast<float*>(in_ptr(j)));
    const float4 v = x[q];
    const float2 lo = fadd2(make_float2(v.x, v.y), make_float2(a.x, a.y));
    const float2 hi = fadd2(make_float2(v.z, v.w), make_float2(a.z, a.w));
    x[q] = make_float4(lo.x, lo.y, hi.x, hi.y);
  }
};
template <class InPtr>
__device__ __forceinline__ AddToInput<InPtr> add_to_input(InPtr f) {
  return AddToInput<InPtr>{f};
}

}  // namespace sgns
