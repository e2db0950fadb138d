// dsgl_team.cuh -- the persistent DSGL engine with a team of warps per worker.
//
// A worker (one compute thread of the reference's Train_SGNS_MPI, include/dsgl.hpp:
// 783-1425) is a serial chain of steps: at the worker counts that keep link-prediction
// quality (at most V / 400) few of them fit a GPU, and one warp per worker (dsgl_window.cu)
// leaves each SM with one or two dependent instruction streams.  Here four compute warps and
// one planner warp train a worker:
//
//   * The planner runs one step ahead.  Everything that does not depend on table values --
//     walk fill and subsampling, the learning rate, negative draws and the output list,
//     the shrink draw and the input list, which rows enter and leave the windows -- is
//     written to a step descriptor in shared memory (three of them in turn).  It also
//     prefetches the rows the step will read into L2.
//   * Compute warp (h, g) owns, in the h-th half of every row's columns, the output rows of
//     group g and the window rows of walk g.  A row part is loaded, updated and stored by its
//     owner, so most table accesses are ordered by one warp's program order; the step's
//     barriers order the rest (an output row may change its group from step to step), and the
//     planner marks the steps where two walks meet in a vertex.
//   * Table rows are read past the L1 (load_l2): few teams leave an SM most of its L1, and a
//     row that other workers have changed since would be read, and written back, as it was.
//     100k vertices, 250 workers: link-prediction AUC 0.7758 -> 0.7771 (bf16), 0.7777 -> 0.7786
//     (fp32), in the same time.
//   * The forward's dot products are summed by halves of the row (the quarters' sums
//     s0 + s1 and s2 + s3), in register tiles as in forward_tiled.
//
// Per step, barriers among the compute warps: (A) rows complete; (M) half sums exchanged;
// (U) outputMd done, input rows may change; and (B), with the planner: gradients complete,
// next descriptor written.
//
// Measured (GB300, kernel time of one training pass, against one warp per worker before and
// now): 100k vertices, 250 workers, d = 128, bf16: 112.5 ms -> 52.4 (one warp: 98.2); 120k
// vertices, 300 workers, d = 256, K = 10, fp32: 52.7 -> 14.3 (25.4); one replayed worker, d =
// 100: 50.9 -> 21.6 (41.2).  A step of a worker alone on its SM takes 6,100 cycles (d = 128,
// w = 10, bf16), of two 7,150, of three 10,100; with the clock read between its parts (7,050
// alone) the forward takes 1,930 of them, outputMd and the stores 2,140, the updates 820, the
// wait for the planner 690, window moves and the other barriers the rest.  160 threads of 128
// registers: an SM holds three teams, and while it gets no more workers a team is the faster
// (timings at shape_for_wpc in sgns_host.cpp); beyond, some would wait for others to end.
//
// Every sum has the operands and the order of window_engine_kernel (eight partial sums per
// dot product when d % 16 == 0, else two; outputMd sequential over the inputs; an input's
// update over the outputs t1, negatives, t2), and a worker's table accesses keep their
// order, so one worker reproduces the oracle's window policy bit for bit.
#pragma once
#include <cuda_runtime.h>

#include "dsgl_device.cuh"

namespace sgns {

struct TeamCall {  // what a dispatch ends in: an occupancy query (ctas) or a launch
  const TrainParams* p;
  int wpc;
  size_t smem;
  int* ctas;
  cudaStream_t s;
};
template <int S, int OM>
cudaError_t team_d(int d, const TeamCall& c);

namespace {

constexpr int kHdrWords = 1004 + 132;  // sigmoid table (1001 -> 1004) + SmallJumps (528 B)
constexpr int kRing = 32;              // position -> slot ring, one entry per planner lane
constexpr int kDescs = 3;              // the planner writes n + 1 while n - 1 and n are read
constexpr int kCompute = 4;            // compute warps per worker

// Step descriptor, in words.
enum {
  D_FLAGS = 0, D_I = 1, D_FIRST = 2, D_O = 3,
  D_ALPHA = 4, D_NPRE = 5,
  D_LIVE = 6,      // per walk: mask of the slots written back because the walk ended
  D_KEYS = 8,      // 5 x uint64 stochastic-rounding event keys, by event kind
  D_MOVE = 20,     // per walk: entering row's vertex (-1: none) and offset, leaving row's
  D_OUT = 28,      // kOMax output rows
  D_META = 40,     // kOMax multiplicities
  D_IN = 52        // 4 w input row offsets (words), then the lists below
};
// STOP: no step.  ALIAS: target 2 is also another output.  SERIAL: walk 0's moves before
// walk 1's.
enum { F_STOP = 1, F_ALIAS = 2, F_SERIAL = 4 };

struct TeamLayout {  // shared memory of one worker, in 4-byte words
  int NS, DP, CS, lmax, rows, out, corr, sen, desc, desc_words, pre, flush, words;
};

__host__ __device__ inline TeamLayout team_layout(int d, int w, int om, int lmax) {
  TeamLayout L;
  L.NS = 2 * w + 1;  // resident rows per walk (an entering row may take the leaving one's slot)
  L.DP = row_shape(d).stride;
  L.CS = (om + 3) & ~3;  // a gradient row
  L.lmax = lmax;
  int off = 0;
  L.rows = off;
  off += 2 * L.NS * L.DP;
  L.out = off;
  off += om * L.DP;
  L.corr = off;
  off += 4 * w * L.CS;
  L.desc = off;
  int dw = D_IN + 4 * w;
  L.pre = dw;
  dw += 2 * 2 * (w + 1);
  L.flush = dw;  // vertex of each slot of each walk
  dw += 2 * L.NS;
  L.desc_words = (dw + 3) & ~3;
  off += kDescs * L.desc_words;
  L.sen = off;
  off += 2 * lmax;
  L.words = (off + 3) & ~3;
  return L;
}

__device__ __forceinline__ void team_barrier(int id, int threads) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Lines of a row of `bytes` bytes into L2 (a hint: it changes no value and no order).
__device__ __forceinline__ void prefetch_row(const void* tab, int64_t row, int bytes) {
  const char* p = static_cast<const char*>(tab) + row * bytes;
  for (int o = 0; o < bytes; o += 128) prefetch_l2(p + o);
}

// ---- the planner ------------------------------------------------------------------------
template <int S>
__device__ __forceinline__ void plan_worker(const TrainParams& p, const SmallJumps& sj, const TeamLayout& L, float* base,
                                            int wid, int bar_b, int bar_b_threads) {
  const int lane = lane_id();
  const int w = p.window, K = p.K, NS = L.NS, DP = L.DP, lmax = L.lmax;
  const int row_bytes = p.d * RowIO<S>::kBytes;
  int* sen = reinterpret_cast<int*>(base + L.sen);
  // dsgl.hpp:790-826
  uint64_t rng = (uint64_t)wid, word_count = 0, last_wc = 0, step_id = 0;
  const uint64_t words_num = (uint64_t)p.words_num, parts = (uint64_t)p.workers;
  uint64_t tw = words_num / parts;
  const int64_t start = (int64_t)(tw * (uint64_t)wid);
  if (words_num % parts > 0 && (uint64_t)wid == parts - 1) tw = words_num - (parts - 1) * tw;
  const int64_t end = start + (int64_t)tw;
  int64_t cur = start;
  int local_iter = p.iter;
  int len[2] = {0, 0}, pos[2] = {0, 0};
  int train_sen_num = 0, neg_count = 0, neg_n = 1, neg_g = 0, grp_g = -1;
  bool change_neg = true;
  uint64_t pool_base = 0, grp_state = 0;
  // lane k counts: 0 pairs, 1 steps, 2 output rows, 3 row loads, 4 row stores
  unsigned long long count = 0;
  NegDraw pf{};
  int pf_g = -1;
  uint64_t pf_gs = 0;
  // window slots, lane s: vertex and position count of slot s; lane p & 31: slot of position p
  int sv0 = 0, sv1 = 0, sr0 = 0, sr1 = 0, rg0 = 0, rg1 = 0;
  auto enter = [&](int walk, int position, bool* fresh_out, int* v_out) -> int {
    const int v = sen[walk * lmax + position];
    const int my_v = walk ? sv1 : sv0, my_r = walk ? sr1 : sr0;
    const unsigned hit = __ballot_sync(kFull, lane < NS && my_r > 0 && my_v == v);
    int s;
    bool fresh = false;
    if (hit) {
      s = __ffs(hit) - 1;
    } else {
      const unsigned fr = __ballot_sync(kFull, lane < NS && my_r == 0);
      s = __ffs(fr) - 1;
      fresh = true;
      if (s < 0) {  // cannot happen: a first window holds at most w + 1 rows
        if (lane == 0) atomicExch(&p.ctr->status, 2);
        s = 0;
      }
    }
    if (lane == s) {
      if (walk) { sv1 = v; sr1 = my_r + 1; } else { sv0 = v; sr0 = my_r + 1; }
    }
    if (lane == (position & (kRing - 1))) {
      if (walk) rg1 = s; else rg0 = s;
    }
    *fresh_out = fresh;
    *v_out = v;
    return s;
  };

  int buf = 0;
  while (true) {
    int* D = reinterpret_cast<int*>(base + L.desc) + buf * L.desc_words;
    int n_pre = 0;
    bool stop = false;
    while (true) {  // until a step is ready or the passes are done
      if (__builtin_expect(word_count - last_wc > 10000, 0)) {  // dsgl.hpp:886-897
        const uint64_t diff = word_count - last_wc;
        if (lane == 0) {
          unsigned long long now = atomicAdd(&p.ctr->wca, (unsigned long long)diff) + diff;
          *reinterpret_cast<volatile float*>(&p.ctr->alpha) = alpha_update(p, now);
        }
        last_wc = word_count;
        __syncwarp();
      }
      if (__builtin_expect(len[0] == 0 || len[1] == 0, 0))
#pragma unroll
        for (int walk = 0; walk < 2; walk++) {  // dsgl.hpp:902-1030
          while (len[walk] == 0) {
            if (cur >= end) break;
            const int n = fill_walk(p, sj, sen + walk * lmax, cur, end, word_count, rng, lmax);
            if (n <= 1) continue;
            len[walk] = n;
            pos[walk] = 0;
            const int hi = n - 1 < w ? n - 1 : w;  // the first window: rows to load
            for (int q = 0; q <= hi; q++) {
              bool fresh;
              int v;
              const int s = enter(walk, q, &fresh, &v);
              if (fresh) {
                if (lane == 0) {
                  D[L.pre + 2 * n_pre] = v;
                  D[L.pre + 2 * n_pre + 1] = (walk * NS + s) * DP;
                  prefetch_row(p.wih, v, row_bytes);
                }
                n_pre++;
              }
            }
          }
        }
      if (__builtin_expect(cur >= end, 0)) {  // dsgl.hpp:1031-1050: walks in flight are dropped
        if (lane == 0) atomicAdd(&p.ctr->wca, (unsigned long long)(word_count - last_wc));
        if (lane == 3) count += (unsigned long long)n_pre;
        n_pre = 0;
        if (--local_iter == 0) {
          stop = true;
          break;
        }
        word_count = 0;
        last_wc = 0;
        cur = start;
        len[0] = len[1] = 0;
        sr0 = sr1 = 0;
        continue;
      }
      break;
    }
    if (stop) {
      if (lane == 0) D[D_FLAGS] = F_STOP;
      team_barrier(bar_b, bar_b_threads);
      break;
    }
    if (__builtin_expect(change_neg, 0)) {  // dsgl.hpp:1054-1088: the pool is its base state and size
      pool_base = rng;
      neg_n = len[1] > len[0] ? len[1] : len[0];
      neg_g = neg_count % neg_n;
      rng = jump_any(rng, (uint64_t)neg_n * (uint64_t)K, p.jumps);
      change_neg = false;
      grp_g = -1;
      pf_g = -1;
    }
    // ---- one step (dsgl.hpp:1089-1159) ----
    if (S == STORE_BF16 && lane <= EV_NEG)
      reinterpret_cast<uint64_t*>(D + D_KEYS)[lane] = sr_event_key(p.sr_seed, lane, (uint32_t)wid, step_id);
    const int t1 = sen[pos[0]], t2 = sen[lmax + pos[1]];
    neg_count++;
    neg_g = neg_g + 1 == neg_n ? 0 : neg_g + 1;
    const int g = neg_g;
    NegDraw nd;
    if (__builtin_expect(g == pf_g, 1)) {
      nd = pf;
      grp_state = pf_gs;
    } else {
      uint64_t gs;
      if (g == 0) gs = pool_base;
      else if (g == grp_g + 1) gs = jump_small(grp_state, K, sj);
      else gs = jump_any(pool_base, (uint64_t)g * (uint64_t)K, p.jumps);
      grp_state = gs;
      nd = neg_draw_issue(p, sj, gs);
    }
    grp_g = g;
    const bool end0 = pos[0] + 1 >= len[0], end1 = pos[1] + 1 >= len[1];
    const int O = select_outputs(p, nd, t1, t2, D + D_OUT, D + D_META);
    int out_row = -1;
    if (lane < O) {
      out_row = D[D_OUT + lane];
      prefetch_row(p.woh, out_row, row_bytes);
    }
    // the next step's draws, a step ahead while the pool stays
    if (train_sen_num + (int)end0 + (int)end1 < 2) {
      const int gn = neg_g + 1 == neg_n ? 0 : neg_g + 1;
      uint64_t gs;
      if (gn == 0) gs = pool_base;
      else if (gn == grp_g + 1) gs = jump_small(grp_state, K, sj);
      else gs = jump_any(pool_base, (uint64_t)gn * (uint64_t)K, p.jumps);
      pf = neg_draw_issue(p, sj, gs);
      pf_gs = gs;
      pf_g = gn;
    } else {
      pf_g = -1;
    }
    rng = lcg_next(rng);
    const int b = (int)fast_mod(rng, p.div_window);
    const int I0 = window_inputs<true>(pos[0], len[0], w, b, 0, D + D_IN,
                                       [&](int c) { return __shfl_sync(kFull, rg0, c & (kRing - 1)) * DP; });
    const int I = I0 + window_inputs<true>(pos[1], len[1], w, b, I0, D + D_IN, [&](int c) {
                    return (NS + __shfl_sync(kFull, rg1, c & (kRing - 1))) * DP;
                  });
    __syncwarp();
    // target 2's row is also target 1 or a negative
    const bool alias = __any_sync(kFull, lane != 1 && lane < O && out_row == t2);
    if (lane == 0) count += (unsigned long long)I;
    if (lane == 1) count++;
    if (lane == 2) count += (unsigned long long)O;
    if (lane == 3) count += (unsigned long long)n_pre;
    const float alpha = *reinterpret_cast<volatile float*>(&p.ctr->alpha);
    // ---- window moves and walk ends after the step (dsgl.hpp:1372-1407) ----
    pos[0]++;
    pos[1]++;
    int mv_enter[2] = {-1, -1}, mv_enter_off[2] = {0, 0}, mv_leave[2] = {-1, -1}, mv_leave_off[2] = {0, 0};
    unsigned live[2] = {0u, 0u};
#pragma unroll
    for (int walk = 0; walk < 2; walk++) {
      int& my_v = walk ? sv1 : sv0;
      int& my_r = walk ? sr1 : sr0;
      int& my_g = walk ? rg1 : rg0;
      if (__builtin_expect(pos[walk] >= len[walk], 0)) {
        live[walk] = __ballot_sync(kFull, lane < NS && my_r > 0);
        if (lane < NS) D[L.flush + walk * NS + lane] = my_v;
        my_r = 0;
        len[walk] = 0;
        train_sen_num++;
      } else {
        const int P = pos[walk];
        // the leaving position's slot; its row leaves when no other position holds it and the
        // entering position does not name the same vertex
        int out_slot = -1;
        bool out_last = false;
        if (P - w - 1 >= 0) {
          out_slot = __shfl_sync(kFull, my_g, (P - w - 1) & (kRing - 1));
          out_last = __shfl_sync(kFull, my_r, out_slot) == 1;
        }
        if (P + w < len[walk]) {
          const int v = sen[walk * lmax + P + w];
          const unsigned hit = __ballot_sync(kFull, lane < NS && my_r > 0 && my_v == v);
          const unsigned fr = __ballot_sync(kFull, lane < NS && (my_r == 0 || (out_last && lane == out_slot)));
          const bool fresh = hit == 0;
          int s = __ffs(fresh ? fr : hit) - 1;
          if (s < 0) {  // cannot happen: 2w+1 positions stay
            if (lane == 0) atomicExch(&p.ctr->status, 2);
            s = 0;
          }
          if (fresh) {
            mv_enter[walk] = v;
            mv_enter_off[walk] = (walk * NS + s) * DP;
            if (lane == 3) count++;
          }
          if (out_last && fresh && s == out_slot) {  // in the place of the row that leaves
            mv_leave[walk] = __shfl_sync(kFull, my_v, s);
            mv_leave_off[walk] = mv_enter_off[walk];
            if (lane == s) my_v = v;
            out_slot = -1;
          } else if (lane == s) {
            my_v = v;
            my_r++;
          }
          if (lane == ((P + w) & (kRing - 1))) my_g = s;
        }
        if (out_slot >= 0) {
          const int r = __shfl_sync(kFull, my_r, out_slot) - 1;
          const int v = __shfl_sync(kFull, my_v, out_slot);
          if (lane == out_slot) my_r = r;
          if (r == 0) {
            mv_leave[walk] = v;
            mv_leave_off[walk] = (walk * NS + out_slot) * DP;
          }
        }
      }
    }
    if (lane == 4)
      count += (unsigned long long)(__popc(live[0]) + __popc(live[1]) + (mv_leave[0] >= 0) + (mv_leave[1] >= 0));
    if (lane < 2) {
      const int v = lane ? mv_enter[1] : mv_enter[0];
      if (v >= 0) prefetch_row(p.wih, v, row_bytes);
    }
    if (train_sen_num >= 2) {
      change_neg = true;
      train_sen_num = 0;
    }
    // The order is walk 0 enters, leaves, then walk 1 does: it matters when a row that one
    // walk writes back is one that the other reads or writes back.
    const bool serial = (live[0] | live[1]) != 0 ||
                        (mv_leave[0] >= 0 && (mv_leave[0] == mv_enter[1] || mv_leave[0] == mv_leave[1])) ||
                        (mv_enter[0] >= 0 && mv_enter[0] == mv_leave[1]);
    if (lane == 0) {
      int4* H = reinterpret_cast<int4*>(D);
      H[0] = make_int4((alias ? F_ALIAS : 0) | (serial ? F_SERIAL : 0), I, I0, O);
      H[1] = make_int4(__float_as_int(alpha), n_pre, (int)live[0], (int)live[1]);
      int4* M = reinterpret_cast<int4*>(D + D_MOVE);
      M[0] = make_int4(mv_enter[0], mv_enter_off[0], mv_leave[0], mv_leave_off[0]);
      M[1] = make_int4(mv_enter[1], mv_enter_off[1], mv_leave[1], mv_leave_off[1]);
    }
    step_id++;
    buf = buf + 1 == kDescs ? 0 : buf + 1;
    team_barrier(bar_b, bar_b_threads);
  }
  if (lane == 0) atomicAdd(&p.ctr->pairs, count);
  if (lane == 1) atomicAdd(&p.ctr->steps, count);
  if (lane == 2) atomicAdd(&p.ctr->outputs, count);
  if (lane == 3) atomicAdd(&p.ctr->row_loads, count);
  if (lane == 4) atomicAdd(&p.ctr->row_stores, count);
  if (lane == 0) atomicSub(&p.ctr->active, 1);
}

// ---- the compute warps ------------------------------------------------------------------
// outputs of a group: the first NO of OM, or the rest
template <int OM> constexpr int kGroup = (OM + 1) / 2 + ((OM + 1) / 2) % 2;

// Dot products and gradients of inputs j0 .. j0 + 8 TI - 1 (d % 16 == 0): warp (h, g) sums
// quarters 2h, 2h + 1 of the outputs i0 .. i0 + NO - 1.  Register tiles: lane = m + 2 og +
// 4 ig holds quarter 2h + m of TI inputs against the outputs of parity og (a chunk of TI + TO
// rows read feeds TI TO products); the two quarters meet by a shuffle, each lane keeping half
// of its inputs.  The half sums then go through `corr` to the warp of the pair that owns the
// output (h = 0 the first half of a lane's outputs, h = 1 the others), which adds its own
// ((s0 + s1) + (s2 + s3), in either order) and writes the gradient in its place.
template <int OM, int NO, int TI>
__device__ __forceinline__ void forward_half(int j0, int h, int i0, int I, int first, int O, const RowShape R,
                                             const float* rows, const float* out_rows, const int* in_off, const int* meta,
                                             const float* exp_table, float alpha, float* corr, int bar) {
  constexpr int CS = (OM + 3) & ~3, TO = (NO + 1) / 2, TH = (TO + 1) / 2;
  const int lane = lane_id(), m = lane & 1, og = (lane >> 1) & 1, ig = lane >> 2;
  const int at = 4 * (2 * h + m) * (R.q4 + 1);
  const float* o0 = out_rows + (i0 + og) * R.stride + at;
  const int last = i0 + og + 2 * (TO - 1) < OM ? 2 * (TO - 1) * R.stride : 0;  // past OM: an unused sum
  const float4* x[TI];
#pragma unroll
  for (int t = 0; t < TI; t++) {
    const int j = j0 + ig + 8 * t;
    x[t] = reinterpret_cast<const float4*>(rows + in_off[j < I ? j : I - 1] + at);
  }
  float2 f[TI][TO];
#pragma unroll
  for (int t = 0; t < TI; t++)
#pragma unroll
    for (int u = 0; u < TO; u++) f[t][u] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int k4 = 0; k4 < R.q4; k4++) {
    float4 xv[TI], ov[TO];  // rows past O hold stale data: unused sums
#pragma unroll
    for (int t = 0; t < TI; t++) xv[t] = x[t][k4];
#pragma unroll
    for (int u = 0; u < TO; u++) ov[u] = reinterpret_cast<const float4*>(o0 + (u < TO - 1 ? 2 * u * R.stride : last))[k4];
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
  float s[TI / 2][TO];  // inputs t + m TI / 2
#pragma unroll
  for (int t = 0; t < TI / 2; t++)
#pragma unroll
    for (int u = 0; u < TO; u++) {
      const float a = __fadd_rn(f[t][u].x, f[t][u].y), b = __fadd_rn(f[t + TI / 2][u].x, f[t + TI / 2][u].y);
      const float got = __shfl_xor_sync(kFull, m ? a : b, 1);
      s[t][u] = __fadd_rn(m ? b : a, got);
    }
  auto pairs = [&](auto&& fn, bool owned) {  // this lane's (input, output) pairs, owned or not
#pragma unroll
    for (int t = 0; t < TI / 2; t++) {
      const int j = j0 + ig + 8 * (t + m * (TI / 2));
      if (j < I) {
        if ((h == 0) == owned) {
#pragma unroll
          for (int u = 0; u < TH; u++) fn(j, i0 + og + 2 * u, s[t][u]);
        } else {
#pragma unroll
          for (int u = TH; u < TO; u++) fn(j, i0 + og + 2 * u, s[t][u]);
        }
      }
    }
  };
  pairs([&](int j, int i, float v) { if (i < O) corr[j * CS + i] = v; }, false);
  team_barrier(bar, 32 * kCompute);
  pairs([&](int j, int i, float v) {
    if (i < O) {
      const int label = j < first ? (i == 0) : (i == 1);  // outputs t1, t2, negatives
      corr[j * CS + i] = step_gradient(__fadd_rn(v, corr[j * CS + i]), label, exp_table, alpha, meta[i]);
    }
  }, true);
}

// The forward of a team: halves of the dot products when d % 16 == 0 (32 inputs a round, 16
// when no more are left), else every dot product is one chain and the warps split the
// outputs, one lane per input.  bar: barrier of the compute warps.
template <int OM, int DFIX>
__device__ __forceinline__ void team_forward(int r, int I, int first, int O, int d_rt, const float* rows,
                                             const float* out_rows, const int* in_off, const int* meta,
                                             const float* exp_table, float alpha, float* corr, int bar) {
  constexpr int CS = (OM + 3) & ~3;
  const int d = DFIX ? DFIX : d_rt;
  const RowShape R = row_shape(d);
  if ((d & 15) == 0) {
    constexpr int NO = kGroup<OM>;
    const int h = r & 1, i0 = (r >> 1) * NO;
    for (int j0 = 0; j0 < I; j0 += 32) {
      if (I - j0 <= 16)
        forward_half<OM, NO, 2>(j0, h, i0, I, first, O, R, rows, out_rows, in_off, meta, exp_table, alpha, corr, bar);
      else
        forward_half<OM, NO, 4>(j0, h, i0, I, first, O, R, rows, out_rows, in_off, meta, exp_table, alpha, corr, bar);
    }
  } else {
    constexpr int NO = (OM + kCompute - 1) / kCompute;
    const int lane = lane_id(), i0 = r * NO;
    if (i0 >= O) return;
    const int last = i0 + NO <= OM ? (NO - 1) * R.stride : 0;
    for (int j0 = 0; j0 < I; j0 += 32) {
      const int j = j0 + lane;
      const float4* x = reinterpret_cast<const float4*>(rows + in_off[j < I ? j : I - 1]);
      float2 f[NO];
#pragma unroll
      for (int u = 0; u < NO; u++) f[u] = make_float2(0.f, 0.f);
#pragma unroll 4
      for (int k4 = 0; k4 < R.q4; k4++) {
        const float4 xv = x[k4];
#pragma unroll
        for (int u = 0; u < NO; u++) {
          const float4 ov = reinterpret_cast<const float4*>(out_rows + i0 * R.stride + (u < NO - 1 ? u * R.stride : last))[k4];
          f[u] = ffma2(make_float2(ov.x, ov.y), make_float2(xv.x, xv.y), f[u]);
          f[u] = ffma2(make_float2(ov.z, ov.w), make_float2(xv.z, xv.w), f[u]);
        }
      }
      if (j < I) {
#pragma unroll
        for (int u = 0; u < NO; u++) {
          const int i = i0 + u;
          if (i < O) {
            const int label = j < first ? (i == 0) : (i == 1);
            // the sum's three empty partners of the eight-sum form
            const float fv = __fadd_rn(__fadd_rn(__fadd_rn(f[u].x, f[u].y), 0.f), 0.f);
            corr[j * CS + i] = step_gradient(fv, label, exp_table, alpha, meta[i]);
          }
        }
      }
    }
  }
}

// outputMd of N outputs from i0 over all inputs, four of them read at a time; x: the rows at
// the lane's columns
template <int OM, int N, int NC>
__device__ __forceinline__ void team_out_md(int I, const float* x, int step, const int* in_off, const float* corr, int i0,
                                            float2 (&m)[N][NC]) {
  constexpr int NB = NC <= 2 ? 4 : 2;
  for (int j = 0; j < I; j += NB) {
    float2 xv[NB][NC];
    float c[NB][N];
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const int k = j + u < I ? j + u : j;
      load_cols<NC>(x + in_off[k], step, xv[u]);
      load_coef<OM, N>(corr, k, i0, c[u]);
    }
#pragma unroll
    for (int u = 0; u < NB; u++)
      if (j + u < I) accumulate_out<N, NC>(c[u], xv[u], m);
  }
}
// updates of inputs [j0, j1), in order, several rows read at a time: an input whose row is
// that of an earlier one of them continues from its updated value
template <int OM, int NC, bool kAll>
__device__ __forceinline__ void team_update(int j0, int j1, int O, float* x, int step, const int* in_off,
                                            const float* corr, const float2 (&o)[OM][NC]) {
  constexpr int NB = NC <= 2 ? 4 : 2;
  for (int j = j0; j < j1; j += NB) {
    int off[NB];
    float2 v[NB][NC];
    float c[NB][OM];
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const int k = j + u < j1 ? j + u : j;
      off[u] = in_off[k];
      load_cols<NC>(x + off[u], step, v[u]);
      load_coef<OM, OM>(corr, k, 0, c[u]);
    }
    float2 a[NB][NC];
#pragma unroll
    for (int u = 0; u < NB; u++) input_addend<OM, NC, kAll>(c[u], o, O, a[u]);
#pragma unroll
    for (int u = 0; u < NB; u++) {
#pragma unroll
      for (int e = 0; e < u; e++)
#pragma unroll
        for (int t = 0; t < NC; t++)
          if (off[u] == off[e]) v[u][t] = v[e][t];
#pragma unroll
      for (int t = 0; t < NC; t++) v[u][t] = fadd2(v[u][t], a[u][t]);
      if (j + u < j1) store_cols<NC>(x + off[u], step, v[u]);
    }
  }
}

// Columns c .. c + 2 NC - 1 of an updated output row to the table, rounded with the bits of
// their 4-column chunk(s); v becomes the values stored.
template <int S, int NC>
__device__ __forceinline__ void store_out_cols(void* tab, int64_t row, int d, int c, float2 (&v)[NC], uint64_t ev) {
  if constexpr (NC == 2) {
    const float4 n = RowIO<S>::store4(tab, row, d, c >> 2, make_float4(v[0].x, v[0].y, v[1].x, v[1].y), ev);
    v[0] = make_float2(n.x, n.y), v[1] = make_float2(n.z, n.w);
  } else if constexpr (S == STORE_BF16) {
    const uint64_t bits = sr_bits4(ev, (uint32_t)row, (uint32_t)(c >> 2));
    const uint32_t u = cvt_rs_bf16x2(v[0].x, v[0].y, (uint32_t)((c & 2) ? bits >> 32 : bits));
    reinterpret_cast<uint32_t*>(static_cast<uint16_t*>(tab) + row * d)[c >> 1] = u;
    v[0] = make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xFFFF0000u));
  } else {
    reinterpret_cast<float2*>(static_cast<float*>(tab) + row * d)[c >> 1] = v[0];
  }
}

__host__ __device__ constexpr int pow2_at_least(int n) {
  int p = 1;
  while (p < n) p *= 2;
  return p;
}

// S: storage.  OM: output capacity (K + 2 <= OM).  DFIX: d at compile time (0: p.d).  NC:
// column pairs per lane (half a row holds at most 64 NC columns).
// One bound for CTAs of one to three workers, so 128 registers a thread.  The kernels for more
// than five negatives and d > 128 spill 270 to 370 bytes of them, all others at most 108.
template <int S, int OM, int DFIX, int NC>
__global__ void __launch_bounds__(32 * (kCompute + 1) * kTeamMaxPerCta) team_engine_kernel(TrainParams p) {
  extern __shared__ __align__(16) float smem[];
  float* exp_s = smem;
  SmallJumps* sj = reinterpret_cast<SmallJumps*>(smem + 1004);
  for (int i = threadIdx.x; i < kExpTableSize + 1; i += blockDim.x) exp_s[i] = p.exp_table[i];
  for (int i = threadIdx.x; i < 33; i += blockDim.x) {
    sj->mul[i] = p.jumps->small_mul[i];
    sj->add[i] = p.jumps->small_add[i];
  }
  __syncthreads();
  constexpr int T = 32 * (kCompute + 1);
  const int team = threadIdx.x / T, r = (threadIdx.x % T) >> 5;
  const int wid = blockIdx.x * (blockDim.x / T) + team;
  if (wid >= p.workers) return;  // a whole team: its barriers are its own
  const int d = DFIX ? DFIX : p.d;
  const TeamLayout L = team_layout(d, p.window, OM, p.lmax);
  float* base = smem + kHdrWords + team * L.words;
  const int bar_a = 1 + 2 * team, bar_b = 2 + 2 * team;
  if (r == kCompute) {
    plan_worker<S>(p, *sj, L, base, wid, bar_b, T);
    return;
  }

  typedef RowIO<S> IO;
  typedef typename IO::Raw Raw;
  constexpr int NO = kGroup<OM>;  // output rows this warp owns, from i0
  // item layout of row accesses: lane -> (row item, chunk), CHP chunks of the half's columns
  constexpr int kMaxCh = DFIX ? (DFIX / 4 + 1) / 2 : 16 * NC;
  constexpr int CHP = pow2_at_least(kMaxCh), RPI = 32 / CHP, NR = (NO + RPI - 1) / RPI;
  const int lane = lane_id(), DP = L.DP;
  const int h = r & 1, g = r >> 1, i0 = g * NO;
  const int d4 = d >> 2;
  const int q0 = d4 * h / 2, CH = d4 * (h + 1) / 2 - q0;
  const int ch = lane % CHP, isub = lane / CHP;
  const bool has_ch = ch < CH;
  const int q = q0 + (has_ch ? ch : 0);
  const bool has_col = lane * 2 * NC < 4 * CH;
  const RowShape R = row_shape(d);
  const int chunk_off = chunk_at(q, R);
  const int tcol = 4 * q0 + (has_col ? lane * 2 * NC : 0);      // first column in the table,
  const int col = chunk_at(tcol >> 2, R) + (tcol & 3);          // its place in a row
  float* rows = base + L.rows;
  float* out_rows = base + L.out;
  float* corr = base + L.corr;
  const int* descs = reinterpret_cast<const int*>(base + L.desc);

  Raw raw[NR];  // the step's output rows, gathered during the step before
  auto gather = [&](const int* D) {
    const int O = D[D_O];
#pragma unroll
    for (int k = 0; k < NR; k++) {
      const int u = isub + RPI * k, i = i0 + u;
      raw[k] = has_ch && u < NO && i < O ? IO::load_l2(p.woh, D[D_OUT + i], d, q) : Raw{};
    }
  };
  auto row4 = [&](int off) -> float4& { return *reinterpret_cast<float4*>(rows + off + chunk_off); };
  auto out4 = [&](int i) -> float4& { return *reinterpret_cast<float4*>(out_rows + i * DP + chunk_off); };
  Raw ent = Raw{};
  int ent_off = -1;

  team_barrier(bar_b, T);
  const int* D = descs;
  int buf = 0;
  if (!(D[D_FLAGS] & F_STOP)) gather(D);
  while (true) {
    const int4 H0 = *reinterpret_cast<const int4*>(D), H1 = *reinterpret_cast<const int4*>(D + 4);
    const int flags = H0.x, I = H0.y, first = H0.z, O = H0.w;
    if (flags & F_STOP) break;
    // the rows that entered, then those of freshly loaded walks (their slots may be the same
    // after a pass has ended with walks in flight)
    if (ent_off >= 0) row4(ent_off) = IO::widen(ent);
    const int n_pre = H1.y;
    if (__builtin_expect(n_pre > 0, 0)) {
      team_barrier(bar_a, 32 * kCompute);  // the other walk's rows of the last step are written back
      const int split = L.NS * DP;  // offsets from here on are walk 1's
      for (int k0 = 0; k0 < n_pre; k0 += 4 * RPI) {
        Raw v[4];
        int off[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
          const int k = k0 + isub + RPI * u;
          off[u] = has_ch && k < n_pre ? D[L.pre + 2 * k + 1] : -1;
          if ((off[u] >= split) != (g == 1)) off[u] = -1;
          if (off[u] >= 0) v[u] = IO::load_l2(p.wih, D[L.pre + 2 * k], d, q);
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (off[u] >= 0) row4(off[u]) = IO::widen(v[u]);
      }
    }
#pragma unroll
    for (int k = 0; k < NR; k++) {
      const int u = isub + RPI * k, i = i0 + u;
      if (has_ch && u < NO && i < O) out4(i) = IO::widen(raw[k]);
    }
    team_barrier(bar_a, 32 * kCompute);
    team_forward<OM, DFIX>(r, I, first, O, d, rows, out_rows, D + D_IN, D + D_META, exp_s, __int_as_float(H1.x), corr,
                              bar_a);
    team_barrier(bar_b, T);
    buf = buf + 1 == kDescs ? 0 : buf + 1;
    const int* Dn = descs + buf * L.desc_words;
    const uint64_t* keys = reinterpret_cast<const uint64_t*>(D + D_KEYS);

    float2 o[OM][NC];  // the step's output rows in this lane's columns
#pragma unroll
    for (int i = 0; i < OM; i++) {
      if (i < O) load_cols<NC>(out_rows + i * DP + col, 0, o[i]);
      else
#pragma unroll
        for (int t = 0; t < NC; t++) o[i][t] = make_float2(0.f, 0.f);
    }
    float2 m[NO][NC];
#pragma unroll
    for (int u = 0; u < NO; u++)
#pragma unroll
      for (int t = 0; t < NC; t++) m[u][t] = make_float2(0.f, 0.f);

    team_out_md<OM, NO, NC>(I, rows + col, 0, D + D_IN, corr, i0, m);
    // Woh += outputMd, the group's rows, straight from the columns.  Target 2's row may also
    // be target 1 or, rarely, a negative: that sum starts from the value stored before.
    const int t1 = D[D_OUT], t2 = D[D_OUT + 1];
    float2 v[NO][NC];
#pragma unroll
    for (int u = 0; u < NO; u++) {
      const int i = i0 + u;
#pragma unroll
      for (int t = 0; t < NC; t++) v[u][t] = fadd2(g == 0 ? o[u][t] : o[u + NO < OM ? u + NO : u][t], m[u][t]);
      if (!(flags & F_ALIAS) && has_col && i < O)
        store_out_cols<S, NC>(p.woh, D[D_OUT + i], d, tcol, v[u],
                              S == STORE_BF16 ? keys[i == 0 ? EV_TARGET1 : i == 1 ? EV_TARGET2 : EV_NEG] : 0);
    }
    if (__builtin_expect(flags & F_ALIAS, 0)) {
      // group 0's rows in order; its target 2 goes to the later group through the negative's
      // shared-memory row (every warp has read the rows by the first barrier)
      team_barrier(bar_a, 32 * kCompute);
      float2 n2[NC];
      if (g == 0 && has_col) {
        store_out_cols<S, NC>(p.woh, t1, d, tcol, v[0], S == STORE_BF16 ? keys[EV_TARGET1] : 0);
#pragma unroll
        for (int t = 0; t < NC; t++) n2[t] = fadd2(t2 == t1 ? v[0][t] : o[1][t], m[1][t]);
        store_out_cols<S, NC>(p.woh, t2, d, tcol, n2, S == STORE_BF16 ? keys[EV_TARGET2] : 0);
        for (int i = NO; i < O; i++)
          if (D[D_OUT + i] == t2) store_cols<NC>(out_rows + i * DP + col, 0, n2);
      }
      team_barrier(bar_a, 32 * kCompute);
#pragma unroll
      for (int u = 0; u < NO; u++) {
        const int i = i0 + u;
        if (i >= 2 && i < O && has_col) {
          if (D[D_OUT + i] == t2) {
            if (g == 1) load_cols<NC>(out_rows + i * DP + col, 0, n2);
#pragma unroll
            for (int t = 0; t < NC; t++) v[u][t] = fadd2(n2[t], m[u][t]);
          }
          store_out_cols<S, NC>(p.woh, D[D_OUT + i], d, tcol, v[u], S == STORE_BF16 ? keys[EV_NEG] : 0);
        }
      }
    }
    // every warp has its outputMd and output columns, and this step's output rows are stored
    team_barrier(bar_a, 32 * kCompute);
    if (!(Dn[D_FLAGS] & F_STOP)) gather(Dn);
    if (has_col) {
      const int j0 = g ? first : 0, j1 = g ? I : first;
      if (O == OM) team_update<OM, NC, true>(j0, j1, O, rows + col, 0, D + D_IN, corr, o);
      else team_update<OM, NC, false>(j0, j1, O, rows + col, 0, D + D_IN, corr, o);
    }
    __syncwarp();

    // ---- window moves, walk ends (walk 0, then walk 1 where the order matters) ----
    ent_off = -1;
    if (__builtin_expect(!(flags & F_SERIAL), 1)) {
      const int4 mv = *reinterpret_cast<const int4*>(D + D_MOVE + 4 * g);
      const bool act = has_ch && isub == 0;
      if (act && mv.x >= 0) {
        ent = IO::load_l2(p.wih, mv.x, d, q);
        ent_off = mv.y;
      }
      __syncwarp();
      if (act && mv.z >= 0) IO::store4(p.wih, mv.z, d, q, row4(mv.w), S == STORE_BF16 ? keys[EV_WALK0 + g] : 0);
    } else {
#pragma unroll 1
      for (int walk = 0; walk < 2; walk++) {
        if (walk == g) {
          const uint64_t ev = S == STORE_BF16 ? keys[EV_WALK0 + walk] : 0;
          const unsigned live = (unsigned)(walk ? H1.w : H1.z);
          for (int s = isub; live && s < L.NS; s += RPI)
            if (has_ch && ((live >> s) & 1u))
              IO::store4(p.wih, D[L.flush + walk * L.NS + s], d, q, row4((walk * L.NS + s) * DP), ev);
          const int4 mv = *reinterpret_cast<const int4*>(D + D_MOVE + 4 * walk);
          if (has_ch && isub == 0) {
            if (mv.x >= 0) {
              ent = IO::load_l2(p.wih, mv.x, d, q);
              ent_off = mv.y;
            }
            if (mv.z >= 0) IO::store4(p.wih, mv.z, d, q, row4(mv.w), ev);
          }
        }
        if (walk == 0) team_barrier(bar_a, 32 * kCompute);
      }
    }
    __syncwarp();
    D = Dn;
  }
}

template <int S, int OM, int DFIX, int NC>
cudaError_t team_do(const TeamCall& c) {
  auto* k = team_engine_kernel<S, OM, DFIX, NC>;
  const int threads = 32 * (kCompute + 1) * c.wpc;
  cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)c.smem);
  if (e != cudaSuccess) return e;
  if (c.ctas) return cudaOccupancyMaxActiveBlocksPerMultiprocessor(c.ctas, k, threads, c.smem);
  k<<<(c.p->workers + c.wpc - 1) / c.wpc, threads, c.smem, c.s>>>(*c.p);
  return cudaGetLastError();
}

}  // namespace

// One storage and output capacity: each is compiled in a translation unit of its own.
template <int S, int OM>
cudaError_t team_d(int d, const TeamCall& c) {
  if (d == 64) return team_do<S, OM, 64, 1>(c);
  if (d == 128) return team_do<S, OM, 128, 1>(c);
  if (d == 256) return team_do<S, OM, 256, 2>(c);
  return d <= 128 ? team_do<S, OM, 0, 1>(c) : team_do<S, OM, 0, 2>(c);
}

}  // namespace sgns
