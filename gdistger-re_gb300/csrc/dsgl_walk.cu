// dsgl_walk.cu -- the corpus producer in front of the trainer: DistGER's
// information-oriented random walk (InCoM; include/walk.hpp:260-387 for the
// entropy/length correlation, :818-1042 for the walker loop) and the per-edge
// common-neighbour counts it reads (candidate->data, walk.hpp:920; the reference loads
// them from a file, graph.hpp:826).
//
// Random source.  The reference draws from std::mt19937 seeded by std::random_device and
// from rand(), so no run can be reproduced; here walker w draws from its own SplitMix64
// stream (Steele, Lea and Flood 2014): r_k = mix64(base_w + k G), base_w = mix64(seed ^
// w G), G = 0x9E3779B97F4A7C15.  A neighbour index is (r >> 32) * deg >> 32 (Lemire's
// multiply-shift); a uniform double is (r >> 11) 2^-53.  Walker w starts at w % V
// (walk.hpp:503-506); the corpus lists walks in walker order, -1 after each.
//
// One move from vertex c of degree ds: ds == 0 ends the walk; u = adj[c][index]; ds == 2
// with adj[c][0] == c ends it; before the first move u == c draws again (at most 64 times
// in a row, then the walk ends -- the reference spins forever there); p = uniform;
// pa = ((1 / (ds - cn)) max(ds, du)) / min(ds, du); trace = tanh(pa) <= p; u is appended,
// then c again on a trace; the walk moves to u only without one.  With trace steps off
// there is no p draw and every move goes on to u.  Every appended vertex
// updates the correlation state (Correlation::iterate, step 1) with f = its earlier visits,
// and the walk stops after more than min_length moves once R*R < r_threshold or R < 0
// (walk.hpp:868-874), or when it holds max_length vertices.
//
// Arithmetic: IEEE double through explicit _rn intrinsics (no contraction), so every
// decision equals the CPU restatement's bit for bit.  x log2 x comes from a host-built
// table of integers; tanh is (E - 1) / (E + 1) with E = exp(2x) = 2^k exp(r), Cody-Waite
// reduction with ln 2 split into its float head and the remainder, exp(r) by Taylor's
// series to r^13 (Horner); tanh(x) = 1 for x >= 20.
//
// What bounds it: a warp's double instruction holds the SM's double unit for 16 cycles, so the
// length pass does as few of them as the exact result allows:
//   * the walk's vertex count is also its update count, so every division of the update is by
//     an integer n <= 1001: a * (1/n) with a host-rounded reciprocal, corrected by its exact
//     remainder (Markstein 1990), is the rounded quotient -- three operations;
//   * the moments of the length alone (ES, ESS, their deviation) are a table over n;
//   * R is needed after min_length moves only, and its test R*R < r first compares
//     ex*ex with r DH DS and takes the square root and quotient only within 2^-40 of equality;
//   * the trace test likewise runs in fp32 unless the draw is within 1e-4 of the threshold.
// About 25 double operations per vertex (35 past min_length) instead of about 200.  The token
// pass knows every walk's length and so repeats only the draws and the neighbour reads.
//
// Kernels: one thread per directed edge for the common-neighbour counts; one thread per
// walker for the walks, taking its next walker as soon as one ends (lengths differ by a
// factor of four), its path history in shared memory, four vertices to 16 bytes.  Between the
// two passes an exclusive scan of length + 1 gives each walk's place, so no per-walk buffer
// is needed.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "sgns_internal.h"

namespace sgns {
namespace {

constexpr uint64_t kGolden = 0x9E3779B97F4A7C15ULL;
constexpr int kMaxRedraws = 64;
constexpr int kScanBlock = 1024;

__device__ __forceinline__ double pow2i(int k) { return __longlong_as_double((long long)(1023 + k) << 52); }

__device__ __forceinline__ double tanh_pos(double x) {
  if (!(x < 20.0)) return 1.0;
  const double y = __dmul_rn(2.0, x);
  const double ln2_hi = (double)(float)0.6931471805599453;
  const double ln2_lo = 0.6931471805599453 - ln2_hi;
  const int k = __double2int_rz(__dadd_rn(__dmul_rn(y, 1.4426950408889634), 0.5));
  const double kd = (double)k;
  const double r = __dsub_rn(__dsub_rn(y, __dmul_rn(kd, ln2_hi)), __dmul_rn(kd, ln2_lo));
  const double c[14] = {1.0,         1.0,          1.0 / 2.0,      1.0 / 6.0,       1.0 / 24.0,
                        1.0 / 120.0, 1.0 / 720.0,  1.0 / 5040.0,   1.0 / 40320.0,   1.0 / 362880.0,
                        1.0 / 3628800.0, 1.0 / 39916800.0, 1.0 / 479001600.0, 1.0 / 6227020800.0};
  double p = c[13];
#pragma unroll
  for (int i = 12; i >= 0; i--) p = __dadd_rn(__dmul_rn(p, r), c[i]);
  const double E = __dmul_rn(p, pow2i(k));
  return __ddiv_rn(__dsub_rn(E, 1.0), __dadd_rn(E, 1.0));
}

// a / n for an integer n with reciprocal r = rn(1 / n): the quotient's distance from a rounding
// boundary is at least 1 / (2 n) of its last place, the corrected sum's error 2^-51 of it
__device__ __forceinline__ double div_by(double a, double n, double r) {
  const double q = __dmul_rn(a, r);
  return __fma_rn(__fma_rn(-q, n, a), r, q);
}

// What an update to a walk of n vertices reads, whatever the walk (kWalkMaxLength + 2 entries,
// built on the host by walk_length_table).
static_assert(kWalkTableDoubles == 4, "LengthTable");
struct __align__(16) LengthTable {
  double dxl;  // (n-1) log2 (n-1) - n log2 n
  double rcp;  // 1 / n
  double es;   // the running mean of the length after the update
  double ds;   // its deviation ESS - ES^2
};

struct WalkArgs {
  const int64_t* indptr;
  const int32_t* indices;
  const int32_t* cn;
  const double* xl;         // x log2 x
  const LengthTable* len;
  int64_t V, walker_num;
  int32_t min_length, max_length;
  double r_threshold;
  uint64_t seed;
  int32_t trace;           // 1: the trace step of walk.hpp:920-1031; 0: moves only
  const int32_t* refused;  // not 0: an input was refused, nothing is walked
  int32_t* lengths;        // pass 1 output
  const int64_t* offsets;  // pass 2 input (exclusive scan of length + 1)
  int32_t* corpus;         // pass 2 output
};

// Correlation state (Correlation::iterate, walk.hpp:330-365, step 1)
struct Corr {
  double H, EH, EHS, EHH;
};
__device__ __forceinline__ void corr_iterate(Corr& c, const LengthTable& t, double xf, double xf1, int n) {
  const double S1 = (double)n, S0 = (double)(n - 1);
  const double dt = __dsub_rn(__dadd_rn(t.dxl, xf1), xf);
  const double H1 = div_by(__dsub_rn(__dmul_rn(S0, c.H), dt), S1, t.rcp);
  c.EH = __dadd_rn(c.EH, div_by(__dsub_rn(H1, c.EH), S1, t.rcp));
  c.EHS = __dadd_rn(c.EHS, div_by(__dsub_rn(__dmul_rn(H1, S1), c.EHS), S1, t.rcp));
  c.EHH = __dadd_rn(c.EHH, div_by(__dsub_rn(__dmul_rn(H1, H1), c.EHH), S1, t.rcp));
  c.H = H1;
}
// R*R < threshold or R < 0 (walk.hpp:868-874), R = ex / sqrt(DH DS)
__device__ __forceinline__ bool corr_stops(const Corr& c, const LengthTable& t, double threshold) {
  const double DH = __dsub_rn(c.EHH, __dmul_rn(c.EH, c.EH));
  const double ex = __dsub_rn(c.EHS, __dmul_rn(c.EH, t.es));
  const double P = __dmul_rn(DH, t.ds);
  // clear of the boundary, of zeros and of the range's ends: the rounded R*R and ex*ex / P
  // differ by a few last places
  if (ex > 1e-100 && ex < 1e100 && P > 1e-100 && P < 1e100 && threshold > 1e-6 && threshold < 1e6) {
    const double a = ex * ex, b = threshold * P, slack = b * 0x1p-40;
    if (a < b - slack) return true;
    if (a > b + slack) return false;
  }
  const double R = ex == 0.0 ? 0.0 : __ddiv_rn(ex, __dsqrt_rn(P));
  return __dmul_rn(R, R) < threshold || R < 0.0;
}
// tanh(((1 / (ds - cn)) max(ds, du)) / min(ds, du)) <= p (walk.hpp:920-1031)
__device__ __forceinline__ bool trace_step(int64_t ds, int64_t du, int32_t cn, uint64_t r) {
  const int64_t mx = ds > du ? ds : du, mn = ds < du ? ds : du, left = ds - cn;
  if (left > 0 && mn > 0) {
    const float x = (float)mx / ((float)left * (float)mn);
    const float e = __expf(2.f * fminf(x, 20.f));
    const float th = __fdividef(e - 1.f, e + 1.f), p = (float)(r >> 40) * 0x1p-24f;
    if (fabsf(th - p) > 1e-4f) return th < p;
  }
  const double p = __dmul_rn((double)(r >> 11), 1.0 / 9007199254740992.0);
  const double pa = __ddiv_rn(__dmul_rn(__ddiv_rn(1.0, (double)left), (double)mx), (double)mn);
  return tanh_pos(pa) <= p;
}

// A walker's draws and moves; both passes make the same ones.
struct Walker {
  int64_t cur;
  uint64_t ctr;
  __device__ __forceinline__ void start(const WalkArgs& a, int64_t w) {
    cur = w % a.V;
    ctr = mix64(a.seed ^ ((uint64_t)w * kGolden));
  }
  // The next candidate: false when the walk ends here.  moved: no longer at the walk's first
  // vertex (before that a candidate equal to it is drawn again).
  __device__ __forceinline__ bool candidate(const WalkArgs& a, bool moved, int32_t* u, bool* trace) {
    const int64_t b = __ldg(&a.indptr[cur]);
    const int64_t ds = __ldg(&a.indptr[cur + 1]) - b;
    if (ds == 0) return false;
    int64_t e = 0;
    for (int redraws = 0;; redraws++) {
      const uint64_t r = mix64(ctr);
      ctr += kGolden;
      e = b + (int64_t)(((r >> 32) * (uint64_t)ds) >> 32);
      *u = __ldg(&a.indices[e]);
      if (ds == 2 && __ldg(&a.indices[b]) == cur) return false;
      if (moved || *u != cur) break;
      if (redraws + 1 >= kMaxRedraws) return false;
    }
    *trace = false;
    if (a.trace) {
      const uint64_t r = mix64(ctr);
      ctr += kGolden;
      const int64_t du = __ldg(&a.indptr[(int64_t)*u + 1]) - __ldg(&a.indptr[*u]);
      *trace = trace_step(ds, du, __ldg(&a.cn[e]), r);
    }
    return true;
  }
};

// Pass 1: lengths[w].  Shared memory: the tables' first max_length + 2 entries, then the path
// histories, four vertices to an int4, [ceil(max_length / 4)][blockDim.x].
__global__ void __launch_bounds__(256) walk_lengths_kernel(WalkArgs a) {
  extern __shared__ __align__(16) unsigned char walk_smem[];
  if (*a.refused) return;
  const int T = blockDim.x, tid = threadIdx.x, entries = a.max_length + 2;
  LengthTable* tab = reinterpret_cast<LengthTable*>(walk_smem);
  double* xl = reinterpret_cast<double*>(tab + entries);
  int4* hist = reinterpret_cast<int4*>(xl + ((entries + 1) & ~1)) + tid;
  for (int i = tid; i < entries; i += T) {
    tab[i] = a.len[i];
    xl[i] = a.xl[i];
  }
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * T;
  int64_t w = (int64_t)blockIdx.x * T + tid;
  Walker k{};
  Corr c{};
  int len = 0;
  auto begin = [&]() {
    k.start(a, w);
    c = Corr{0.0, 0.0, 0.0, 0.0};
    hist[0] = make_int4((int32_t)k.cur, -1, -1, -1);
    len = 1;
  };
  // appends v; true when the walk stops there
  auto append = [&](int32_t v) -> bool {
    int f = 0;
    for (int g = 0; 4 * g < len; g++) {
      const int4 h = hist[g * T];
      f += (h.x == v) + (h.y == v) + (h.z == v) + (h.w == v);
    }
    if ((len & 3) == 0) hist[(len >> 2) * T] = make_int4(v, -1, -1, -1);
    else reinterpret_cast<int32_t*>(&hist[(len >> 2) * T])[len & 3] = v;
    len++;
    const LengthTable t = tab[len];
    corr_iterate(c, t, xl[f], xl[f + 1], len);
    // len - 1 vertices appended so far
    if (len - 1 > a.min_length && corr_stops(c, t, a.r_threshold)) return true;
    return len >= a.max_length;
  };
  if (w < a.walker_num) begin();
  while (w < a.walker_num) {
    int32_t u;
    bool trace, done = len >= a.max_length || !k.candidate(a, len > 1, &u, &trace);
    if (!done) {
      done = append(u);
      if (!trace) k.cur = u;
      else if (!done) done = append((int32_t)k.cur);
    }
    if (done) {
      a.lengths[w] = len;
      w += stride;
      if (w < a.walker_num) begin();
    }
  }
}

// Pass 2: the walk's tokens and its -1 at offsets[w].
__global__ void __launch_bounds__(256) walk_tokens_kernel(WalkArgs a) {
  if (*a.refused) return;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  Walker k{};
  int32_t *out = nullptr, *last = nullptr;  // next token, place of the -1
  bool moved = false;
  auto begin = [&]() {
    k.start(a, w);
    out = a.corpus + a.offsets[w];
    last = a.corpus + a.offsets[w + 1] - 1;
    *out++ = (int32_t)k.cur;
    moved = false;
  };
  if (w < a.walker_num) begin();
  while (w < a.walker_num) {
    int32_t u;
    bool trace;
    if (out < last && k.candidate(a, moved, &u, &trace)) {
      moved = true;
      *out++ = u;
      if (!trace) k.cur = u;
      else if (out < last) *out++ = (int32_t)k.cur;
    } else {
      *out = -1;
      w += stride;
      if (w < a.walker_num) begin();
    }
  }
}

// ---- exclusive scan of (lengths[w] + 1) into offsets[0..n] (int64) -------------------
__device__ __forceinline__ int64_t block_inclusive_scan(int64_t v, int64_t* warp_sums) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t t = __shfl_up_sync(0xFFFFFFFFu, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) warp_sums[wid] = v;
  __syncthreads();
  if (wid == 0) {
    int64_t s = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t t = __shfl_up_sync(0xFFFFFFFFu, s, o);
      if (lane >= o) s += t;
    }
    warp_sums[lane] = s;
  }
  __syncthreads();
  if (wid > 0) v += warp_sums[wid - 1];
  return v;
}

__global__ void __launch_bounds__(kScanBlock) scan_tiles_kernel(const int32_t* lengths, int64_t n, int64_t* offsets,
                                                                int64_t* tile_sums) {
  __shared__ int64_t ws[32];
  const int64_t i = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
  const int64_t v = i < n ? (int64_t)lengths[i] + 1 : 0;
  const int64_t inc = block_inclusive_scan(v, ws);
  if (i < n) offsets[i] = inc - v;  // exclusive within the tile
  if (threadIdx.x == kScanBlock - 1) tile_sums[blockIdx.x] = inc;
}

// one block: exclusive scan of the tile sums in rounds of kScanBlock; tile_sums[n_tiles]
// receives the total
__global__ void __launch_bounds__(kScanBlock) scan_tile_sums_kernel(int64_t* tile_sums, int64_t n_tiles) {
  __shared__ int64_t ws[32];
  __shared__ int64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < n_tiles; base += kScanBlock) {
    const int64_t i = base + threadIdx.x;
    const int64_t v = i < n_tiles ? tile_sums[i] : 0;
    const int64_t inc = block_inclusive_scan(v, ws);
    const int64_t c0 = carry;
    if (i < n_tiles) tile_sums[i] = c0 + inc - v;
    __syncthreads();
    if (threadIdx.x == kScanBlock - 1) carry = c0 + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) tile_sums[n_tiles] = carry;
}

__global__ void add_tile_offsets_kernel(int64_t* offsets, int64_t n, const int64_t* tile_sums, int64_t n_tiles,
                                        WalkReport* report) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) offsets[i] += tile_sums[i / kScanBlock];
  if (i == 0) offsets[n] = report->total = tile_sums[n_tiles];
}

// ---- common-neighbour counts ----------------------------------------------------------
// The entries of an edge's shorter adjacency list are searched in the longer one: up to
// `own` of them by one thread (edge_cn_kernel), else by a warp (edge_cn_long_kernel).  The
// long lists are those of edges between hubs, which follow one another (a hub's edges are
// consecutive, and its neighbours begin with the other hubs where ids follow degree), so the
// second kernel spreads them over the GPU.  What bounds them: the searches' dependent loads.  A
// power law's (gamma 2.1, ids by degree) 2.2M vertices and 32M edges, and 20k and 321k: 81 and
// 0.77 ms a call with the long lists left to the warps that came to them, 77 and 0.33 with a warp
// for every edge, 44 and 0.26 now.  1.1M vertices and 6.3M edges without hubs: 0.40, 4.2, 0.33.
constexpr int kEdgeWarps = 8, kEdgeThreads = 32 * kEdgeWarps, kOwnEntries = 24;

// the largest u in [lo, hi) with indptr[u] <= e
__device__ __forceinline__ int64_t source_of(const int64_t* __restrict__ indptr, int64_t e, int64_t lo, int64_t hi) {
  while (hi - lo > 1) {
    const int64_t mid = (lo + hi) >> 1;
    if (__ldg(&indptr[mid]) <= e) lo = mid;
    else hi = mid;
  }
  return lo;
}
// 1 when the sorted list of n >= 1 entries holds x.  Lists of one length take the same steps
// whatever x is, so the lanes of a warp that search one list stay together.
__device__ __forceinline__ int holds(const int32_t* __restrict__ list, int n, int32_t x) {
  while (n > 1) {  // the last entry <= x, if any, is one of list[0..n)
    const int h = n >> 1;
    list += __ldg(list + h) <= x ? h : 0;
    n -= h;
  }
  return __ldg(list) == x;
}
// An edge's two lists, the shorter one first
struct EdgeLists {
  const int32_t *s, *l;
  int ns, nl;
  __device__ __forceinline__ EdgeLists(const int64_t* __restrict__ indptr, const int32_t* __restrict__ indices, int64_t u,
                                       int32_t v) {
    const int64_t ub = __ldg(&indptr[u]), vb = __ldg(&indptr[v]);
    const int nu = (int)(__ldg(&indptr[u + 1]) - ub), nv = (int)(__ldg(&indptr[(int64_t)v + 1]) - vb);
    const bool u_short = nu <= nv;
    s = indices + (u_short ? ub : vb), l = indices + (u_short ? vb : ub);
    ns = u_short ? nu : nv, nl = u_short ? nv : nu;
  }
};

// One thread per directed edge e = (u, v), 32 consecutive ones to a warp: the sources of the
// first and the last are found in indptr, every other source between them.  cn[e]: the count,
// or ~u for an edge left to edge_cn_long_kernel.
// status bits: 1 = a neighbour outside [0, V), 2 = an adjacency list not strictly increasing.
__global__ void __launch_bounds__(kEdgeThreads) edge_cn_kernel(const int64_t* __restrict__ indptr,
                                                               const int32_t* __restrict__ indices, int64_t V, int64_t E,
                                                               int own, int32_t* __restrict__ cn, int32_t* status) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * kEdgeThreads;
  for (int64_t base = (int64_t)blockIdx.x * kEdgeThreads + threadIdx.x - lane; base < E; base += stride) {
    int64_t u = 0;
    if (lane < 2) u = source_of(indptr, lane == 0 ? base : base + 32 < E ? base + 31 : E - 1, 0, V);
    const int64_t u0 = __shfl_sync(0xFFFFFFFFu, u, 0), u1 = __shfl_sync(0xFFFFFFFFu, u, 1);
    const int64_t e = base + lane;
    if (e < E) {
      u = source_of(indptr, e, u0, u1 + 1);
      const int32_t v = __ldg(&indices[e]);
      int c = 0;
      if (v < 0 || v >= V) {
        atomicOr(status, 1);
      } else {
        if (e > __ldg(&indptr[u]) && __ldg(&indices[e - 1]) >= v) atomicOr(status, 2);
        const EdgeLists a(indptr, indices, u, v);
        if (a.ns > own) c = ~(int32_t)u;
        else
          for (int i = 0; i < a.ns; i++) c += holds(a.l, a.nl, __ldg(a.s + i));
      }
      cn[e] = c;
    }
  }
}

// The edges left by edge_cn_kernel.  A block looks through eight runs of `run` edges, one per
// warp, that lie evenly over all edges, and its warps take what is left of them in turn.
__global__ void __launch_bounds__(kEdgeThreads) edge_cn_long_kernel(const int64_t* __restrict__ indptr,
                                                                    const int32_t* __restrict__ indices, int64_t E,
                                                                    int run, int32_t* cn) {
  __shared__ int64_t queue_e[kEdgeThreads];
  __shared__ int32_t queue_u[kEdgeThreads];
  __shared__ int queued, taken;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t runs = (E + run - 1) / run;
  if (threadIdx.x == 0) queued = taken = 0;
  for (int64_t first = blockIdx.x; first < runs; first += kEdgeWarps * (int64_t)gridDim.x) {
    const int64_t e = (first + warp * (int64_t)gridDim.x) * run + lane;
    const int32_t left = lane < run && e < E ? cn[e] : 0;
    if (!__syncthreads_or(left < 0)) continue;
    if (left < 0) {
      const int k = atomicAdd(&queued, 1);
      queue_e[k] = e;
      queue_u[k] = ~left;
    }
    __syncthreads();
    while (true) {
      int k = 0;
      if (lane == 0) k = atomicAdd(&taken, 1);
      k = __shfl_sync(0xFFFFFFFFu, k, 0);
      if (k >= queued) break;
      const EdgeLists a(indptr, indices, queue_u[k], __ldg(&indices[queue_e[k]]));
      int c = 0;
      for (int i = lane; i - lane < a.ns; i += 32) c += i < a.ns ? holds(a.l, a.nl, __ldg(a.s + i)) : 0;
      c = __reduce_add_sync(0xFFFFFFFFu, c);
      if (lane == 0) cn[queue_e[k]] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0) queued = taken = 0;  // before the next round's first barrier
  }
}

// CSR checks before any kernel follows the graph's pointers.  status bits: 4 = indptr[0]
// != 0, indptr[V] != E or indptr decreasing; 1 = a neighbour outside [0, V).
__global__ void __launch_bounds__(256) validate_csr_kernel(const int64_t* __restrict__ indptr,
                                                           const int32_t* __restrict__ indices, int64_t V, int64_t E,
                                                           int32_t* status) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (int64_t u = t0; u <= V; u += stride) {
    const int64_t x = indptr[u];
    const bool bad = (u == 0 && x != 0) || (u == V && x != E) || (u > 0 && indptr[u - 1] > x);
    if (bad) atomicOr(status, 4);
  }
  for (int64_t e = t0; e < E; e += stride) {
    const int32_t v = indices[e];
    if (v < 0 || v >= V) atomicOr(status, 1);
  }
}

// Offsets that a caller brings, before any walk is written at them.  report: total, the last
// offset; refused bits: 8 = the first is not 0 or a walk has not 1 to max_length vertices and its
// -1, 16 = the last is above cap.  8 bytes a walk: no difference in a call of 2M walks (10.3 ms
// with it and without).
__global__ void __launch_bounds__(256) validate_offsets_kernel(const int64_t* __restrict__ offsets, int64_t n,
                                                               int max_length, int64_t cap, WalkReport* report) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; w < n; w += stride) {
    const int64_t x = offsets[w], next = offsets[w + 1];
    const uint64_t vertices = (uint64_t)next - (uint64_t)x - 1;
    if ((w == 0 && x != 0) || vertices - 1 >= (uint64_t)max_length) atomicOr(&report->refused, 8);
    if (w == n - 1) {
      report->total = next;
      if (next > cap) atomicOr(&report->refused, 16);
    }
  }
}

}  // namespace

cudaError_t launch_validate_offsets(const int64_t* offsets, int64_t walker_num, int max_length, int64_t cap,
                                    WalkReport* report, int num_sms, cudaStream_t s) {
  const int64_t want = (walker_num + 255) / 256, most = (int64_t)num_sms * 16;
  validate_offsets_kernel<<<(unsigned)(want < most ? want : most), 256, 0, s>>>(offsets, walker_num, max_length, cap,
                                                                                report);
  return cudaGetLastError();
}

cudaError_t launch_validate_csr(const int64_t* indptr, const int32_t* indices, int64_t V, int64_t E,
                                int32_t* status, int num_sms, cudaStream_t s) {
  const int64_t want = ((V > E ? V : E) + 256) / 256;
  const int64_t cap = (int64_t)num_sms * 16;
  validate_csr_kernel<<<(unsigned)(want < cap ? want : cap), 256, 0, s>>>(indptr, indices, V, E, status);
  return cudaGetLastError();
}

static size_t walk_table_smem(int max_length) {
  const size_t entries = (size_t)max_length + 2;
  return entries * sizeof(LengthTable) + ((entries + 1) & ~(size_t)1) * sizeof(double);
}
static size_t walk_smem(int max_length, int threads) {
  return walk_table_smem(max_length) + sizeof(int4) * (size_t)((max_length + 3) / 4) * threads;
}
// Threads per block of the length pass: the most walkers resident on an SM (228 KB of shared
// memory, 1 KB reserved per block), the larger block on a tie.
static int walk_block_threads(int max_length) {
  int best = 32, resident = 0;
  for (int t = 32; t <= 256; t += 32) {
    const size_t smem = walk_smem(max_length, t);
    if (smem > 232448) break;
    const int r = (int)(233472 / (smem + 1024)) * t;
    if (r >= resident) best = t, resident = r;
  }
  return best;
}

size_t walk_scratch_bytes(int64_t walker_num) {
  const int64_t tiles = (walker_num + kScanBlock - 1) / kScanBlock;
  return sizeof(int32_t) * (size_t)walker_num + sizeof(int64_t) * (size_t)(tiles + 1);
}

// Pass 1 (lengths) and the scan: offsets, walker_num + 1 entries, the last = total tokens (also
// in the report).
cudaError_t launch_info_walks_count(const int64_t* indptr, const int32_t* indices, const int32_t* cn,
                                    const double* xl, const double* len_table, int64_t V, int64_t walker_num,
                                    int min_length, int max_length, double r_threshold, uint64_t seed, int trace,
                                    void* scratch, int num_sms, int64_t* offsets, WalkReport* report, cudaStream_t s) {
  const int64_t tiles = (walker_num + kScanBlock - 1) / kScanBlock;
  int64_t* tile_sums = static_cast<int64_t*>(scratch);
  int32_t* lengths = reinterpret_cast<int32_t*>(tile_sums + tiles + 1);
  const WalkArgs a{indptr, indices, cn, xl, reinterpret_cast<const LengthTable*>(len_table), V, walker_num, min_length,
                   max_length, r_threshold, seed, trace, &report->refused, lengths, nullptr, nullptr};
  const int T = walk_block_threads(max_length);
  const size_t smem = walk_smem(max_length, T);
  cudaError_t e = cudaFuncSetAttribute(walk_lengths_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, walk_lengths_kernel, T, smem);
  if (e != cudaSuccess) return e;
  const int64_t want = (walker_num + T - 1) / T;
  const int64_t resident = (int64_t)num_sms * (per_sm > 0 ? per_sm : 1);  // threads take walkers in turn
  walk_lengths_kernel<<<(unsigned)(want < resident ? want : resident), T, smem, s>>>(a);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  scan_tiles_kernel<<<(unsigned)tiles, kScanBlock, 0, s>>>(lengths, walker_num, offsets, tile_sums);
  scan_tile_sums_kernel<<<1, kScanBlock, 0, s>>>(tile_sums, tiles);
  add_tile_offsets_kernel<<<(unsigned)((walker_num + 256) / 256), 256, 0, s>>>(offsets, walker_num, tile_sums, tiles,
                                                                              report);
  return cudaGetLastError();
}

// Pass 2: the walks again, written at their offsets.
cudaError_t launch_info_walks_emit(const int64_t* indptr, const int32_t* indices, const int32_t* cn, int64_t V,
                                   int64_t walker_num, uint64_t seed, int trace, const int64_t* offsets,
                                   int32_t* corpus, const WalkReport* report, int num_sms, cudaStream_t s) {
  WalkArgs a{};
  a.indptr = indptr, a.indices = indices, a.cn = cn, a.V = V, a.walker_num = walker_num;
  a.seed = seed, a.trace = trace, a.refused = &report->refused, a.offsets = offsets, a.corpus = corpus;
  const int64_t want = (walker_num + 255) / 256, resident = (int64_t)num_sms * 8;
  walk_tokens_kernel<<<(unsigned)(want < resident ? want : resident), 256, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_edge_common_neighbors(const int64_t* indptr, const int32_t* indices, int64_t V, int64_t E,
                                         int32_t* cn, int32_t* status, int num_sms, cudaStream_t s) {
  if (E == 0) return cudaSuccess;
  const int64_t want = (E + kEdgeThreads - 1) / kEdgeThreads, cap = (int64_t)num_sms * 64;
  const int64_t warps = (int64_t)num_sms * 8 * kEdgeWarps;  // eight blocks per SM
  // Up to four edges per warp of the GPU (39k) a thread's own chain of searches is the call:
  // nearly all go to a warp (2,000 vertices of a power law, 31k edges: 81 -> 65 us; above, at 114k
  // edges of a flat graph, 53 -> 77).
  const int own = E <= 4 * warps ? 2 : kOwnEntries;
  edge_cn_kernel<<<(unsigned)std::min(want, cap), kEdgeThreads, 0, s>>>(indptr, indices, V, E, own, cn, status);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int run = (int)std::min<int64_t>(32, (E + warps - 1) / warps);
  const int64_t blocks = (E + (int64_t)run * kEdgeWarps - 1) / ((int64_t)run * kEdgeWarps);
  edge_cn_long_kernel<<<(unsigned)std::min(blocks, cap), kEdgeThreads, 0, s>>>(indptr, indices, E, run, cn);
  return cudaGetLastError();
}

}  // namespace sgns
