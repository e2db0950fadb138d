// dsgl_ingest.cu -- walk-file text to the trainer's corpus, on the GPU.
//
// The text is the reference's walk format (include/path.hpp:92,108: " %u" per vertex,
// "\n" after each walk), tokenised on the separators the reference's reader uses
// (word2vec.cu:1008, " \n\r\t").  Output: vertex ids with -1 after each walk that holds
// at least one id -- the layout of graph->local_corpus (path.hpp:96,110) that
// Train_SGNS_MPI reads.  The buffer is read as one file: position n acts as a final
// newline, so the last walk ends even without one.
//
// Three passes over 8 KB tiles, 32 bytes to a thread, as eight 4-byte words with byte-wise
// (SWAR) class masks:
//   1. each thread counts its outputs; a tile's Span says how many, whether its first
//      significant byte is a newline whose walk end depends on what precedes it, and the kind
//      of its last significant byte;
//   2. the tile Spans are scanned (64-bit output counts): by one block where 1024 tiles (8 MB)
//      hold the text, else in groups of 1024 tiles by one block each, the group totals by one
//      block, then the group prefixes added to the tiles';
//   3. each thread finds its outputs again and lists the bytes that end them in shared memory,
//      beside the text as digit values; the lanes of its warp take that list evenly, sum each
//      id from the eight bytes that end it with dp4a (longer ids byte by byte) and store in
//      order.
// The usual text -- every newline directly behind a digit, no byte but digits, spaces and
// newlines -- takes a short path: a newline there is decided by the byte before it, so the
// outputs are a plain sum.  Any other tile builds its threads' Spans from bit masks and scans
// them; Span combination is associative, so the order of the scans does not matter.
//
// What bounds it: instruction issue (87% of it in pass 3: about 165 per warp and 1 KB to
// classify, 90 to list the outputs, 40 per 32 tokens).  1.2 GB of text, 160M tokens, whose bytes
// take 175 us in pass 1 and 270 us in pass 3: pass 1 536 -> 292 us, pass 3 1,090 -> 573 us
// against masks for every tile, digit-by-digit ids, scattered stores and a maximum per warp on
// one word (with that last one pass 3 takes 932 us).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "dsgl_device.cuh"

namespace sgns {

namespace {

constexpr int kIngThreads = 256;
constexpr int kIngBytes = 32;                       // bytes per thread
constexpr int kIngTile = kIngThreads * kIngBytes;   // 8192 bytes per tile
constexpr int kIngHalo = 16;                        // bytes kept before the tile
constexpr int kScanBlock = 1024;

enum : uint32_t { SIG_NONE = 0, SIG_DIGIT = 1, SIG_NL = 2 };

struct Span {
  unsigned long long cnt;  // outputs, not counting a pending first newline
  uint32_t pend;           // first significant byte is a newline
  uint32_t last;           // kind of the last significant byte
};

__host__ __device__ __forceinline__ Span span_combine(Span a, Span b) {
  Span r;
  r.cnt = a.cnt + b.cnt + ((b.pend && a.last == SIG_DIGIT) ? 1ull : 0ull);
  r.pend = a.last != SIG_NONE ? a.pend : b.pend;
  r.last = b.last != SIG_NONE ? b.last : a.last;
  return r;
}

__device__ __forceinline__ Span span_identity() { return Span{0ull, 0u, SIG_NONE}; }

// byte i of the text with a virtual newline at n and blanks after it
__device__ __forceinline__ uint8_t text_byte(const uint8_t* b, int64_t n, int64_t i) {
  return i < n ? __ldg(b + i) : (i == n ? (uint8_t)'\n' : (uint8_t)' ');
}

// 16 text bytes from g: one load where they lie inside the text and it starts on a 16-byte
// boundary (tiles are 8 KB apart, so every chunk is then aligned), byte by byte otherwise.
__device__ __forceinline__ uint4 text16(const uint8_t* b, int64_t n, int64_t g, bool aligned) {
  if (aligned && g >= 0 && g + 16 <= n) return __ldg(reinterpret_cast<const uint4*>(b + g));
  uint8_t t[16];
#pragma unroll
  for (int k = 0; k < 16; k++) t[k] = g + k < 0 ? (uint8_t)' ' : text_byte(b, n, g + k);
  return make_uint4(t[0] | t[1] << 8 | t[2] << 16 | (uint32_t)t[3] << 24, t[4] | t[5] << 8 | t[6] << 16 | (uint32_t)t[7] << 24,
                    t[8] | t[9] << 8 | t[10] << 16 | (uint32_t)t[11] << 24,
                    t[12] | t[13] << 8 | t[14] << 16 | (uint32_t)t[15] << 24);
}

// Byte-class tests on 4 bytes at once (SWAR; no carry crosses a byte): 0x80 in each byte
// that is NOT a decimal digit, resp. in each NONZERO byte.
__device__ __forceinline__ uint32_t nondigit80(uint32_t w) {
  const uint32_t t = w ^ 0x30303030u;  // digits become 0..9
  return (((t & 0x7F7F7F7Fu) + 0x76767676u) | t) & 0x80808080u;
}
__device__ __forceinline__ uint32_t nonzero80(uint32_t x) {
  return (((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x) & 0x80808080u;
}
// one bit per byte from a 0x80-per-byte mask
__device__ __forceinline__ uint32_t nibble(uint32_t m80) { return (m80 * 0x00204081u) >> 28; }

// Class masks of a thread's 32 bytes (bit j = byte j): digits, newlines and, when
// kCheck, anything that is not a digit, newline, space, tab or CR.
struct Masks {
  uint32_t dig, nl, bad;
};
template <bool kCheck>
__device__ __forceinline__ Masks classify(const uint32_t (&w)[8]) {
  Masks m{0u, 0u, 0u};
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const uint32_t dg = nondigit80(w[k]) ^ 0x80808080u;
    const uint32_t nl = nonzero80(w[k] ^ 0x0A0A0A0Au) ^ 0x80808080u;
    m.dig |= nibble(dg) << (4 * k);
    m.nl |= nibble(nl) << (4 * k);
    if (kCheck) {
      const uint32_t bl = (nonzero80(w[k] ^ 0x20202020u) & nonzero80(w[k] ^ 0x09090909u) &
                           nonzero80(w[k] ^ 0x0D0D0D0Du)) ^ 0x80808080u;
      m.bad |= nibble(0x80808080u & ~(dg | nl | bl)) << (4 * k);
    }
  }
  return m;
}

// Outputs of a thread's 32 bytes as bit masks: ends of ids (last digit) and newlines that
// end a walk given the kind of significant byte before the span (carry: SIG_*; SIG_NONE
// leaves the first newline undecided and reported in *pend).
struct Emits {
  uint32_t ids, walks;
};
__device__ __forceinline__ Emits emits(const Masks& m, bool next_digit, uint32_t carry, uint32_t* pend) {
  Emits e;
  e.ids = m.dig & ~((m.dig >> 1) | (next_digit ? 0x80000000u : 0u));
  e.walks = 0;
  *pend = 0;
  const uint32_t sig = m.dig | m.nl;
  uint32_t nls = m.nl;
  while (nls) {
    const int p = __ffs(nls) - 1;
    nls &= nls - 1;
    const uint32_t before = sig & ((1u << p) - 1u);
    if (before) {
      if ((m.dig >> (31 - __clz(before))) & 1u) e.walks |= 1u << p;
    } else if (carry == SIG_DIGIT) {
      e.walks |= 1u << p;
    } else if (carry == SIG_NONE) {
      *pend = 1;
    }
  }
  return e;
}

// Span of one thread's 32 bytes from its masks and its outputs with no carry.
__device__ __forceinline__ Span span_of(const Masks& m, const Emits& e, uint32_t pend) {
  const uint32_t sig = m.dig | m.nl;
  Span sp;
  sp.cnt = __popc(e.ids) + __popc(e.walks);
  sp.pend = pend;
  sp.last = sig == 0 ? SIG_NONE : (((m.dig >> (31 - __clz(sig))) & 1u) ? SIG_DIGIT : SIG_NL);
  return sp;
}

// Block-wide exclusive scan of Spans (blockDim.x == kIngThreads); returns the thread's
// exclusive prefix and writes the block total to *total.
__device__ __forceinline__ Span block_exclusive(Span v, Span* total) {
  __shared__ Span warp_tot[kIngThreads / 32];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  Span inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    Span u;
    u.cnt = __shfl_up_sync(kFull, inc.cnt, o);
    u.pend = __shfl_up_sync(kFull, inc.pend, o);
    u.last = __shfl_up_sync(kFull, inc.last, o);
    if (lane >= o) inc = span_combine(u, inc);
  }
  if (lane == 31) warp_tot[wp] = inc;
  __syncthreads();
  Span before = span_identity();
  for (int k = 0; k < wp; k++) before = span_combine(before, warp_tot[k]);
  Span ex;
  ex.cnt = __shfl_up_sync(kFull, inc.cnt, 1);
  ex.pend = __shfl_up_sync(kFull, inc.pend, 1);
  ex.last = __shfl_up_sync(kFull, inc.last, 1);
  if (lane == 0) ex = span_identity();
  Span all = span_identity();
  for (int k = 0; k < kIngThreads / 32; k++) all = span_combine(all, warp_tot[k]);
  *total = all;
  __syncthreads();
  return span_combine(before, ex);
}

// 0x80 in each digit byte / newline byte of a valid text's word: digits are the bytes with bit
// 4, newlines the others with bit 1 (space, tab and CR have neither).
__device__ __forceinline__ uint32_t valid_digit80(uint32_t w) { return (w << 3) & 0x80808080u; }
__device__ __forceinline__ uint32_t valid_newline80(uint32_t w) { return (w << 6) & ~(w << 3) & 0x80808080u; }

__global__ void __launch_bounds__(kIngThreads) ingest_count_kernel(const uint8_t* b, int64_t n, bool aligned,
                                                                  Span* tile_span, long long* err) {
  __shared__ int sums[kIngThreads / 32];
  const int64_t first = (int64_t)blockIdx.x * kIngTile + (int64_t)threadIdx.x * kIngBytes;
  const int lane = threadIdx.x & 31;
  const uint4 v0 = text16(b, n, first, aligned), v1 = text16(b, n, first + 16, aligned);
  const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
  // the bytes before and after: the neighbouring lanes' words, or a byte of the text
  uint32_t before = __shfl_up_sync(kFull, w[7], 1), after = __shfl_down_sync(kFull, w[0], 1);
  if (lane == 0) before = first > 0 ? (uint32_t)text_byte(b, n, first - 1) << 24 : 0x20000000u;
  if (lane == 31) after = text_byte(b, n, first + kIngBytes);
  uint32_t nd[10];  // 0x80 in each byte that is not a digit; [0] before, [9] after
  nd[0] = nondigit80(before);
  nd[9] = nondigit80(after);
#pragma unroll
  for (int k = 0; k < 8; k++) nd[k + 1] = nondigit80(w[k]);
  uint32_t acc = 0, odd = 0;  // outputs, in four byte-wide sums; bytes that the short path does not take
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const uint32_t me = nd[k + 1];
    const uint32_t not_nl = nonzero80(w[k] ^ 0x0A0A0A0Au), not_sp = nonzero80(w[k] ^ 0x20202020u);
    const uint32_t prev = __funnelshift_l(nd[k], me, 8), next = __funnelshift_r(me, nd[k + 2], 8);
    odd |= me & not_nl & not_sp;          // neither digit, newline nor space
    odd |= ~not_nl & prev & 0x80808080u;  // a newline not directly behind a digit
    acc += ((~me & next & 0x80808080u) | (~not_nl & ~prev & 0x80808080u)) >> 7;  // last digits, walk ends
  }
  const bool has_sig = (nd[8] != 0x80808080u) || (nonzero80(w[7] ^ 0x0A0A0A0Au) != 0x80808080u);
  // the last thread's last word has to show the tile's last significant byte
  const bool slow = odd != 0 || (threadIdx.x == kIngThreads - 1 && !has_sig);
  if (!__syncthreads_or(slow)) {
    int c = (int)((acc * 0x01010101u) >> 24);
    c = __reduce_add_sync(kFull, c);
    if (lane == 0) sums[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == kIngThreads - 1) {
      unsigned long long t = 0;
      for (int k = 0; k < kIngThreads / 32; k++) t += (unsigned long long)sums[k];
      const uint32_t dig = ~nd[8] & 0x80808080u, nl = ~nonzero80(w[7] ^ 0x0A0A0A0Au) & 0x80808080u;
      tile_span[blockIdx.x] = Span{t, 0u, dig > nl ? SIG_DIGIT : SIG_NL};
    }
    return;
  }
  Span v = span_identity();
  if (first <= n) {
    const Masks m = classify<true>(w);
    if (m.bad) atomicMin(err, (long long)(first + __ffs(m.bad) - 1));
    uint32_t pend;
    const Emits e = emits(m, !(nd[9] & 0x80u), SIG_NONE, &pend);
    v = span_of(m, e, pend);
  }
  Span total;
  block_exclusive(v, &total);
  if (threadIdx.x == 0) tile_span[blockIdx.x] = total;
}

// Exclusive scan of Spans by one block, 1024 consecutive Spans per round (coalesced reads,
// block scan, carry to the next round); the text starts as if after a newline.  Used on the
// tiles of a short text and on the group totals of a long one: out[i] = prefix of i, the last
// entry the whole text.
// *clear (the call's largest-id word) is zeroed on the way.
__global__ void __launch_bounds__(kScanBlock) ingest_scan_kernel(const Span* tile_span, int64_t ntiles, Span* out,
                                                                 unsigned long long* clear) {
  __shared__ Span warp_tot[kScanBlock / 32];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  if (threadIdx.x == 0) *clear = 0ull;
  Span carry = Span{0ull, 0u, SIG_NL};
  for (int64_t r0 = 0; r0 < ntiles; r0 += kScanBlock) {
    const int64_t t = r0 + threadIdx.x;
    const Span v = t < ntiles ? tile_span[t] : span_identity();
    Span inc = v;
    for (int o = 1; o < 32; o <<= 1) {
      Span u;
      u.cnt = __shfl_up_sync(kFull, inc.cnt, o);
      u.pend = __shfl_up_sync(kFull, inc.pend, o);
      u.last = __shfl_up_sync(kFull, inc.last, o);
      if (lane >= o) inc = span_combine(u, inc);
    }
    if (lane == 31) warp_tot[wp] = inc;
    __syncthreads();
    if (wp == 0) {  // scan of the 32 warp totals
      Span w = warp_tot[lane];
      for (int o = 1; o < 32; o <<= 1) {
        Span u;
        u.cnt = __shfl_up_sync(kFull, w.cnt, o);
        u.pend = __shfl_up_sync(kFull, w.pend, o);
        u.last = __shfl_up_sync(kFull, w.last, o);
        if (lane >= o) w = span_combine(u, w);
      }
      warp_tot[lane] = w;  // inclusive over warps
    }
    __syncthreads();
    Span before = wp > 0 ? warp_tot[wp - 1] : span_identity();
    Span ex;
    ex.cnt = __shfl_up_sync(kFull, inc.cnt, 1);
    ex.pend = __shfl_up_sync(kFull, inc.pend, 1);
    ex.last = __shfl_up_sync(kFull, inc.last, 1);
    if (lane == 0) ex = span_identity();
    if (t < ntiles) out[t] = span_combine(carry, span_combine(before, ex));
    carry = span_combine(carry, warp_tot[kScanBlock / 32 - 1]);
    __syncthreads();
  }
  if (threadIdx.x == 0) out[ntiles] = carry;
}

// Pass 2, first level: one block per group of kScanBlock consecutive tiles; out[t] = prefix
// of tile t within its group, group_tot[g] = the group's Span.
__global__ void __launch_bounds__(kScanBlock) ingest_scan_groups_kernel(const Span* tile_span, int64_t ntiles,
                                                                       Span* out, Span* group_tot) {
  __shared__ Span warp_tot[kScanBlock / 32];
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const int64_t t = (int64_t)blockIdx.x * kScanBlock + threadIdx.x;
  const Span v = t < ntiles ? tile_span[t] : span_identity();
  Span inc = v;
  for (int o = 1; o < 32; o <<= 1) {
    Span u;
    u.cnt = __shfl_up_sync(kFull, inc.cnt, o);
    u.pend = __shfl_up_sync(kFull, inc.pend, o);
    u.last = __shfl_up_sync(kFull, inc.last, o);
    if (lane >= o) inc = span_combine(u, inc);
  }
  if (lane == 31) warp_tot[wp] = inc;
  __syncthreads();
  if (wp == 0) {
    Span w = warp_tot[lane];
    for (int o = 1; o < 32; o <<= 1) {
      Span u;
      u.cnt = __shfl_up_sync(kFull, w.cnt, o);
      u.pend = __shfl_up_sync(kFull, w.pend, o);
      u.last = __shfl_up_sync(kFull, w.last, o);
      if (lane >= o) w = span_combine(u, w);
    }
    warp_tot[lane] = w;
  }
  __syncthreads();
  Span ex;
  ex.cnt = __shfl_up_sync(kFull, inc.cnt, 1);
  ex.pend = __shfl_up_sync(kFull, inc.pend, 1);
  ex.last = __shfl_up_sync(kFull, inc.last, 1);
  if (lane == 0) ex = span_identity();
  if (t < ntiles) out[t] = span_combine(wp > 0 ? warp_tot[wp - 1] : span_identity(), ex);
  if (threadIdx.x == 0) group_tot[blockIdx.x] = warp_tot[kScanBlock / 32 - 1];
}

// Pass 2, last step: every tile's prefix behind its group's; out[ntiles] = the whole text.
__global__ void ingest_scan_add_kernel(Span* out, int64_t ntiles, const Span* group_pre, int64_t ngroups) {
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t <= ntiles; t += (int64_t)gridDim.x * blockDim.x)
    out[t] = t < ntiles ? span_combine(group_pre[t / kScanBlock], out[t]) : group_pre[ngroups];
}

// A valid text's word as digit values, other bytes 0x80.
__device__ __forceinline__ uint32_t digit_values(uint32_t w) {
  const uint32_t t = w << 3;  // 0x80: a digit (valid_digit80)
  uint32_t digit;             // its sign spread over its byte (__byte_perm takes no sign bit)
  asm("prmt.b32 %0, %1, 0, 0xBA98;" : "=r"(digit) : "r"(t));
  return (w & digit & 0x0F0F0F0Fu) | (~t & 0x80808080u);
}

__global__ void __launch_bounds__(kIngThreads) ingest_emit_kernel(const uint8_t* b, int64_t n, bool aligned,
                                                                 const Span* tile_prefix,
                                                                 int32_t* tokens, long long* err,
                                                                 unsigned long long* max_id /* largest id + 1 */) {
  // digit_values of the text from base - halo; the spare word is read, not used, by an id that
  // ends at the tile's last byte
  __shared__ __align__(16) uint8_t s[kIngHalo + kIngTile + 4];
  __shared__ uint16_t ends[kIngTile];  // a warp's outputs by the byte that ends them
  __shared__ int warp_sum[kIngThreads / 32];
  const int64_t base = (int64_t)blockIdx.x * kIngTile;
  const int64_t first = base + (int64_t)threadIdx.x * kIngBytes;
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  const uint4 v0 = text16(b, n, first, aligned), v1 = text16(b, n, first + 16, aligned);
  const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
  uint32_t before = __shfl_up_sync(kFull, w[7], 1), after = __shfl_down_sync(kFull, w[0], 1);
  if (lane == 0) before = first > 0 ? (uint32_t)text_byte(b, n, first - 1) << 24 : 0x20000000u;
  if (lane == 31) after = text_byte(b, n, first + kIngBytes);
  uint4* sv = reinterpret_cast<uint4*>(s + kIngHalo) + 2 * threadIdx.x;
  sv[0] = make_uint4(digit_values(w[0]), digit_values(w[1]), digit_values(w[2]), digit_values(w[3]));
  sv[1] = make_uint4(digit_values(w[4]), digit_values(w[5]), digit_values(w[6]), digit_values(w[7]));
  if (threadIdx.x == 0) {
    const uint4 h = text16(b, n, base - kIngHalo, aligned);
    sv[-1] = make_uint4(digit_values(h.x), digit_values(h.y), digit_values(h.z), digit_values(h.w));
  }
  // the count pass has checked every byte.  Outputs: last digits, and newlines directly behind
  // a digit; a newline elsewhere sends the tile down the long path.
  uint32_t dg[10];
  dg[0] = valid_digit80(before);
  dg[9] = valid_digit80(after);
#pragma unroll
  for (int k = 0; k < 8; k++) dg[k + 1] = valid_digit80(w[k]);
  uint32_t out = 0, odd = 0;
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    uint32_t bits = 0;  // 128 x the outputs of eight bytes, one bit each
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint32_t me = dg[k + h + 1], nl = valid_newline80(w[k + h]);
      const uint32_t prev = __funnelshift_l(dg[k + h], me, 8), next = __funnelshift_r(me, dg[k + h + 2], 8);
      odd |= nl & ~prev;
      bits = __dp4a((me & ~next) | (nl & prev), h ? 0x80402010u : 0x08040201u, bits);
    }
    out |= k == 0 ? bits >> 7 : bits << (4 * k - 7);
  }
  if (first > n) out = 0, odd = 0;
  const unsigned long long tile_at = tile_prefix[blockIdx.x].cnt;
  unsigned long long warp_at;  // outputs before this warp's
  int at, total;               // the thread's first output in its warp, and the warp's outputs
  {
    const int c = __popc(out);
    int inc = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(kFull, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) warp_sum[wp] = inc;
    at = inc - c;
    total = __shfl_sync(kFull, inc, 31);
  }
  if (!__syncthreads_or(odd != 0)) {
    int prior = 0;
#pragma unroll
    for (int k = 0; k < kIngThreads / 32; k++) prior += k < wp ? warp_sum[k] : 0;
    warp_at = tile_at + prior;
  } else {
    Masks m{0u, 0u, 0u};
    Emits e{0u, 0u};
    uint32_t pend = 0;
    Span v = span_identity();
    if (first <= n) {
      m = classify<false>(w);
      e = emits(m, dg[9] & 0x80u, SIG_NONE, &pend);
      v = span_of(m, e, pend);
    }
    Span all;
    const Span ex = span_combine(tile_prefix[blockIdx.x], block_exclusive(v, &all));
    if (pend && ex.last == SIG_DIGIT) e.walks |= 1u << (__ffs(m.nl) - 1);
    out = e.ids | e.walks;
    warp_at = __shfl_sync(kFull, ex.cnt, 0);
    at = (int)(ex.cnt - warp_at);
    total = __shfl_sync(kFull, at + __popc(out), 31);
  }
  uint16_t* mine = ends + wp * (32 * kIngBytes);
  while (out) {  // outputs in text order
    mine[at++] = (uint16_t)(threadIdx.x * kIngBytes + 31 - __clz(out & (0u - out)));
    out &= out - 1;
  }
  __syncwarp();
  uint32_t mx = 0;  // largest id + 1
  int32_t* dst = tokens + warp_at;
  for (int k = lane; k < total; k += 32) {
    const int j = mine[k];
    // the eight bytes that end at byte j, last first: hi = j .. j-3, lo = j-4 .. j-7
    const uint32_t* p = reinterpret_cast<const uint32_t*>(s) + ((kIngHalo + j - 7) >> 2);
    const uint32_t sel = 0x0123u + 0x1111u * ((j + 1) & 3);
    const uint32_t a0 = p[0], a1 = p[1], a2 = p[2];
    const uint32_t lo = __byte_perm(a0, a1, sel), hi = __byte_perm(a1, a2, sel);
    // keep the digits below the lowest 0x80
    const uint32_t nh = hi & 0x80808080u, nl = lo & 0x80808080u;
    const uint32_t h = hi & (nh - 1) & ~nh, l = nh ? 0u : lo & (nl - 1) & ~nl;
    uint32_t val = __dp4a(l, 0x0A010000u, 0u);
    val = __dp4a(l, 0x00000A01u, val * 100u);
    val = __dp4a(h, 0x0A010000u, val * 100u);
    val = __dp4a(h, 0x00000A01u, val * 100u);
    if (!(nh | nl)) {
      // eight digits or more: up to three before them
      const uint8_t* last = s + kIngHalo + j;
      unsigned long long all = val, scale = 100000000ull;
      int L = 8;
      while (L < 11 && last[-L] < 10) {
        all += scale * last[-L];
        scale *= 10;
        L++;
      }
      if (L > 10 || all > 0x7FFFFFFFull) {  // an eleventh digit, or above 2^31 - 1
        atomicMin(err, (long long)(base + j));
        all = 0;
      }
      val = (uint32_t)all;
    }
    if (hi & 0x80u) val = 0xFFFFFFFFu;  // the newline itself: -1
    dst[k] = (int32_t)val;
    mx = max(mx, val + 1u);
  }
  mx = __reduce_max_sync(kFull, mx);
  // one L2 word takes 1.2M warps' maxima longer (0.8 ns each) than the rest of the kernel: only
  // those above the value that the SM's L1 holds, which is never more than the true one, go there
  if (lane == 0 && mx > __ldca(max_id)) atomicMax(max_id, (unsigned long long)mx);  // 0: no id
}

// Occurrences of each vertex (the reference's vertex_cn, path.hpp:98); lanes holding the
// same id add once per warp.
__global__ void vertex_count_kernel(const int32_t* tokens, int64_t n, int32_t* counts, int64_t V) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x; i0 < n; i0 += stride) {
    const int64_t i = i0 + threadIdx.x;
    const int32_t v = i < n ? tokens[i] : -1;
    const bool ok = v >= 0 && v < V;
    const unsigned grp = __match_any_sync(kFull, ok ? v : -1);
    if (ok && (__ffs(grp) - 1) == (int)(threadIdx.x & 31)) atomicAdd(&counts[v], __popc(grp));
  }
}

}  // namespace

// scratch: tile Spans, tile prefixes (+ the whole text), the error and largest-id words
// (64 bytes), then the group totals and group prefixes (+ the whole text)
size_t ingest_scratch_bytes(int64_t n) {
  const int64_t ntiles = (n + 1 + kIngTile - 1) / kIngTile, ngroups = (ntiles + kScanBlock - 1) / kScanBlock;
  return sizeof(Span) * (size_t)(2 * ntiles + 1) + 64 + sizeof(Span) * (size_t)(2 * ngroups + 1);
}

cudaError_t launch_ingest_count(const uint8_t* bytes, int64_t n, void* scratch, unsigned long long* n_out,
                                long long* err_pos, cudaStream_t s) {
  const int64_t ntiles = (n + 1 + kIngTile - 1) / kIngTile;
  Span* tile_span = static_cast<Span*>(scratch);
  Span* prefix = tile_span + ntiles;
  long long* err = reinterpret_cast<long long*>(prefix + ntiles + 1);
  unsigned long long* mx = reinterpret_cast<unsigned long long*>(err + 1);
  cudaError_t e;
  if ((e = cudaMemsetAsync(err, 0x7F, sizeof *err, s)) != cudaSuccess) return e;  // kIngestNoError
  const bool aligned = (reinterpret_cast<uintptr_t>(bytes) & 15) == 0;
  ingest_count_kernel<<<(unsigned)ntiles, kIngThreads, 0, s>>>(bytes, n, aligned, tile_span, err);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (ntiles <= kScanBlock) {  // one group: its prefixes are the text's
    ingest_scan_kernel<<<1, kScanBlock, 0, s>>>(tile_span, ntiles, prefix, mx);
  } else {
    // tile prefixes in two levels: within groups of kScanBlock tiles (one block each), the
    // group totals by one block, then the group prefixes added to the tiles'
    const int64_t ngroups = (ntiles + kScanBlock - 1) / kScanBlock;
    Span* group_tot = reinterpret_cast<Span*>(reinterpret_cast<char*>(prefix + ntiles + 1) + 64);
    Span* group_pre = group_tot + ngroups;
    ingest_scan_groups_kernel<<<(unsigned)ngroups, kScanBlock, 0, s>>>(tile_span, ntiles, prefix, group_tot);
    ingest_scan_kernel<<<1, kScanBlock, 0, s>>>(group_tot, ngroups, group_pre, mx);
    ingest_scan_add_kernel<<<(unsigned)std::min<int64_t>((ntiles + 256) / 256, 152 * 8), 256, 0, s>>>(
        prefix, ntiles, group_pre, ngroups);
  }
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  struct {  // the whole text's Span and, behind it, the error word
    Span whole;
    long long err;
  } got;
  if ((e = cudaMemcpyAsync(&got, prefix + ntiles, sizeof(Span) + sizeof(long long), cudaMemcpyDeviceToHost, s)) !=
          cudaSuccess ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess)
    return e;
  *n_out = got.whole.cnt;
  *err_pos = got.err;
  return cudaSuccess;
}

cudaError_t launch_ingest_emit(const uint8_t* bytes, int64_t n, void* scratch, int32_t* tokens, long long* err_pos,
                               long long* max_id, cudaStream_t s) {
  const int64_t ntiles = (n + 1 + kIngTile - 1) / kIngTile;
  Span* tile_span = static_cast<Span*>(scratch);
  Span* prefix = tile_span + ntiles;
  long long* err = reinterpret_cast<long long*>(prefix + ntiles + 1);
  unsigned long long* mx = reinterpret_cast<unsigned long long*>(err + 1);
  cudaError_t e;
  const bool aligned = (reinterpret_cast<uintptr_t>(bytes) & 15) == 0;
  ingest_emit_kernel<<<(unsigned)ntiles, kIngThreads, 0, s>>>(bytes, n, aligned, prefix, tokens, err, mx);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  long long got[2];  // the error and largest-id words
  if ((e = cudaMemcpyAsync(got, err, sizeof got, cudaMemcpyDeviceToHost, s)) != cudaSuccess ||
      (e = cudaStreamSynchronize(s)) != cudaSuccess)
    return e;
  *err_pos = got[0];
  *max_id = got[1] - 1;
  return cudaSuccess;
}

cudaError_t launch_vertex_count(const int32_t* tokens, int64_t n, int32_t* counts, int64_t V, int num_sms,
                                cudaStream_t s) {
  cudaError_t e;
  if ((e = cudaMemsetAsync(counts, 0, sizeof(int32_t) * (size_t)V, s)) != cudaSuccess) return e;
  if (n == 0) return cudaSuccess;
  int64_t blocks = (n + 255) / 256;
  if (blocks > (int64_t)num_sms * 8) blocks = (int64_t)num_sms * 8;
  vertex_count_kernel<<<(unsigned)blocks, 256, 0, s>>>(tokens, n, counts, V);
  return cudaGetLastError();
}

}  // namespace sgns
