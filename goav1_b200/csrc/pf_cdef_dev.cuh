// pf_cdef_dev.cuh - CDEF device helpers shared by the decoder-side CDEF
// kernel (pf_cdef.cu) and the encoder strength search (pf_search.cu).
// Arithmetic follows goav1's cdef/direction.go:37-79, :432-501 and
// cdef/filter.go:79-191, :603-612.
#pragma once

#include <cuda_fp16.h>

#include "pf_common.cuh"

namespace pf {

constexpr int kVeryLarge = 0x4000;

// ---- CDEF on vertical sample pairs ----
//
// A staged unit is an array of 32-bit words: word (r, c) holds the samples of
// rows r and r + 1 of column c, so every tap of two vertically adjacent
// samples is one aligned word whatever its offset, and both are filtered by
// the same packed instructions.  A sample n of 8 or 10 bits is held as the
// fp16 value 1 + n / 1024 (bits 0x3c00 | n), an absent one as -3 (kPairNone):
// below every sample in a signed 16-bit maximum, above every one in an
// unsigned minimum, and too far from any for a tap to count, so it drops out
// of the filter by itself.  Everything the filter forms from samples is a
// whole or half multiple of 2^-10 below 2^11 of them, which fp16 holds
// exactly: the result is the same integer as the reference's
// (tests/test_cdef_pair_arithmetic.py runs through every difference,
// strength and shift).  12-bit samples do not fit: they are staged as plain
// integers (absent: kVeryLarge) and filtered by packed 16-bit integers.  Words
// that hold more than 12 bits, which no bitstream has, are staged the same way
// and filtered one by one in 32-bit integers.
constexpr int kPH = 68;  // rows -2 .. 65 of a unit
constexpr int kPX = 4;   // words left of the unit's first column
constexpr int kPW = 96;  // words a row: a multiple of the 32 banks, so a tap's row offset moves no lane's bank
constexpr uint32_t kPairBias = 0x3c003c00u;
constexpr uint32_t kPairNone = 0xc200c200u;
constexpr uint32_t kPairRawNone = 0x40004000u;

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }

// constrain() of one threshold and shift on pairs (cdef/filter.go:603-612):
// min(|d|, max(0, thr - (|d| >> shift))) with d's sign.
// thr - floor(|d| / 2^shift) is the fp16 rounding of
//   1 + (thr - (|d| + 1/2 - 2^(shift-1)) / 2^shift) / 1024,
// whose last place in [1, 2) is 2^-10: the sum is at least 2^-(shift+1) off
// every tie, and below 1 only where the threshold has run out, which the
// saturating subtraction turns into 0.
struct PairTap {
  uint32_t k, m, o;  // 1 + thr / 1024; -2^-shift; (1/2 - 2^(shift-1)) / 1024, each in both halves
};

// The constants from their bits: 1 + thr / 1024 is 0x3c00 + thr, -2^-shift has
// the exponent 15 - shift, and 2^(shift-1) - 1/2 is shift ones in binary
// (thr at most 1023, shift at most 8).
__host__ __device__ __forceinline__ PairTap pair_tap(int thr, int shift) {
  const uint32_t m = 0xbc00u - ((uint32_t)shift << 10);
  const uint32_t o = shift ? 0x8000u + (((uint32_t)shift + 3) << 10) + 1024u - (2048u >> shift) : 0u;
  return PairTap{kPairBias + (uint32_t)thr * 0x10001u, m * 0x10001u, o * 0x10001u};
}

__device__ __forceinline__ __half2 pair_constrain(__half2 d, const PairTap& t) {
  const __half2 a = __habs2(d);
  const __half2 v = __hfma2(__hadd2(a, bits_h2(t.o)), bits_h2(t.m), bits_h2(t.k));
  const __half2 c = __hmin2(__hadd2_sat(v, __float2half2_rn(-1.f)), a);
  return bits_h2(h2_bits(c) | (h2_bits(d) & 0x80008000u));
}

// x + (8 + sum - (sum < 0) >> 4): sum / 16 rounded half away from zero, by
// letting the addition to the sample (last place 2^-10 in [1, 2)) round.  The
// factor is 1/16 and its last place more, which takes the ties of up to 64
// sixteenths away from zero and nothing else across one.  A value below
// sample 0 or above 1023 is not a whole one; the clamp that follows takes it
// to the range.
__device__ __forceinline__ __half2 pair_round(__half2 x, __half2 sum) { return __hfma2(sum, bits_h2(0x2c012c01u), x); }

// One pair through the filter (cdef/filter.go:79-169); c points at its word.
// po: the primary taps' word offsets (entry dir + 2), s0 / s1 the secondary
// ones' (dir + 4, dir).  w0, w1: the primary weights (4, 2 or 3, 3).  The
// clamp applies with both filters on; where a block's own primary strength is
// zero it changes nothing (the secondary taps alone stay inside their own
// range), so it needs no per-block test.
template <bool kPri, bool kSec>
__device__ __forceinline__ uint32_t pair_filter(const uint32_t* c, const PairTap& pri, __half2 w0, __half2 w1,
                                                const PairTap& sec, int2 po, int2 s0, int2 s1) {
  const uint32_t xb = c[0];
  const __half2 x = bits_h2(xb);
  uint32_t hi = xb, lo = xb;
  auto range = [&](uint32_t a, uint32_t b) {
    if (kPri && kSec) {
      lo = __vimin3_u16x2(lo, a, b);
      hi = __vimax3_s16x2(hi, a, b);
    }
  };
  auto tap = [&](uint32_t a, const PairTap& t) { return pair_constrain(__hsub2(bits_h2(a), x), t); };
  __half2 sum = __float2half2_rn(0.f);
  if (kPri) {
    const uint32_t a0 = c[po.x], a1 = c[-po.x], a2 = c[po.y], a3 = c[-po.y];
    sum = __hmul2(w0, __hadd2(tap(a0, pri), tap(a1, pri)));
    sum = __hfma2(w1, __hadd2(tap(a2, pri), tap(a3, pri)), sum);
    range(a0, a1);
    range(a2, a3);
  }
  if (kSec) {
    const uint32_t b0 = c[s0.x], b1 = c[-s0.x], b2 = c[s1.x], b3 = c[-s1.x];
    const __half2 n = __hadd2(__hadd2(tap(b0, sec), tap(b1, sec)), __hadd2(tap(b2, sec), tap(b3, sec)));
    range(b0, b1);
    range(b2, b3);
    const uint32_t b4 = c[s0.y], b5 = c[-s0.y], b6 = c[s1.y], b7 = c[-s1.y];
    const __half2 f = __hadd2(__hadd2(tap(b4, sec), tap(b5, sec)), __hadd2(tap(b6, sec), tap(b7, sec)));
    range(b4, b5);
    range(b6, b7);
    sum = __hadd2(sum, __hfma2(n, __float2half2_rn(2.f), f));
  }
  uint32_t y = h2_bits(pair_round(x, sum));
  if (kPri && kSec) y = __vminu2(__vmaxu2(y, lo), hi);
  return y;
}

// (dy, dx) of the two taps of each CDEF direction entry, cdef/filter.go:53-66.
static __constant__ int8_t c_cdef_dir[12][2][2] = {
    {{1, 0}, {2, 0}},   {{1, 0}, {2, -1}}, {{-1, 1}, {-2, 2}}, {{0, 1}, {-1, 2}},
    {{0, 1}, {0, 2}},   {{0, 1}, {1, 2}},  {{1, 1}, {2, 2}},   {{1, 0}, {2, 1}},
    {{1, 0}, {2, 0}},   {{1, 0}, {2, -1}}, {{-1, 1}, {-2, 2}}, {{0, 1}, {-1, 2}},
};

__device__ __forceinline__ int pair_off(int e, int k, int pitch) { return c_cdef_dir[e][k][0] * pitch + c_cdef_dir[e][k][1]; }

// Direction cost over one 8x8 block (cdef/direction.go:37-79 partial sums,
// :469-501 cost): for direction D the samples (i, j), shifted to 8 bits
// and less 128, are summed into partials p[dir_k(D, i, j)], and the cost is
// the weighted sum of their squares.  dir_k is that index; dir_count is how
// many samples each partial sums.
__host__ __device__ constexpr int dir_k(int D, int i, int j) {
  return D == 0 ? i + j : D == 1 ? i + (j >> 1) : D == 2 ? i : D == 3 ? 3 + i - (j >> 1) :
         D == 4 ? 7 + i - j : D == 5 ? 3 - (i >> 1) + j : D == 6 ? j : (i >> 1) + j;
}
__host__ __device__ constexpr int dir_count(int D, int k) {
  int n = 0;
  for (int i = 0; i < 8; i++)
    for (int j = 0; j < 8; j++) n += dir_k(D, i, j) == k;
  return n;
}

// The cost of a direction's partial sums (direction.go:469-501).
template <int D>
__host__ __device__ __forceinline__ int32_t dir_cost_sums(const int32_t (&p)[15]) {
  if (D == 2 || D == 6) {
    int32_t s = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) s += p[i] * p[i];
    return s * 105;
  }
  if (D == 0 || D == 4) {
    const int32_t div[8] = {840, 420, 280, 210, 168, 140, 120, 105};
    int32_t s = 0;
#pragma unroll
    for (int i = 0; i < 7; i++) s += (p[i] * p[i] + p[14 - i] * p[14 - i]) * div[i];
    return s + p[7] * p[7] * 105;
  }
  return (p[3] * p[3] + p[4] * p[4] + p[5] * p[5] + p[6] * p[6] + p[7] * p[7]) * 105 +
         (p[0] * p[0] + p[10] * p[10]) * 420 + (p[1] * p[1] + p[9] * p[9]) * 210 +
         (p[2] * p[2] + p[8] * p[8]) * 140;
}

// The direction cost on packed sample pairs: w[i][m] holds samples (i, 2m) and
// (i, 2m + 1) of the block in its low and high halves, shifted to 8 bits.  Each pair is
// added as one 32-bit word into the accumulator of its even sample's index
// (the odd sample's index differs from it by the same -1, 0 or +1 for every
// pair of a direction), with the samples shifted to 8 bits and left biased
// by +128: a half never sums more than eight values below 256, so it never
// carries into the other.  The halves are then split into the partial sums,
// the bias taken off by each sum's sample count, and the cost formed from
// them, so the result is the same integer as summing the shifted, unbiased
// samples one by one.
template <int D>
__host__ __device__ __forceinline__ int32_t dir_cost_pairs(const uint32_t (&w)[8][4]) {
  constexpr int kDelta = dir_k(D, 0, 1) - dir_k(D, 0, 0);
  uint32_t acc[15];
#pragma unroll
  for (int k = 0; k < 15; k++) acc[k] = 0;
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int m = 0; m < 4; m++) acc[dir_k(D, i, 2 * m)] += w[i][m];
  int32_t p[15];
#pragma unroll
  for (int k = 0; k < 15; k++) {
    int32_t v = (int32_t)(acc[k] & 0xffffu);
    if (k - kDelta >= 0 && k - kDelta < 15) v += (int32_t)(acc[k - kDelta] >> 16);
    p[k] = v - 128 * dir_count(D, k);
  }
  return dir_cost_sums<D>(p);
}

// Two of the eight direction costs of a block staged as vertical pairs (blk:
// its first word), for group g of 0..3, into cost[0..7]: the block is read
// and masked once for both, and a light direction goes with a heavy one.  The
// words (2m, i) are the pairs (i, 2m), (i, 2m + 1) of the transposed block,
// and transposing a block turns direction D's lines into those of
// (8 - D) & 7 (dir_k(D, i, j) = dir_k((8 - D) & 7, j, i), for D = 4 read
// backwards, which its symmetric weights do not see).  mask: the sample bits
// that remain after the shift to 8 bits.
__device__ __forceinline__ void dir_costs_vert(int g, const uint32_t* blk, int shift, uint32_t mask, int32_t* cost) {
  uint32_t w[8][4];
#pragma unroll
  for (int m = 0; m < 4; m++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const uint4 q = *reinterpret_cast<const uint4*>(blk + 2 * m * kPW + 4 * h);
      w[4 * h][m] = (q.x >> shift) & mask, w[4 * h + 1][m] = (q.y >> shift) & mask;
      w[4 * h + 2][m] = (q.z >> shift) & mask, w[4 * h + 3][m] = (q.w >> shift) & mask;
    }
  switch (g) {
    case 0:
      cost[0] = dir_cost_pairs<0>(w);
      cost[2] = dir_cost_pairs<6>(w);
      break;
    case 1:
      cost[4] = dir_cost_pairs<4>(w);
      cost[6] = dir_cost_pairs<2>(w);
      break;
    case 2:
      cost[1] = dir_cost_pairs<7>(w);
      cost[3] = dir_cost_pairs<5>(w);
      break;
    default:
      cost[5] = dir_cost_pairs<3>(w);
      cost[7] = dir_cost_pairs<1>(w);
  }
}

__device__ __forceinline__ int constrain_shift(int threshold, int damping) {
  if (threshold == 0) return 0;
  return imax(damping - (31 - __clz(threshold)), 0);
}

__device__ __forceinline__ int adjust_strength(int strength, int32_t variance) {
  if (variance == 0) return 0;
  const int32_t v = variance >> 6;
  const int i = v != 0 ? imin(31 - __clz(v), 12) : 0;
  return (strength * (4 + i) + 8) >> 4;
}

// The same on pairs of plain integers below kVeryLarge.  constrain() has no
// short packed form in integers; its positive and its negative results are
// summed apart: with limit = max(0, thr - (|d| >> shift)) they are
// max(0, min(d, limit)) and max(0, min(-d, limit)).  Ten instructions a tap
// for two samples, where one sample took eight; 8 x 4K at 12 bits: 114.9 us a
// frame sample by sample, 91.4 so (103.2 with the constrain table this replaced).
__device__ __forceinline__ PairTap pair_tap_ints(int thr, int shift) {  // thr + 1, the shift's mask, the shift
  return PairTap{(uint32_t)(thr + 1) * 0x10001u, (0xffffu >> shift) * 0x10001u, (uint32_t)shift};
}

template <bool kPri, bool kSec>
__device__ __forceinline__ uint32_t pair_filter_ints(const uint32_t* c, const PairTap& pri, uint32_t w0, uint32_t w1,
                                                     const PairTap& sec, int2 po, int2 s0, int2 s1) {
  constexpr uint32_t kLeast = 0x80008000u, kOne = 0x00010001u, kNoneBits = (kVeryLarge - 1) * 0x10001u;
  const uint32_t x = c[0], minus = __viaddmax_s16x2(~x, kOne, kLeast);
  uint32_t hi = x, lo = x;
  auto range = [&](uint32_t a, uint32_t b) {
    if (kPri && kSec) {
      lo = __vimin3_u16x2(lo, a, b);
      hi = __vimax3_s16x2(hi, a & kNoneBits, b & kNoneBits);
    }
  };
  auto tap = [&](uint32_t a, const PairTap& t, uint32_t& up, uint32_t& down) {
    const uint32_t d = __viaddmax_s16x2(a, minus, kLeast), nd = ~d;
    const uint32_t m = __viaddmax_s16x2(nd, kOne, d);  // |d|
    const uint32_t limit = __viaddmax_s16x2(~((m >> t.o) & t.m), t.k, 0);
    up += __vimin_s16x2_relu(d, limit);
    down += __viaddmin_s16x2_relu(nd, kOne, limit);
  };
  uint32_t up = 0, down = 0;  // the weighted sums of the positive and the negative results
  if (kPri) {
    const uint32_t a0 = c[po.x], a1 = c[-po.x], a2 = c[po.y], a3 = c[-po.y];
    uint32_t u0 = 0, d0 = 0, u1 = 0, d1 = 0;
    tap(a0, pri, u0, d0);
    tap(a1, pri, u0, d0);
    tap(a2, pri, u1, d1);
    tap(a3, pri, u1, d1);
    up = u0 * w0 + u1 * w1;
    down = d0 * w0 + d1 * w1;
    range(a0, a1);
    range(a2, a3);
  }
  if (kSec) {
    const uint32_t b0 = c[s0.x], b1 = c[-s0.x], b2 = c[s1.x], b3 = c[-s1.x];
    uint32_t u = 0, d = 0;
    tap(b0, sec, u, d);
    tap(b1, sec, u, d);
    tap(b2, sec, u, d);
    tap(b3, sec, u, d);
    up += 2 * u;
    down += 2 * d;
    range(b0, b1);
    range(b2, b3);
    const uint32_t b4 = c[s0.y], b5 = c[-s0.y], b6 = c[s1.y], b7 = c[-s1.y];
    tap(b4, sec, up, down);
    tap(b5, sec, up, down);
    tap(b6, sec, up, down);
    tap(b7, sec, up, down);
    range(b4, b5);
    range(b6, b7);
  }
  // x + (8 + sum - (sum < 0) >> 4) rounds half away from zero.
  const uint32_t plus = __viaddmax_s16x2(up + kOne, ~down, 0), less = __viaddmax_s16x2(down + kOne, ~up, 0);
  const uint32_t add = ((plus + 0x00080008u) >> 4) & 0x0fff0fffu, sub = ((less + 0x00080008u) >> 4) & 0x0fff0fffu;
  uint32_t y = __viaddmax_s16x2(x + add + kOne, ~sub, kLeast);
  if (kPri && kSec) y = __vmins2(__vmaxs2(y, lo), hi);
  return y;
}

// The same one sample after the other in 32-bit integers, for any 16-bit
// samples, with absent ones as the reference has them: a tap of kVeryLarge
// that the clamp's maximum masks.  Packed integers cannot hold the differences
// of samples of 0x4000 and more, nor tell them from an absent one; the line
// lies at 12 bits, far enough below that no absent tap counts.  8 x 4K at 12
// bits with such a sample in every unit: 166 us a frame (91 without).
__device__ __forceinline__ PairTap pair_tap_wide(int thr, int shift) { return PairTap{(uint32_t)thr, (uint32_t)shift, 0}; }

template <bool kPri, bool kSec>
__device__ __forceinline__ uint32_t pair_filter_wide(const uint32_t* c, const PairTap& pri, int w0, int w1,
                                                     const PairTap& sec, int2 po, int2 s0, int2 s1) {
  uint32_t y2 = 0;
#pragma unroll 1
  for (int h = 0; h < 32; h += 16) {
    const int x = (c[0] >> h) & 0xffff;
    int lo = x, hi = x;
    auto tap = [&](int o, const PairTap& t) {
      const int v = (c[o] >> h) & 0xffff, d = v - x, m = abs(d);
      lo = imin(lo, v);
      hi = imax(hi, v & (kVeryLarge - 1));
      const int l = imin(imax((int)t.k - (m >> t.m), 0), m);
      return d < 0 ? -l : l;
    };
    int sum = 0;
    if (kPri) sum += w0 * (tap(po.x, pri) + tap(-po.x, pri)) + w1 * (tap(po.y, pri) + tap(-po.y, pri));
    if (kSec)
      sum += 2 * (tap(s0.x, sec) + tap(-s0.x, sec) + tap(s1.x, sec) + tap(-s1.x, sec)) + tap(s0.y, sec) +
             tap(-s0.y, sec) + tap(s1.y, sec) + tap(-s1.y, sec);
    int y = x + ((8 + sum - (sum < 0)) >> 4);
    // By the block's own strength: a masked sample can lie outside its taps' range.
    if (kPri && kSec && pri.k) y = imin(imax(y, lo), hi);
    y2 |= (uint32_t)(y & 0xffff) << h;
  }
  return y2;
}

// One direction's cost of a block staged as vertical pairs, any samples.
template <int D>
__device__ __forceinline__ int32_t dir_cost_wide(const uint32_t* blk, int shift) {
  int32_t p[15];
#pragma unroll
  for (int k = 0; k < 15; k++) p[k] = -128 * dir_count(D, k);
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) p[dir_k(D, i, j)] += (int32_t)((blk[i * kPW + j] & 0xffffu) >> shift);
  return dir_cost_sums<D>(p);
}

__device__ __forceinline__ int32_t dir_cost_wide_any(int d, const uint32_t* blk, int shift) {
  switch (d) {
    case 0: return dir_cost_wide<0>(blk, shift);
    case 1: return dir_cost_wide<1>(blk, shift);
    case 2: return dir_cost_wide<2>(blk, shift);
    case 3: return dir_cost_wide<3>(blk, shift);
    case 4: return dir_cost_wide<4>(blk, shift);
    case 5: return dir_cost_wide<5>(blk, shift);
    case 6: return dir_cost_wide<6>(blk, shift);
    default: return dir_cost_wide<7>(blk, shift);
  }
}

}  // namespace pf
