// pf_deblock.cu - AV1 deblocking on the GPU.
//
// Follows goav1's mask-driven deblock: internal/av1/decoder/
// postfilter_loopfilter_masks.go:229-268 (all vertical edges of the frame,
// then all horizontal edges; chroma gated off when both luma frame levels or
// the plane's base level are zero), postfilter_loopfilter_masks_sb.go:21-188
// (the per-128x128-region bitmask walk, edges outside the 4-aligned crop and
// column/row 0 dropped), loopfilter/sb.go:99-153 (width class from the mask
// lanes, level fallback to the left/above cell) and sb.go:156-446 (the
// 4/6/8/16-wide edge kernels).
//
// Same-direction edges never overlap (AV1 ties filter width to transform
// spacing), so every 4-sample edge unit of one direction is independent.
#include <cuda_fp16.h>

#include <type_traits>

#include "pf_common.cuh"

namespace pf {

// The inner samples of the unit's four lines: P[i][k] = p_k, Q[i][k] = q_k of
// line i (k < 4).  `q` points at q0 of line 0; dir 0 (vertical edge) steps
// lines by rows, dir 1 by columns.  With `words`, eight 4-sample words are
// read (4 bytes, or 8 for 16-bit samples): for a vertical edge the p3..p0
// and q0..q3 runs of each line, for a horizontal edge the four lines'
// samples of each of the eight rows; else sample by sample.
template <typename T>
__device__ __forceinline__ void lpf_inner(const T* q, int stride, int dir, bool words, int (&P)[4][4],
                                          int (&Q)[4][4]) {
  if (!words) {
    const int sa = dir == 0 ? stride : 1, sb = dir == 0 ? 1 : stride;
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        P[i][k] = q[i * sa - (k + 1) * sb];
        Q[i][k] = q[i * sa + k * sb];
      }
    return;
  }
  typedef typename std::conditional<sizeof(T) == 1, uint32_t, uint2>::type W;
  auto lane = [](const W& w, int j) -> int {
    if constexpr (sizeof(T) == 1) {
      return (w >> (8 * j)) & 0xff;
    } else {
      return ((j < 2 ? w.x : w.y) >> (16 * (j & 1))) & 0xffff;
    }
  };
  W v[8];
  if (dir == 0) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      v[2 * i] = *reinterpret_cast<const W*>(q + (int64_t)i * stride - 4);
      v[2 * i + 1] = *reinterpret_cast<const W*>(q + (int64_t)i * stride);
    }
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        P[i][k] = lane(v[2 * i], 3 - k);
        Q[i][k] = lane(v[2 * i + 1], k);
      }
  } else {
#pragma unroll
    for (int j = 0; j < 8; j++) v[j] = *reinterpret_cast<const W*>(q + (int64_t)(j - 4) * stride);
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int k = 0; k < 4; k++) {
        P[i][k] = lane(v[3 - k], i);
        Q[i][k] = lane(v[4 + k], i);
      }
  }
}

// loopfilter/sb.go:348-446 (lpfUnit16); reduces to lpfUnit8 at bd == 8.
// q points at q0 of the first line; sa steps along the edge, sb across it
// (both in elements).  One line after the other in 32-bit integers: 12-bit
// samples, planes whose rows are not aligned to four samples, and samples or
// levels beyond the format's range.
template <typename T>
__device__ __forceinline__ void lpf_unit(T* q, int sa, int sb, int bd, int E, int I, int H, int wd,
                                         const int (&P)[4][4], const int (&Q)[4][4]) {
  const int bd8 = bd - 8;
  const int F = 1 << bd8;
  E <<= bd8;
  I <<= bd8;
  H <<= bd8;
  const unsigned twoI = 2u * I, twoF = 2u * F, twoH = 2u * H;
  const int maxPix = (1 << bd) - 1;
  const int diffMin = -128 << bd8, diffMax = (128 << bd8) - 1;
  // The four lines never overlap, so the inner samples of all four (P, Q:
  // p3..q3) were read by the caller before any line is filtered.
#pragma unroll
  for (int i = 0; i < 4; i++, q += sa) {
    const int p1 = P[i][1], p0 = P[i][0], q0 = Q[i][0], q1 = Q[i][1];
    if ((unsigned)(p1 - p0 + I) > twoI || (unsigned)(q1 - q0 + I) > twoI ||
        abs(p0 - q0) * 2 + (abs(p1 - q1) >> 1) > E)
      continue;
    int p2 = 0, q2 = 0, p3 = 0, q3 = 0;
    if (wd > 4) {
      p2 = P[i][2];
      q2 = Q[i][2];
      if ((unsigned)(p2 - p1 + I) > twoI || (unsigned)(q2 - q1 + I) > twoI) continue;
      if (wd > 6) {
        p3 = P[i][3];
        q3 = Q[i][3];
        if ((unsigned)(p3 - p2 + I) > twoI || (unsigned)(q3 - q2 + I) > twoI) continue;
      }
    }
    bool flat8in = false;
    if (wd >= 6) {
      flat8in = (unsigned)(p2 - p0 + F) <= twoF && (unsigned)(p1 - p0 + F) <= twoF &&
                (unsigned)(q1 - q0 + F) <= twoF && (unsigned)(q2 - q0 + F) <= twoF;
      if (wd >= 8 && flat8in) flat8in = (unsigned)(p3 - p0 + F) <= twoF && (unsigned)(q3 - q0 + F) <= twoF;
    }
    if (flat8in) {
      if (wd >= 16) {
        const int p6 = q[-7 * sb], p5 = q[-6 * sb], p4 = q[-5 * sb];
        const int q4 = q[4 * sb], q5 = q[5 * sb], q6 = q[6 * sb];
        if ((unsigned)(p6 - p0 + F) <= twoF && (unsigned)(p5 - p0 + F) <= twoF &&
            (unsigned)(p4 - p0 + F) <= twoF && (unsigned)(q4 - q0 + F) <= twoF &&
            (unsigned)(q5 - q0 + F) <= twoF && (unsigned)(q6 - q0 + F) <= twoF) {
          // The twelve outputs as one running sum: each output's 16-weight
          // window differs from the previous one by two samples in, two out.
          int t = p6 * 7 + p5 * 2 + p4 * 2 + p3 + p2 + p1 + p0 + q0 + 8;
          q[-6 * sb] = (T)(t >> 4);
          t += p3 + q1 - 2 * p6;
          q[-5 * sb] = (T)(t >> 4);
          t += p2 + q2 - p6 - p5;
          q[-4 * sb] = (T)(t >> 4);
          t += p1 + q3 - p6 - p4;
          q[-3 * sb] = (T)(t >> 4);
          t += p0 + q4 - p6 - p3;
          q[-2 * sb] = (T)(t >> 4);
          t += q0 + q5 - p6 - p2;
          q[-sb] = (T)(t >> 4);
          t += q1 + q6 - p6 - p1;
          q[0] = (T)(t >> 4);
          t += q2 + q6 - p5 - p0;
          q[sb] = (T)(t >> 4);
          t += q3 + q6 - p4 - q0;
          q[2 * sb] = (T)(t >> 4);
          t += q4 + q6 - p3 - q1;
          q[3 * sb] = (T)(t >> 4);
          t += q5 + q6 - p2 - q2;
          q[4 * sb] = (T)(t >> 4);
          t += 2 * q6 - p1 - q3;
          q[5 * sb] = (T)(t >> 4);
          continue;
        }
      }
      if (wd >= 8) {
        q[-3 * sb] = (T)((p3 * 3 + p2 * 2 + p1 + p0 + q0 + 4) >> 3);
        q[-2 * sb] = (T)((p3 * 2 + p2 + p1 * 2 + p0 + q0 + q1 + 4) >> 3);
        q[-sb] = (T)((p3 + p2 + p1 + p0 * 2 + q0 + q1 + q2 + 4) >> 3);
        q[0] = (T)((p2 + p1 + p0 + q0 * 2 + q1 + q2 + q3 + 4) >> 3);
        q[sb] = (T)((p1 + p0 + q0 + q1 * 2 + q2 + q3 * 2 + 4) >> 3);
        q[2 * sb] = (T)((p0 + q0 + q1 + q2 * 2 + q3 * 3 + 4) >> 3);
        continue;
      }
      q[-2 * sb] = (T)((p2 * 3 + p1 * 2 + p0 * 2 + q0 + 4) >> 3);
      q[-sb] = (T)((p2 + p1 * 2 + p0 * 2 + q0 * 2 + q1 + 4) >> 3);
      q[0] = (T)((p1 + p0 * 2 + q0 * 2 + q1 * 2 + q2 + 4) >> 3);
      q[sb] = (T)((p0 + q0 * 2 + q1 * 2 + q2 * 3 + 4) >> 3);
      continue;
    }
    const bool hev = (unsigned)(p1 - p0 + H) > twoH || (unsigned)(q1 - q0 + H) > twoH;
    int f;
    if (hev)
      f = imin(imax(imin(imax(p1 - q1, diffMin), diffMax) + 3 * (q0 - p0), diffMin), diffMax);
    else
      f = imin(imax(3 * (q0 - p0), diffMin), diffMax);
    const int f1 = imin(f + 4, diffMax) >> 3;
    const int f2 = imin(f + 3, diffMax) >> 3;
    q[-sb] = (T)imin(imax(p0 + f2, 0), maxPix);
    q[0] = (T)imin(imax(q0 - f1, 0), maxPix);
    if (!hev) {
      f = (f1 + 1) >> 1;
      q[-2 * sb] = (T)imin(imax(p1 + f, 0), maxPix);
      q[sb] = (T)imin(imax(q1 - f, 0), maxPix);
    }
  }
}

// The unit's four lines as two pairs, both lines of a pair in one register
// (16 bits each): every sample below 2,048 is, as a bit pattern, the half
// precision number sample * 2^-24 (subnormal up to 1,023), and sums,
// differences and multiples within +-2,047 of that unit are exact.  So the
// masks' differences are packed half additions with absolute values as
// operand modifiers, the narrow filter's shifts are multiplications whose
// rounding to the unit is the shift's (the numerator is kept odd, so a tie
// never occurs), and the wide filters' sums are 32-bit integer additions of
// the same registers.  Against the line-by-line integers, one thread
// a unit both: 12.2 us to 9.0 for both directions of a 1920x1080 8-bit frame
// (of 60), 48.9 to 35.9 for a 3840x2160 10-bit one (of 8).
__device__ __forceinline__ __half2 lpf_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t lpf_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ uint32_t lpf_le(__half2 a, uint32_t b) { return __hle2_mask(a, lpf_h2(b)); }
// a where m's bits are set, else b.
__device__ __forceinline__ uint32_t lpf_pick(uint32_t m, uint32_t a, uint32_t b) { return (a & m) | (b & ~m); }
__device__ __forceinline__ __half2 lpf_gap(__half2 a, __half2 b, __half2 c, __half2 d) {
  return __hmax2(__habs2(__hsub2(a, b)), __habs2(__hsub2(c, d)));
}

// A unit's limits, both halves alike.
struct LpfLimits {
  uint32_t edge, inner, hev, flat;  // 2 * E + 1; I; H; the flat tests' bound
  uint32_t lo, hi, top;  // narrow filter: 2 * diffMin, 2 * diffMax - 7; the largest sample
};

__device__ __forceinline__ uint32_t lpf_both(int v) { return (uint32_t)v * 0x10001u; }

// Four samples of each side for the two lines of pair j from the words read
// by lpf_words: s[0..7] = p3..p0, q0..q3.
template <typename T, int kDir, typename W>
__device__ __forceinline__ void lpf_split(const W (&w)[8], int j, uint32_t (&s)[8]) {
  if constexpr (kDir == 1) {
#pragma unroll
    for (int k = 0; k < 8; k++) {
      if constexpr (sizeof(T) == 1)
        s[k] = __byte_perm(w[k], 0, j == 0 ? 0x4140 : 0x4342);
      else
        s[k] = j == 0 ? w[k].x : w[k].y;
    }
  } else {
#pragma unroll
    for (int side = 0; side < 2; side++) {
      const W a = w[4 * j + side], b = w[4 * j + 2 + side];
      uint32_t* o = s + 4 * side;
      if constexpr (sizeof(T) == 1) {
        const uint32_t t0 = __byte_perm(a, b, 0x5140), t1 = __byte_perm(a, b, 0x7362);
        o[0] = __byte_perm(t0, 0, 0x4140);
        o[1] = __byte_perm(t0, 0, 0x4342);
        o[2] = __byte_perm(t1, 0, 0x4140);
        o[3] = __byte_perm(t1, 0, 0x4342);
      } else {
        o[0] = __byte_perm(a.x, b.x, 0x5410);
        o[1] = __byte_perm(a.x, b.x, 0x7632);
        o[2] = __byte_perm(a.y, b.y, 0x5410);
        o[3] = __byte_perm(a.y, b.y, 0x7632);
      }
    }
  }
}

// Samples k and k + 1 of the pair's lines, for a vertical edge: line 0's two
// samples and line 1's.
template <typename T>
struct LpfTwo {
  typedef uint32_t V;
};
template <>
struct LpfTwo<uint8_t> {
  typedef uint16_t V;
};
template <typename T>
__device__ __forceinline__ void lpf_store_two(T* line0, T* line1, uint32_t s0, uint32_t s1) {
  typedef typename LpfTwo<T>::V V;
  if constexpr (sizeof(T) == 1) {
    const uint32_t c = __byte_perm(s0, s1, 0x6240);
    *reinterpret_cast<V*>(line0) = (V)c;
    *reinterpret_cast<V*>(line1) = (V)(c >> 16);
  } else {
    *reinterpret_cast<V*>(line0) = __byte_perm(s0, s1, 0x5410);
    *reinterpret_cast<V*>(line1) = __byte_perm(s0, s1, 0x7632);
  }
}
template <typename T>
__device__ __forceinline__ void lpf_store_four(T* line0, T* line1, const uint32_t* s) {
  if constexpr (sizeof(T) == 1) {
    const uint32_t a = __byte_perm(s[0], s[1], 0x6240), b = __byte_perm(s[2], s[3], 0x6240);
    *reinterpret_cast<uint32_t*>(line0) = __byte_perm(a, b, 0x5410);
    *reinterpret_cast<uint32_t*>(line1) = __byte_perm(a, b, 0x7632);
  } else {
    *reinterpret_cast<uint2*>(line0) = make_uint2(__byte_perm(s[0], s[1], 0x5410), __byte_perm(s[2], s[3], 0x5410));
    *reinterpret_cast<uint2*>(line1) = make_uint2(__byte_perm(s[0], s[1], 0x7632), __byte_perm(s[2], s[3], 0x7632));
  }
}
// The pair's two samples of one row, for a horizontal edge.
template <typename T>
__device__ __forceinline__ void lpf_store_row(T* row, uint32_t s) {
  if constexpr (sizeof(T) == 1)
    *reinterpret_cast<uint16_t*>(row) = (uint16_t)__byte_perm(s, 0, 0x4420);
  else
    *reinterpret_cast<uint32_t*>(row) = s;
}

// The 14-tap filter of the pair's lines where flat: o holds p3..q3, s takes
// the new ones, the outer samples are read and written here.  `q` points at
// q0 of the pair's first line.
template <typename T, int kDir>
__device__ __forceinline__ void lpf_wide(T* q, int stride, const LpfLimits& l, uint32_t flat,
                                             const uint32_t (&o)[8], uint32_t (&s)[8]) {
  uint32_t p6, p5, p4, q4, q5, q6;
  typedef typename std::conditional<sizeof(T) == 1, uint32_t, uint2>::type W;
  W w[4];
  if constexpr (kDir == 0) {
    w[0] = *reinterpret_cast<const W*>(q - 8);
    w[1] = *reinterpret_cast<const W*>(q + stride - 8);
    w[2] = *reinterpret_cast<const W*>(q + 4);
    w[3] = *reinterpret_cast<const W*>(q + stride + 4);
    if constexpr (sizeof(T) == 1) {
      const uint32_t t0 = __byte_perm(w[0], w[1], 0x5140), t1 = __byte_perm(w[0], w[1], 0x7362);
      const uint32_t u0 = __byte_perm(w[2], w[3], 0x5140), u1 = __byte_perm(w[2], w[3], 0x7362);
      p6 = __byte_perm(t0, 0, 0x4342), p5 = __byte_perm(t1, 0, 0x4140), p4 = __byte_perm(t1, 0, 0x4342);
      q4 = __byte_perm(u0, 0, 0x4140), q5 = __byte_perm(u0, 0, 0x4342), q6 = __byte_perm(u1, 0, 0x4140);
    } else {
      p6 = __byte_perm(w[0].x, w[1].x, 0x7632);
      p5 = __byte_perm(w[0].y, w[1].y, 0x5410), p4 = __byte_perm(w[0].y, w[1].y, 0x7632);
      q4 = __byte_perm(w[2].x, w[3].x, 0x5410), q5 = __byte_perm(w[2].x, w[3].x, 0x7632);
      q6 = __byte_perm(w[2].y, w[3].y, 0x5410);
    }
  } else {
    auto row = [&](int k) -> uint32_t {
      if constexpr (sizeof(T) == 1)
        return __byte_perm(*reinterpret_cast<const uint16_t*>(q + (int64_t)k * stride), 0, 0x4140);
      else
        return *reinterpret_cast<const uint32_t*>(q + (int64_t)k * stride);
    };
    p6 = row(-7), p5 = row(-6), p4 = row(-5), q4 = row(4), q5 = row(5), q6 = row(6);
  }
  const __half2 p0h = lpf_h2(o[3]), q0h = lpf_h2(o[4]);
  const __half2 d = __hmax2(__hmax2(lpf_gap(lpf_h2(p6), p0h, lpf_h2(q6), q0h), lpf_gap(lpf_h2(p5), p0h, lpf_h2(q5), q0h)),
                            lpf_gap(lpf_h2(p4), p0h, lpf_h2(q4), q0h));
  const uint32_t m = lpf_le(d, l.flat) & flat;
  if (!m) return;
  // The twelve outputs as one running sum: each output's 16-weight window
  // differs from the previous one by two samples in, two out.  Both lines at
  // once: no half exceeds 16 * 1023 + 8.
  const uint32_t p3 = o[0], p2 = o[1], p1 = o[2], p0 = o[3], q0 = o[4], q1 = o[5], q2 = o[6], q3 = o[7];
  // For 8-bit samples only each half's low byte is used.
  auto out = [](uint32_t t) { return sizeof(T) == 1 ? t >> 4 : (t >> 4) & 0x0fff0fff; };
  uint32_t t = p6 * 7 + (p5 + p4) * 2 + p3 + p2 + p1 + p0 + q0 + 0x00080008u;
  const uint32_t n5 = out(t);
  t += p3 + q1 - 2 * p6;
  const uint32_t n4 = out(t);
  t += p2 + q2 - p6 - p5;
  s[0] = lpf_pick(m, out(t), s[0]);
  t += p1 + q3 - p6 - p4;
  s[1] = lpf_pick(m, out(t), s[1]);
  t += p0 + q4 - p6 - p3;
  s[2] = lpf_pick(m, out(t), s[2]);
  t += q0 + q5 - p6 - p2;
  s[3] = lpf_pick(m, out(t), s[3]);
  t += q1 + q6 - p6 - p1;
  s[4] = lpf_pick(m, out(t), s[4]);
  t += q2 + q6 - p5 - p0;
  s[5] = lpf_pick(m, out(t), s[5]);
  t += q3 + q6 - p4 - q0;
  s[6] = lpf_pick(m, out(t), s[6]);
  t += q4 + q6 - p3 - q1;
  s[7] = lpf_pick(m, out(t), s[7]);
  t += q5 + q6 - p2 - q2;
  const uint32_t m4 = out(t);
  t += 2 * q6 - p1 - q3;
  const uint32_t m5 = out(t);
  p5 = lpf_pick(m, n5, p5), p4 = lpf_pick(m, n4, p4);
  q4 = lpf_pick(m, m4, q4), q5 = lpf_pick(m, m5, q5);
  if constexpr (kDir == 0) {
    lpf_store_two(q - 6, q + stride - 6, p5, p4);
    lpf_store_two(q + 4, q + stride + 4, q4, q5);
  } else {
    lpf_store_row(q - (int64_t)6 * stride, p5);
    lpf_store_row(q - (int64_t)5 * stride, p4);
    lpf_store_row(q + (int64_t)4 * stride, q4);
    lpf_store_row(q + (int64_t)5 * stride, q5);
  }
}

// The two lines of one pair under the kWd-sample edge filter: s = p3..q3,
// replaced by the filtered samples.  Returns the lines' filter mask; `wide`
// becomes the mask of lines whose samples beyond p1 and q1 changed.
template <typename T, int kDir, int kWd>
__device__ __forceinline__ uint32_t lpf_pair(T* q, int stride, const LpfLimits& l, uint32_t (&s)[8], uint32_t& wide) {
  const __half2 p3 = lpf_h2(s[0]), p2 = lpf_h2(s[1]), p1 = lpf_h2(s[2]), p0 = lpf_h2(s[3]);
  const __half2 q0 = lpf_h2(s[4]), q1 = lpf_h2(s[5]), q2 = lpf_h2(s[6]), q3 = lpf_h2(s[7]);
  const __half2 d = __hsub2(q0, p0), e = __hsub2(p1, q1);
  const __half2 near = lpf_gap(p1, p0, q1, q0);
  __half2 in = near;
  if (kWd > 4) in = __hmax2(in, lpf_gap(p2, p1, q2, q1));
  if (kWd > 6) in = __hmax2(in, lpf_gap(p3, p2, q3, q2));
  // 2 * |d| + (|e| >> 1) <= E  <=>  4 * |d| + |e| <= 2 * E + 1 (= l.edge).
  const uint32_t on =
      lpf_le(in, l.inner) & lpf_le(__hfma2(__habs2(d), lpf_h2(0x44004400u), __habs2(e)), l.edge);
  uint32_t flat = 0;
  if (kWd > 4) {
    __half2 fl = __hmax2(near, lpf_gap(p2, p0, q2, q0));
    if (kWd > 6) fl = __hmax2(fl, lpf_gap(p3, p0, q3, q0));
    flat = on & lpf_le(fl, l.flat);
  }
  wide = 0;
  if (!on) return 0;
  uint32_t nm = on & ~flat;
  uint32_t o[8];
#pragma unroll
  for (int k = 0; k < 8; k++) o[k] = s[k];
  if (nm) {
    const __half2 one = lpf_h2(0x00010001u), sixteenth = lpf_h2(0x2c002c00u);
    const uint32_t hev = ~lpf_le(near, l.hev);
    const __half2 lo = lpf_h2(l.lo), hi = lpf_h2(l.hi);
    // Doubled: base = clamp(p1 - q1) of the lines with a high edge variance,
    // f = clamp(base + 3 * (q0 - p0)); g1 = 2 * min(f + 4, max) - 7 and g2 =
    // 2 * min(f + 3, max) - 7, so that g / 16 rounds to the shift by three.
    const __half2 e2 = __hadd2(e, e);
    const __half2 base = __hmax2(__hmin2(e2, __hadd2(hi, lpf_h2(0x00070007u))), lo);
    const __half2 f = __hmax2(__hfma2(d, lpf_h2(0x46004600u), lpf_h2(lpf_bits(base) & hev)), lo);
    const __half2 g1 = __hmin2(__hadd2(f, one), hi), g2 = __hmin2(__hsub2(f, one), hi);
    const __half2 f1 = __hmul2(g1, sixteenth);
    // (f1 + 1) >> 1 as (2 * f1 + 1) / 4, rounded.
    const __half2 r = __hfma2(f1, lpf_h2(0x40004000u), one);
    auto clip = [&](__half2 v) { return __vimin_s16x2_relu(lpf_bits(v), l.top); };
    s[3] = lpf_pick(nm, clip(__hfma2(g2, sixteenth, p0)), s[3]);
    s[4] = lpf_pick(nm, clip(__hfma2(g1, lpf_h2(0xac00ac00u), q0)), s[4]);
    nm &= ~hev;
    s[2] = lpf_pick(nm, clip(__hfma2(r, lpf_h2(0x34003400u), p1)), s[2]);
    s[5] = lpf_pick(nm, clip(__hfma2(r, lpf_h2(0xb400b400u), q1)), s[5]);
  }
  if (flat) {
    auto out = [](uint32_t t) { return sizeof(T) == 1 ? t >> 3 : (t >> 3) & 0x1fff1fff; };
    if (kWd >= 8) {
      uint32_t t = o[0] * 3 + o[1] * 2 + o[2] + o[3] + o[4] + 0x00040004u;
      s[1] = lpf_pick(flat, out(t), s[1]);
      t += o[2] + o[5] - o[0] - o[1];
      s[2] = lpf_pick(flat, out(t), s[2]);
      t += o[3] + o[6] - o[0] - o[2];
      s[3] = lpf_pick(flat, out(t), s[3]);
      t += o[4] + o[7] - o[0] - o[3];
      s[4] = lpf_pick(flat, out(t), s[4]);
      t += o[5] + o[7] - o[1] - o[4];
      s[5] = lpf_pick(flat, out(t), s[5]);
      t += o[6] + o[7] - o[2] - o[5];
      s[6] = lpf_pick(flat, out(t), s[6]);
      if (kWd == 16) lpf_wide<T, kDir>(q, stride, l, flat, o, s);
      wide = flat;
    } else {
      uint32_t t = o[1] * 3 + (o[2] + o[3]) * 2 + o[4] + 0x00040004u;
      s[2] = lpf_pick(flat, out(t), s[2]);
      t += o[4] + o[5] - o[1] * 2;
      s[3] = lpf_pick(flat, out(t), s[3]);
      t += o[5] + o[6] - o[1] - o[2];
      s[4] = lpf_pick(flat, out(t), s[4]);
      t += o[6] * 2 - o[2] - o[3];
      s[5] = lpf_pick(flat, out(t), s[5]);
    }
  }
  return on;
}

// The bits set in any of the six outer samples on each line of a 14-tap
// unit (and p7 / q7 of a vertical edge's words).
template <int kDir>
__device__ __forceinline__ uint32_t lpf_outer_bits(const uint16_t* q, int stride) {
  uint32_t b = 0;
  auto at = [&](const uint16_t* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    b |= v.x | v.y;
  };
  if constexpr (kDir == 0) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      at(q + (int64_t)i * stride - 8);
      at(q + (int64_t)i * stride + 4);
    }
  } else {
#pragma unroll
    for (int k = 4; k < 7; k++) {
      at(q + (int64_t)k * stride);
      at(q - (int64_t)(k + 1) * stride);
    }
  }
  return b;
}

template <typename T, int kDir, int kWd, typename W>
__device__ __forceinline__ void lpf_unit_pairs(T* q, int stride, const LpfLimits& l, const W (&w)[8]) {
#pragma unroll
  for (int j = 0; j < 2; j++) {
    uint32_t s[8], wide;
    lpf_split<T, kDir>(w, j, s);
    T* line = kDir == 0 ? q + 2 * j * stride : q + 2 * j;
    if (!lpf_pair<T, kDir, kWd>(line, stride, l, s, wide)) continue;
    // A word of both pairs' or of more samples than changed is written only
    // where no other edge of this direction has a part in it: p3..p0 and
    // q0..q3 lie in transforms of at least eight samples where the class is.
    if constexpr (kDir == 0) {
      if (wide) {
        lpf_store_four(line - 4, line + stride - 4, s);
        lpf_store_four(line, line + stride, s + 4);
      } else {
        lpf_store_two(line - 2, line + stride - 2, s[2], s[3]);
        lpf_store_two(line, line + stride, s[4], s[5]);
      }
    } else {
      if (wide) {
        if (kWd == 16) lpf_store_row(line - (int64_t)4 * stride, s[0]);
        lpf_store_row(line - (int64_t)3 * stride, s[1]);
        lpf_store_row(line + (int64_t)2 * stride, s[6]);
        if (kWd == 16) lpf_store_row(line + (int64_t)3 * stride, s[7]);
      }
      lpf_store_row(line - (int64_t)2 * stride, s[2]);
      lpf_store_row(line - stride, s[3]);
      lpf_store_row(line, s[4]);
      lpf_store_row(line + stride, s[5]);
    }
  }
}

// loopfilter/threshold.go:18-47.
__device__ __forceinline__ int deblock_limit(const LfArgs& a, int L) {
  const int sh = a.sharpness;
  int limit = L >> ((sh > 0) + (sh > 4));
  if (sh > 0 && limit > 9 - sh) limit = 9 - sh;
  return limit < 1 ? 1 : limit;
}

// Whether the plane's rows start on 4-sample boundaries.
template <typename T>
__device__ __forceinline__ bool db_words(const DPlane& pl) {
  return (((uintptr_t)pl.ptr | (uintptr_t)pl.stride) & (4 * sizeof(T) - 1)) == 0;
}

// The masks are trusted like the reference trusts them, but a 14-tap edge
// whose outer taps would leave the allocated plane (only a malformed mask can
// ask for one; the reference would fault on it) is skipped instead of touched.
__device__ __forceinline__ bool db_wide_fits(const DPlane& pl, int dir, int c4, int r4) {
  const int at = (dir == 0 ? c4 : r4) * 4;
  return at - 7 >= 0 && at + 6 < (dir == 0 ? pl.aw : pl.ah);
}

// One unit line by line.
template <typename T>
__device__ __noinline__ void deblock_unit_lines(const DFrame& f, const LfArgs& a, int dir, int plane, int c4, int r4,
                                                int L, int wd) {
  const DPlane& pl = f.pl[plane];
  if (wd == 16 && !db_wide_fits(pl, dir, c4, r4)) return;
  const int stride = (int)(pl.stride / sizeof(T)), limit = deblock_limit(a, L);
  T* q = row_ptr<T>(pl, r4 * 4) + c4 * 4;
  int P[4][4], Q[4][4];
  lpf_inner<T>(q, stride, dir, db_words<T>(pl), P, Q);
  lpf_unit<T>(q, dir == 0 ? stride : 1, dir == 0 ? 1 : stride, f.bd, 2 * (L + 2) + limit, limit, L >> 4, wd, P, Q);
}

// One 4x4 unit (c4, r4) of `plane` with an edge of class kWd and level L: dir
// 0 filters its left (vertical) edge, dir 1 its top (horizontal) edge.  Its
// words: for a vertical edge line i's p3..p0 and q0..q3 as 2 i and 2 i + 1,
// for a horizontal one the rows p3..q3.  False if the samples or the level
// are beyond the packed forms.
template <typename T, int dir, int kWd, typename W>
__device__ __forceinline__ bool deblock_unit(const DFrame& f, const LfArgs& a, int plane, int c4, int r4, int L,
                                             const W (&w)[8]) {
  const DPlane& pl = f.pl[plane];
  if (kWd == 16 && !db_wide_fits(pl, dir, c4, r4)) return true;
  const int stride = (int)(pl.stride / sizeof(T));
  T* q = row_ptr<T>(pl, r4 * 4) + c4 * 4;
  // Those hold for the samples and levels of a bitstream; a 10-bit frame's
  // 16-bit words can hold more.
  if (L > 63) return false;
  // The outer samples' word q4..q7: q7, which no filter needs, can be past the
  // allocated row (a malformed mask again).
  if (kWd == 16 && dir == 0 && c4 * 4 + 8 > pl.aw) return false;
  if constexpr (sizeof(T) == 2) {
    uint32_t over = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) over |= w[j].x | w[j].y;
    if (kWd == 16) over |= lpf_outer_bits<dir>(q, stride);
    if (over & 0xfc00fc00u) return false;
  }
  const int bd = sizeof(T) == 1 ? 8 : 10, up = bd - 8, limit = deblock_limit(a, L);
  LpfLimits l;
  l.edge = lpf_both(((4 * (L + 2) + 2 * limit) << up) + 1);
  l.inner = lpf_both(limit << up);
  l.hev = lpf_both((L >> 4) << up);
  l.flat = lpf_both(1 << up);
  l.lo = lpf_both(0x8000 | (256 << up));
  l.hi = lpf_both((256 << up) - 9);
  l.top = lpf_both((1 << bd) - 1);
  lpf_unit_pairs<T, dir, kWd>(q, stride, l, w);
  return true;
}

// Batched deblocking: each work item is one tile of 32 x 8 * kU edge units of
// one plane of one frame, kU units a thread.  The threads copy the tile's
// samples and levels to shared memory, look up their units' classes and list
// the units with an edge by class; the warps then take the lists 32 units at
// a time, one class a warp, so no lane waits for a wider filter's path than
// its own, nor for units without an edge (about half of them).  A CTA's start
// and its way to the tile cost as much as 256 units' filtering, so a tile is
// 1,024 units except where a call has few (db_units_log2).  From one
// thread a unit: 9.0 us to 6.7 for both directions of a 1920x1080 8-bit frame
// (of 60), 35.9 to 29.4 for a 3840x2160 10-bit one (of 8).  Of the 6.7, 2.6
// are a CTA's start, its way to the tile and the copies (the passes move 6.2
// MB each), 1.1 the lists and 3.0 the filters.  Three or five CTAs an SM: 7.2
// and 6.4 (10-bit 30.7 and 29.6).
constexpr int kDbPitch = 32 * 8 + 16;  // bytes of the widest row: 16-bit samples, 16 bytes of halo
struct DbShared {
  int n[3];
  uint16_t unit[2][1024];  // class 0 upwards and class 2 downwards; class 1
  uint8_t level[33 * 33];
  uint4 rows[(128 * kDbPitch) / 16];
};

__device__ __forceinline__ void db_copy16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
template <int kBytes>
__device__ __forceinline__ void db_copy(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(kBytes) : "memory");
}

struct DbTile {
  int plane, tx, ty;
};

__device__ __forceinline__ DbTile db_locate(const FrameJob& J, int local) {
  int plane = 0;
  while (plane < 2 && local >= J.db_tx[plane] * J.db_ty[plane]) {
    local -= J.db_tx[plane] * J.db_ty[plane];
    plane++;
  }
  const int ty = local / J.db_tx[plane];
  return DbTile{plane, local - ty * J.db_tx[plane], ty};
}

template <typename T, int kDir>
__device__ __forceinline__ void db_tile(const FrameJob& J, const DbTile& t, DbShared& sh) {
  if (J.lf.gate_chroma[t.plane]) return;
  constexpr int kWord = 4 * sizeof(T), kRun = 16 / sizeof(T);  // bytes of a unit's row; samples in 16 bytes
  constexpr int kPitch = 32 * kWord + (kDir == 0 ? 16 : 0);
  constexpr int kHalo = kDir == 0 ? 16 : 4 * kPitch;  // left: 16 bytes a row; above: four rows
  static_assert(132 * 32 * 8 <= 128 * kDbPitch, "rows with the halo above");
  const int lgU = J.db_tile, th = 8 << lgU;  // units a thread; unit rows of the tile
  const int c0 = t.tx * 32, r0 = t.ty * th;
  const int at = threadIdx.x, lane = at & 31;
  const LfArgs& a = J.lf;
  const DPlane& pl = J.io.pl[t.plane];
  const int ssx = t.plane ? J.io.ssx : 0, ssy = t.plane ? J.io.ssy : 0;
  const bool pairs = J.io.bd <= 10 && db_words<T>(pl);
  if (pairs) {
    const uint32_t rows = (uint32_t)__cvta_generic_to_shared(sh.rows);
    const int w = pl.aw - c0 * 4, h = imin(pl.ah - r0 * 4, th * 4);  // samples from the tile's corner on
    const T* src0 = row_ptr<T>(pl, r0 * 4) + c0 * 4;
    const bool wide = (((uintptr_t)pl.ptr | (uintptr_t)pl.stride) & 15) == 0;
    // 16 bytes (or those left of the row) at sample x of row y.
    auto copy = [&](int x, int y, uint32_t dst) {
      const T* src = reinterpret_cast<const T*>(reinterpret_cast<const char*>(src0) + (int64_t)y * pl.stride) + x;
      if (wide && x + kRun <= w) {
        db_copy16(dst, src);
      } else {
#pragma unroll
        for (int i = 0; i < 16 / kWord; i++)
          if (x + 4 * i + 4 <= w) db_copy<kWord>(dst + i * kWord, src + 4 * i);
      }
    };
    constexpr int kLg = sizeof(T) == 1 ? 3 : 4;  // 16-byte runs of a row
    const int first = kDir == 1 && r0 > 0 ? -4 : 0;
    const int run = at & ((1 << kLg) - 1);
    for (int y = first + (at >> kLg); y < h; y += 256 >> kLg)
      copy(run * kRun, y, rows + kHalo + y * kPitch + run * 16);
    if (kDir == 0 && c0 > 0)
      for (int y = at; y < h; y += 256) copy(-kRun, y, rows + y * kPitch);
  }
  if (at < 3) sh.n[at] = 0;
  // The units' classes, kU neighbours along the edge a thread: they share
  // the mask words, the widest lane with a unit's bit set counts.  Edge
  // positions are inside the 4-aligned crop (frameWorkLoopFilterPlaneSize),
  // and p3..q3 of the four lines inside the allocated plane for every unit
  // past the first column / row.
  const int lc = kDir == 0 ? lane : (at & ((32 >> lgU) - 1)) << lgU;
  const int lr = kDir == 0 ? (at >> 5) << lgU : at >> (5 - lgU);
  const int w4 = imin((((J.io.width + ssx) >> ssx) + 3) >> 2, pl.aw >> 2);
  const int h4 = imin((((J.io.height + ssy) >> ssy) + 3) >> 2, pl.ah >> 2);
  const int comp = t.plane == 0 ? kDir : t.plane + 1;
  unsigned bits[3] = {0, 0, 0};  // the thread's units by class
  int total = 0;
  if (c0 + lc < w4 && r0 + lr < h4) {
    const int c4 = c0 + lc, r4 = r0 + lr;
    const int lgW = 5 - ssx, lgH = 5 - ssy;
    const int pcol = c4 & ((1 << lgW) - 1), prow = r4 & ((1 << lgH) - 1);
    const uint16_t* region = a.masks + (size_t)((r4 >> lgH) * a.sb128_w + (c4 >> lgW)) * PF_LF_MASK_WORDS;
    const int pos = kDir == 0 ? pcol : prow, bit = kDir == 0 ? prow : pcol;
    const int word = 4 - (kDir == 0 ? ssy : ssx);  // log2 of a mask word's units
    const int half = bit >> word, b = bit & ((1 << word) - 1);
    const int nclass = t.plane ? 2 : 3;
    const uint16_t* m = region + (t.plane ? 384 : 0) + ((kDir * 32 + pos) * nclass) * 2 + half;
    const unsigned m0 = __ldg(&m[0]), m1 = __ldg(&m[2]), m2 = t.plane ? 0 : __ldg(&m[4]);
    const uint8_t* lv = a.level_cache + 4 * ((size_t)r4 * a.mi_cols + c4) + comp;
    // Units inside the frame, without the first column's / row's.
    const int along = kDir == 0 ? h4 - r4 : w4 - c4;
    const unsigned in = (1u << imin(1 << lgU, along)) - 1u;
#pragma unroll
    for (int u = 0; u < 4; u++)
      if ((in >> u) & 1)
        sh.level[(lr + 1 + (kDir == 0 ? u : 0)) * 33 + lc + 1 + (kDir == 0 ? 0 : u)] =
            __ldg(&lv[4 * u * (kDir == 0 ? a.mi_cols : 1)]);
    if ((kDir == 0 ? c4 : r4) > 0) {
      bits[2] = (m2 >> b) & in;
      bits[1] = (m1 >> b) & in & ~bits[2];
      bits[0] = (m0 >> b) & in & ~(bits[2] | bits[1]);
      total = __popc(bits[0]) | __popc(bits[1]) << 10 | __popc(bits[2]) << 20;
    }
  }
  // The halo's levels.
  if (kDir == 0 ? (c0 > 0 && at < th && r0 + at < h4) : (r0 > 0 && at < 32 && c0 + at < w4)) {
    const int c4 = kDir == 0 ? c0 - 1 : c0 + at, r4 = kDir == 0 ? r0 + at : r0 - 1;
    sh.level[kDir == 0 ? (at + 1) * 33 : at + 1] = __ldg(&a.level_cache[4 * ((size_t)r4 * a.mi_cols + c4) + comp]);
  }
  int pre = total;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(~0u, pre, d);
    if (lane >= d) pre += v;
  }
  __syncthreads();
  int base[3] = {0, 0, 0};
  if (lane == 31) {
#pragma unroll
    for (int c = 0; c < 3; c++) base[c] = atomicAdd(&sh.n[c], (pre >> (10 * c)) & 1023);
  }
  pre -= total;
#pragma unroll
  for (int c = 0; c < 3; c++) {
    int i = __shfl_sync(~0u, base[c], 31) + ((pre >> (10 * c)) & 1023);
    for (unsigned m = bits[c]; m; m &= m - 1, i++) {
      const int u = __ffs(m) - 1;
      const int id = (lr + (kDir == 0 ? u : 0)) * 32 + lc + (kDir == 0 ? 0 : u);
      sh.unit[c == 1][c == 2 ? 1023 - i : i] = (uint16_t)id;
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  const int n0 = sh.n[0], n1 = sh.n[1], n2 = sh.n[2];
  const int w2 = (n2 + 31) >> 5, w1 = w2 + ((n1 + 31) >> 5), w0 = w1 + ((n0 + 31) >> 5);
  for (int w = at >> 5; w < w0; w += 8) {
    const int c = w < w2 ? 2 : w < w1 ? 1 : 0;
    const int i = (w - (c == 2 ? 0 : c == 1 ? w2 : w1)) * 32 + lane;
    if (i >= (c == 2 ? n2 : c == 1 ? n1 : n0)) continue;
    const int id = sh.unit[c == 1][c == 2 ? 1023 - i : i];
    const int uc = id & 31, ur = id >> 5;
    const int c4 = c0 + uc, r4 = r0 + ur;
    // The level: the cell's, or where that is 0 its left / upper neighbour's
    // (sb.go:122-128, :142-148).
    const uint8_t* lv = &sh.level[(ur + 1) * 33 + uc + 1];
    const int L = lv[0] != 0 ? lv[0] : lv[kDir == 0 ? -1 : -33];
    if (L == 0) continue;
    bool done = false;
    if (pairs) {
      typedef typename std::conditional<sizeof(T) == 1, uint32_t, uint2>::type W;
      W v[8];
      const char* src = reinterpret_cast<const char*>(sh.rows) + 4 * ur * kPitch + uc * kWord + (kDir == 0 ? 16 - kWord : 0);
#pragma unroll
      for (int j = 0; j < 8; j++)
        v[j] = *reinterpret_cast<const W*>(src + (kDir == 0 ? (j >> 1) * kPitch + (j & 1) * kWord : j * kPitch));
      if (c == 0)
        done = deblock_unit<T, kDir, 4>(J.io, a, t.plane, c4, r4, L, v);
      else if (t.plane)
        done = deblock_unit<T, kDir, 6>(J.io, a, t.plane, c4, r4, L, v);
      else if (c == 1)
        done = deblock_unit<T, kDir, 8>(J.io, a, 0, c4, r4, L, v);
      else
        done = deblock_unit<T, kDir, 16>(J.io, a, 0, c4, r4, L, v);
    }
    if (!done)
      deblock_unit_lines<T>(J.io, a, kDir, t.plane, c4, r4, L, c == 0 ? 4 : t.plane ? 6 : c == 1 ? 8 : 16);
  }
}

template <int kDir>
__device__ __forceinline__ void db_item(const FrameJob& J, int local, DbShared& sh) {
  const DbTile t = db_locate(J, local);
  if (J.io.bd == 8)
    db_tile<uint8_t, kDir>(J, t, sh);
  else
    db_tile<uint16_t, kDir>(J, t, sh);
}

template <bool kLoop, int kDir>
__global__ void __launch_bounds__(256, 4) k_deblock_batch(BatchArgs b) {
  stage_begin();
  const int stage = kDir == 0 ? ST_DEBLOCK_V : ST_DEBLOCK_H;
  const int* base = b.base + stage * (b.n + 1);
  __shared__ DbShared sh;
  for_each_item<kLoop>(
      b, stage,
      [&](int item) {
        const int fi = find_frame(base, b.n, item);
        db_item<kDir>(b.jobs[fi], item - base[fi], sh);
      },
      [&](int item) {
        // The tile's samples and the 8 on each side its edges can reach.
        const int fi = find_frame(base, b.n, item);
        const FrameJob& J = b.jobs[fi];
        const DbTile t = db_locate(J, item - base[fi]);
        const int tw = 32, th = 8 << J.db_tile;
        const int x0 = t.tx * 128, y0 = t.ty * th * 4;
        if (J.io.bd == 8)
          prefetch_block<uint8_t>(J.io.pl[t.plane], x0 - 8, x0 + tw * 4 + 8, y0 - 8, y0 + th * 4 + 8);
        else
          prefetch_block<uint16_t>(J.io.pl[t.plane], x0 - 8, x0 + tw * 4 + 8, y0 - 8, y0 + th * 4 + 8);
      });
}

template <int kDir>
__global__ void __launch_bounds__(256, 4) k_deblock_one(const __grid_constant__ FrameJob J) {
  stage_begin();
  __shared__ DbShared sh;
  db_item<kDir>(J, blockIdx.x, sh);
}

template <int kDir>
static cudaError_t launch_dir(const StageLaunch& l) {
  if (l.one) return launch_stage(k_deblock_one<kDir>, l.total, 256, 0, l.st, l.dependent, *l.one);
  static int wave = 0;
  if (batch_loops(l.args)) return launch_stage(k_deblock_batch<true, kDir>, l.grid, 256, 0, l.st, l.dependent, l.args);
  return launch_stage(k_deblock_batch<false, kDir>, l.grid, 256, 0, l.st, l.dependent,
                      with_wave(l.args, k_deblock_batch<false, kDir>, 256, 0, wave));
}

cudaError_t launch_deblock(const StageLaunch& l, int dir) {
  if (l.total <= 0) return cudaSuccess;
  return dir == 0 ? launch_dir<0>(l) : launch_dir<1>(l);
}

}  // namespace pf
