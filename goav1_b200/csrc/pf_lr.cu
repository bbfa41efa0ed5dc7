// pf_lr.cu - loop restoration (Wiener / SGRproj) on the GPU.
//
// One CTA per (64-wide column, restoration stripe, plane).  The
// geometry is goav1's: tile/restoration_schedule.go:61-109, :400-409 (unit
// grid), tile/restoration_geometry.go:54-236 (unit rects shifted up by 8/4
// rows, stripes of 64/32 rows with the first one 8/4 rows shorter, 64-wide
// processing units).  Each stripe reads the post-CDEF plane with a 3-sample
// replicated frame border (restoration_boundary.go:126-180) and, across
// interior stripe boundaries, the pre-CDEF rows the CDEF kernel saved
// (setupRestorationStripeBoundaryFromSaved, restoration_boundary.go:553-614:
// rows above = saved[max(i+2,0)], rows below = saved[min(i,1)]).  The
// filters are restoration/wiener.go:59-211 and restoration/selfguided.go:
// 111-390 (box sums, a/b tables, 6/5 and 4/3 weights, projection with the
// int16 wrap).  Visible output columns depend only on +/-3 source columns,
// so the reference's rounding of the last Wiener unit width up to 16 changes
// no stored sample and is not replicated.
//
// Every sample of the tile inside the MI-aligned plane is written to the
// destination: restored samples where a Wiener/SGR unit covers the cropped
// plane, the post-CDEF sample everywhere else.
//
// Bound by instruction issue (76 % of the slots; both integer pipes about 60 %
// busy, DRAM 4 %), so the filters work on whole words: sample pairs for the
// sums and products (dp4a squares of 8-bit samples, dp2a for two Wiener
// taps), one word for an SGR box's a and b, two output columns a thread; and
// chroma tiles are as wide as luma's where their unit is, since a 32x32 tile
// cost a CTA's set-up for a quarter of the samples.  us per frame: 60 x 1080p
// 8-bit, a third of the units of each kind, 18.9 before, 10.4 now (7.6 and
// 4.4 warp instructions per luma sample); 8 x 4K 10-bit 78.9 and 44.9; one
// 1080p frame 28.7 and 19.5.  The encoder's search at 1080p: 144 and 68 us.
#include "pf_common.cuh"
#include "pf_tables.h"

namespace pf {

__constant__ int16_t c_sgr_params[16][4];
__constant__ uint8_t c_xbx[256];  // a - 1 by z: x / (x + 1) in 1/256, less one

// ---- the staged window and the two filters ----
//
// The window holds a tile (at most 64x64) with its 3-sample halo as 16-bit
// samples: sample (x, y) of the tile at row y + 3, column x + 4, so that a
// sample pair starting on an even x is one word, four samples of the frame
// are two, and every table below is built from whole words.
constexpr int kWinRows = 70;
constexpr int kWinWords = 36;  // 72 columns: x = -4 .. 67
constexpr int kTabPitch = 68;  // SGR tables: column x at x + 1, x = -1 .. 64

struct LrSmem {
  alignas(16) uint32_t win[kWinRows * kWinWords];
  union {
    // SGR a and b of one box in one word, (a - 1) << 22 | b (a - 1 <= 255; b,
    // a 32-bit product shifted by 12, below 2^20), so that the sum of three neighbours is one addition
    // chain: radius 1 for rows -1..h, radius 2 for the rows -1, 1, 3, ... it
    // is computed on.
    struct {
      uint32_t t1[66 * kTabPitch];
      uint32_t t2[33 * kTabPitch];
    } sgr;
    uint32_t wt[35 * 64];  // Wiener row-pass output as vertical pairs: rows 2k and 2k + 1 of a column
  };
  uint8_t xbx[256];  // a - 1 by z: data-dependent lookup, so shared memory and not constant
};

__device__ __forceinline__ int32_t rpot(int32_t v, int bits) {
  return bits <= 0 ? v : (v + (int32_t)(1 << (bits - 1))) >> bits;
}

// How a CTA shares a tile's output: thread tid has the column pair
// x = 2 * (tid % (PW / 2)) over a run of an even number of rows.
struct LrRun {
  int x, ya, yb;
};
__device__ __forceinline__ LrRun lr_run(int h, int PW) {
  const int lg = PW == 64 ? 5 : 4, segs = 256 >> lg;
  const int rows = ((h + segs - 1) / segs + 1) & ~1;
  const int ya = (threadIdx.x >> lg) * rows;
  return LrRun{2 * (int)(threadIdx.x & ((1 << lg) - 1)), ya, imin(h, ya + rows)};
}

// The symmetric 7-tap filter of a pair of neighbours from packed sample
// pairs: `in` holds the eight samples s0..s7 as four words when kEven (the
// first output is s0..s6's, the second s1..s7's), and s-1..s8 as five
// otherwise (s0 in the first word's upper half).  Two taps are one dp2a; the
// centre tap can exceed its 8-bit operand and is a multiplication of its own.
struct WienerTaps {
  int t01, t12, t2, t0, t0h, t2h, t21, t10, c;
};
__device__ __forceinline__ WienerTaps wiener_taps(int f0, int f1, int f2) {
  auto two = [](int lo, int hi) { return (lo & 0xff) | (hi & 0xff) << 8; };
  return WienerTaps{two(f0, f1), two(f1, f2), two(f2, 0), two(f0, 0), two(0, f0),
                    two(0, f2),  two(f2, f1), two(f1, f0), 128 - 2 * (f0 + f1 + f2)};
}
// Two unsigned 16-bit samples times two signed 8-bit taps, added to c.
__device__ __forceinline__ int dp2a_us(uint32_t a, int b, int c) {
  int d;
  asm("dp2a.lo.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// Samples s0..s6 with s0 in a word's lower half: words (s0 s1)(s2 s3)(s4 s5)(s6 -).
__device__ __forceinline__ int wiener_low(const WienerTaps& f, uint32_t a, uint32_t b, uint32_t c, uint32_t d, int init) {
  int s = dp2a_us(a, f.t01, init);
  s = dp2a_us(b, f.t2, s);
  s = dp2a_us(c, f.t21, s);
  s = dp2a_us(d, f.t0, s);
  return s + (int)(b >> 16) * f.c;
}
// Samples s0..s6 with s0 in a word's upper half: (- s0)(s1 s2)(s3 s4)(s5 s6).
__device__ __forceinline__ int wiener_high(const WienerTaps& f, uint32_t a, uint32_t b, uint32_t c, uint32_t d, int init) {
  int s = dp2a_us(a, f.t0h, init);
  s = dp2a_us(b, f.t12, s);
  s = dp2a_us(c, f.t2h, s);
  s = dp2a_us(d, f.t10, s);
  return s + (int)(c & 0xffffu) * f.c;
}

// Wiener filter of the staged window (restoration/wiener.go:132-211), w x h
// <= 64 x 64; h and v are the first three horizontal / vertical taps.
// out(y, x, v0, v1) receives the outputs of columns x and x + 1 (x even; the
// second is past the tile when x + 1 == w).  Every thread of the CTA calls
// it; it leaves the window untouched and ends without a barrier.
template <class Out>
__device__ __forceinline__ void lr_wiener_window(LrSmem& sm, int w, int h, int bd, const int8_t* hf, const int8_t* vf,
                                                 int PW, Out&& out) {
  const int maxv = (1 << bd) - 1;
  // restoration/wiener.go:202-211 (wienerRounds), :132-196.
  int round0 = 3, round1 = 11;
  const int range = bd + 7 - round0 + 2;
  if (range > 16) {
    round0 += range - 16;
    round1 -= range - 16;
  }
  const int top = (1 << (bd + 1 + 7 - round0)) - 1;
  // Row pass: a thread takes two rows of a column pair and leaves each
  // column's two results as one word.
  {
    const WienerTaps f = wiener_taps(hf[0], hf[1], hf[2]);
    const int init = (1 << (bd + 6)) + (1 << (round0 - 1));
    const int lg = PW == 64 ? 5 : 4;
    const int xw = threadIdx.x & ((1 << lg) - 1), step = 256 >> lg;
    if (2 * xw < w)
      for (int k = threadIdx.x >> lg; 2 * k < h + 6; k += step) {
        int o[2][2];
#pragma unroll
        for (int r = 0; r < 2; r++) {
          const uint32_t* p = &sm.win[(2 * k + r) * kWinWords + xw];
          const uint32_t a = p[0], b = p[1], c = p[2], d = p[3], e = p[4];
          o[r][0] = __vimin_s32_relu(wiener_high(f, a, b, c, d, init) >> round0, top);
          o[r][1] = __vimin_s32_relu(wiener_low(f, b, c, d, e, init) >> round0, top);
        }
        *reinterpret_cast<uint2*>(&sm.wt[k * 64 + 2 * xw]) =
            make_uint2(__byte_perm(o[0][0], o[1][0], 0x5410), __byte_perm(o[0][1], o[1][1], 0x5410));
      }
  }
  __syncthreads();
  // Column pass: two rows of the column pair at a time from four rows' worth
  // of words, one of them new.
  const LrRun t = lr_run(h, PW);
  if (t.x < w && t.ya < t.yb) {
    const WienerTaps f = wiener_taps(vf[0], vf[1], vf[2]);
    const int init = (1 << (round1 - 1)) - (1 << (bd + round1 - 1));
    const uint32_t* p = &sm.wt[(t.ya >> 1) * 64 + t.x];
    uint2 a = *reinterpret_cast<const uint2*>(p), b = *reinterpret_cast<const uint2*>(p + 64),
          c = *reinterpret_cast<const uint2*>(p + 128);
#pragma unroll 4
    for (int y = t.ya; y < t.yb; y += 2) {
      p += 64;
      const uint2 d = *reinterpret_cast<const uint2*>(p + 128);
      out(y, t.x, __vimin_s32_relu(wiener_low(f, a.x, b.x, c.x, d.x, init) >> round1, maxv),
          __vimin_s32_relu(wiener_low(f, a.y, b.y, c.y, d.y, init) >> round1, maxv));
      if (y + 1 < t.yb)
        out(y + 1, t.x, __vimin_s32_relu(wiener_high(f, a.x, b.x, c.x, d.x, init) >> round1, maxv),
            __vimin_s32_relu(wiener_high(f, a.y, b.y, c.y, d.y, init) >> round1, maxv));
      a = b;
      b = c;
      c = d;
    }
  }
}

// a and b of one SGR box (restoration/selfguided.go:132-231), packed as in
// LrSmem: the box's sum and sum of squares, area N (9 or 25), strength sv.
// 8-bit variances are never negative; deeper ones are rounded first and can be.
template <int N, bool k8>
__device__ __forceinline__ uint32_t sgr_ab(uint32_t sum, uint32_t sq, int bd, uint32_t sv, const uint8_t* xbx) {
  constexpr uint32_t kOneByN = (4096 + N / 2) / N;
  uint32_t p;
  if (k8) {
    p = sq * N - sum * sum;
  } else {
    const uint32_t av = (uint32_t)rpot((int32_t)sq, 2 * (bd - 8)), bv = (uint32_t)rpot((int32_t)sum, bd - 8);
    p = max(av * N, bv * bv) - bv * bv;  // words beyond 12 bits reach above 2^31
  }
  uint32_t z = (p * sv + (1u << 19)) >> 20;
  z = z < 255u ? z : 255u;
  const uint32_t a1 = xbx[z];  // a - 1
  const uint32_t b = ((255u - a1) * sum * kOneByN + 2048u) >> 12;
  return (a1 << 22) + b;
}

// Sums over three (h3, q3) and five (h5, q5) columns of one window row around
// a column pair, of the samples and of their squares: .x of the first column,
// .y of the second.  8-bit sample sums stay packed in .x (five rows of five
// fit a half); deeper ones do not fit.
struct BoxRow {
  uint2 h3, h5, q3, q5;
};

template <bool R2, bool k8>
__device__ __forceinline__ BoxRow box_row(const uint32_t* p) {
  const uint32_t A = p[0], B = p[1], C = p[2];  // samples x-2 .. x+3
  BoxRow o;
  if (k8) {
    o.h3.x = __byte_perm(A, B, 0x5432) + B + __byte_perm(B, C, 0x5432);
    o.h5.x = o.h3.x + A + C;
    // Bytes of a word squared and summed by one dp4a (the upper byte of an
    // 8-bit sample is a zero to fill with).
    const uint32_t a3 = __byte_perm(A, B, 0x1642), b3 = __byte_perm(B, C, 0x1420);
    o.q3 = make_uint2(__dp4a(a3, a3, 0u), __dp4a(b3, b3, 0u));
    if (R2) {
      const uint32_t a5 = __byte_perm(A, C, 0x1140), b5 = __byte_perm(A, C, 0x1162);
      o.q5 = make_uint2(__dp4a(a5, a5, o.q3.x), __dp4a(b5, b5, o.q3.y));
    }
  } else {
    const uint32_t x0 = A & 0xffff, x1 = A >> 16, x2 = B & 0xffff, x3 = B >> 16, x4 = C & 0xffff, x5 = C >> 16;
    const uint32_t m = x2 * x2 + x3 * x3;
    o.h3 = make_uint2(x1 + x2 + x3, x2 + x3 + x4);
    o.q3 = make_uint2(x1 * x1 + m, x4 * x4 + m);
    if (R2) {
      o.h5 = make_uint2(x0 + x4 + o.h3.x, x1 + x5 + o.h3.y);
      o.q5 = make_uint2(x0 * x0 + (x4 * x4 + o.q3.x), x1 * x1 + (x5 * x5 + o.q3.y));
    }
  }
  return o;
}

// Sums of three rows' pairs, unpacked.
template <bool k8>
__device__ __forceinline__ uint2 pair_sum(uint2 a, uint2 b, uint2 c) {
  const uint32_t x = a.x + b.x + c.x;
  return k8 ? make_uint2(x & 0xffff, x >> 16) : make_uint2(x, a.y + b.y + c.y);
}

// Self-guided filter of the staged window (restoration/selfguided.go:111-390)
// for a parameter set whose radius-2 (R2) and radius-1 (R1) filters are on or
// off, with the decoded projection weights xq0 / xq1; the same contract as
// lr_wiener_window, with a barrier at its end.  sm.xbx must hold the table.
//
// Tables: a thread has a column pair and slides down it two box rows at a
// time (radius 1 has a box on every row, radius 2 on the rows -1, 1, 3, ...),
// each window row's 3- and 5-column sums made once for both radii and both
// columns, the row sums added up from the last few rows' registers.
// Filters: a thread has a column pair over a run of rows; the three-column
// sums of a table row are two additions for both columns, and the rows' terms
// slide down in registers: 6 C + 5 (S - C) = 5 S + C for radius 2, and
// 4 S(y+1) + 3 (S(y) + S(y+2)) + C(y) + C(y+2) for radius 1.  The tables' a
// is one less than a; the missing weights (32, or 16 on radius 2's odd rows)
// and the rounding ride on constants that the additions have room for.
template <bool R2, bool R1, bool k8, class Out>
__device__ __forceinline__ void lr_sgr_window_t(LrSmem& sm, int w, int h, int bd, uint32_t s2, uint32_t s1, int xq0,
                                                int xq1, int PW, Out&& out) {
  const int tid = threadIdx.x;
  {
    const int npairs = (w + 2) / 2 + 1;  // column pairs x = -2, 0, ..
    const int segs = 256 / npairs, n2 = (h + 3) >> 1, per = (n2 + segs - 1) / segs;
    const int seg = tid / npairs, p = tid - seg * npairs;
    const int k0 = seg * per, k1 = imin(n2, k0 + per);
    if (seg < segs && k0 < k1) {
      const int c = 2 * p - 1;  // table column of the pair's first
      const bool c0in = c >= 0 && c <= w + 1, c1 = c + 1 <= w + 1;
      const uint32_t* win = &sm.win[2 * k0 * kWinWords + p];
      uint32_t* o1 = &sm.sgr.t1[2 * k0 * kTabPitch + c];
      uint32_t* o2 = &sm.sgr.t2[k0 * kTabPitch + c];
      const BoxRow r0 = box_row<R2, k8>(win), r1 = box_row<R2, k8>(win + kWinWords);
      BoxRow rc = box_row<R2, k8>(win + 2 * kWinWords), rb = r1;
      auto add2 = [](uint2 a, uint2 b) { return make_uint2(a.x + b.x, a.y + b.y); };
      uint2 t0{}, u0{};
      if (R2) {
        t0 = add2(r0.h5, r1.h5);
        u0 = add2(r0.q5, r1.q5);
      }
      win += 3 * kWinWords;
#pragma unroll 1
      for (int k = k0; k < k1; k++, win += 2 * kWinWords, o1 += 2 * kTabPitch, o2 += kTabPitch) {
        // Box rows 2k and 2k + 1: window rows 2k .. 2k + 4 are r0, rb, rc, rd, re.
        const BoxRow rd = box_row<R2, k8>(win), re = box_row<R2, k8>(win + kWinWords);
        if (R1) {
#pragma unroll
          for (int r = 0; r < 2; r++) {
            const BoxRow &a = r ? rc : rb, &b = r ? rd : rc, &d = r ? re : rd;
            if (r == 1 && 2 * k + 1 > h + 1) break;
            const uint2 s = pair_sum<k8>(a.h3, b.h3, d.h3);
            if (c0in) o1[r * kTabPitch] = sgr_ab<9, k8>(s.x, a.q3.x + b.q3.x + d.q3.x, bd, s1, sm.xbx);
            if (c1) o1[r * kTabPitch + 1] = sgr_ab<9, k8>(s.y, a.q3.y + b.q3.y + d.q3.y, bd, s1, sm.xbx);
          }
        }
        if (R2) {
          const uint2 t1 = add2(rc.h5, rd.h5), u1 = add2(rc.q5, rd.q5);
          const uint2 s = pair_sum<k8>(t0, t1, re.h5);
          if (c0in) o2[0] = sgr_ab<25, k8>(s.x, u0.x + u1.x + re.q5.x, bd, s2, sm.xbx);
          if (c1) o2[1] = sgr_ab<25, k8>(s.y, u0.y + u1.y + re.q5.y, bd, s2, sm.xbx);
          t0 = t1;
          u0 = u1;
        }
        rb = rd;
        rc = re;
      }
    }
  }
  __syncthreads();
  const LrRun t = lr_run(h, PW);
  if (t.x < w && t.ya < t.yb) {
    const int maxv = (1 << bd) - 1;
    // Projection (selfguided.go:233-247): (v + 1024) >> 11 as a 16-bit
    // integer is the upper half of 32 v + 32768.
    const int kd = 32 * (2048 - 16 * (xq0 + xq1)), k0 = 32 * xq0, k1 = 32 * xq1;
    constexpr uint32_t kB = (1u << 22) - 1;
    struct Term {
      int a[2], b[2];
    };
    // Three-column sums S and centres C of a table row for the pair.
    auto row = [&](const uint32_t* p, Term& s, Term& c) {
      const uint2 e = *reinterpret_cast<const uint2*>(p), f = *reinterpret_cast<const uint2*>(p + 2);
      const uint32_t m = e.y + f.x, s0 = e.x + m, s1 = m + f.y;
      s.a[0] = s0 >> 22, s.b[0] = s0 & kB, s.a[1] = s1 >> 22, s.b[1] = s1 & kB;
      c.a[0] = e.y >> 22, c.b[0] = e.y & kB, c.a[1] = f.x >> 22, c.b[1] = f.x & kB;
    };
    auto row2 = [&](int k, Term& z) {
      Term s, c;
      row(&sm.sgr.t2[k * kTabPitch + t.x], s, c);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        z.a[i] = 5 * s.a[i] + c.a[i];
        z.b[i] = 5 * s.b[i] + c.b[i];
      }
    };
    // Outer rows' term X = 3 S + C, the middle row's Y = 4 S with the constants.
    auto row1 = [&](int k, Term& X, Term& Y) {
      Term s, c;
      row(&sm.sgr.t1[k * kTabPitch + t.x], s, c);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        X.a[i] = 3 * s.a[i] + c.a[i];
        X.b[i] = 3 * s.b[i] + c.b[i];
        Y.a[i] = 4 * s.a[i] + 32;
        Y.b[i] = 4 * s.b[i] + 256;
      }
    };
    Term z0, x0, x1, y1, skip;
    if (R2) row2(t.ya >> 1, z0);
    if (R1) {
      row1(t.ya, x0, skip);
      row1(t.ya + 1, x1, y1);
    }
#pragma unroll 1
    for (int y = t.ya; y < t.yb; y += 2) {
      Term z1;
      if (R2) row2((y >> 1) + 1, z1);
#pragma unroll
      for (int r = 0; r < 2; r++) {
        if (r == 1 && y + 1 >= t.yb) break;
        const uint32_t d2 = sm.win[(y + r + 3) * kWinWords + (t.x >> 1) + 2];
        const int dg[2] = {(int)(d2 & 0xffff), (int)(d2 >> 16)};
        Term x2, y2;
        if (R1) row1(y + r + 2, x2, y2);
        int v[2];
#pragma unroll
        for (int i = 0; i < 2; i++) {
          int p = dg[i] * kd + 32768;
          if (R2) {
            const int f = r == 0 ? ((z0.a[i] + z1.a[i] + 32) * dg[i] + (z0.b[i] + z1.b[i] + 256)) >> 9
                                 : ((z1.a[i] + 16) * dg[i] + (z1.b[i] + 128)) >> 8;
            p += f * k0;
          }
          if (R1) {
            const int f = ((x0.a[i] + y1.a[i] + x2.a[i]) * dg[i] + (x0.b[i] + y1.b[i] + x2.b[i])) >> 9;
            p += f * k1;
          }
          v[i] = __vimin_s32_relu(p >> 16, maxv);
        }
        out(y + r, t.x, v[0], v[1]);
        if (R1) {
          x0 = x1;
          x1 = x2;
          y1 = y2;
        }
      }
      if (R2) z0 = z1;
    }
  }
  __syncthreads();
}

// The self-guided filter with parameter set `set` and the coded xqd pair
// (restoration/selfguided.go:111-127, DecodeSGRXQ), dispatched on which of
// its two radii are on (r0 is 0 or 2, r1 is 0 or 1).
template <bool k8, class Out>
__device__ __forceinline__ void lr_sgr_window(LrSmem& sm, int w, int h, int bd, int set, int xqd0, int xqd1, int PW,
                                              Out&& out) {
  const int r0 = c_sgr_params[set][0], r1 = c_sgr_params[set][1];
  const int s0 = c_sgr_params[set][2], s1 = c_sgr_params[set][3];
  if (r0 == 0)
    lr_sgr_window_t<false, true, k8>(sm, w, h, bd, s0, s1, 0, 128 - xqd1, PW, out);
  else if (r1 == 0)
    lr_sgr_window_t<true, false, k8>(sm, w, h, bd, s0, s1, xqd0, 0, PW, out);
  else
    lr_sgr_window_t<true, true, k8>(sm, w, h, bd, s0, s1, xqd0, 128 - xqd0 - xqd1, PW, out);
}

// Stages rows [0, wh) of a window: row(r) is the source row r's pointer to
// sample 0 of the plane (columns are clamped to 0 .. Wc - 1), x0 the tile's
// first column, w its width.  A task is four columns of a row; loads go out
// before the first is used.
template <typename T, class Row>
__device__ __forceinline__ void lr_stage(uint32_t* win, int x0, int w, int wh, int Wc, bool words, Row&& row) {
  const int groups = (w + 11) >> 2;  // columns -4 .. w + 3 and up
  const uint32_t inv = (65536u + (uint32_t)groups - 1) / (uint32_t)groups;  // i / groups for i < 1,260
  const int total = groups * wh;
  constexpr int kTasks = (18 * kWinRows + 255) / 256;
  uint2 v[kTasks];
#pragma unroll
  for (int k = 0; k < kTasks; k++) {
    const int i = threadIdx.x + 256 * k;
    if (i >= total) continue;
    const int r = (int)((i * inv) >> 16), g = i - r * groups;
    const int x = x0 - 4 + 4 * g;
    const T* src = row(r);
    if (words && x >= 0 && x + 4 <= Wc) {
      if constexpr (sizeof(T) == 1)
        v[k].x = *reinterpret_cast<const uint32_t*>(src + x);
      else
        v[k] = *reinterpret_cast<const uint2*>(src + x);
    } else {
      uint32_t s[4];
#pragma unroll
      for (int j = 0; j < 4; j++) s[j] = src[iclip(x + j, 0, Wc - 1)];
      if constexpr (sizeof(T) == 1)
        v[k].x = s[0] | s[1] << 8 | s[2] << 16 | s[3] << 24;
      else
        v[k] = make_uint2(s[0] | s[1] << 16, s[2] | s[3] << 16);
    }
  }
#pragma unroll
  for (int k = 0; k < kTasks; k++) {
    const int i = threadIdx.x + 256 * k;
    if (i >= total) continue;
    const int r = (int)((i * inv) >> 16), g = i - r * groups;
    uint2 o = v[k];
    if constexpr (sizeof(T) == 1)
      o = make_uint2(__byte_perm(v[k].x, 0, 0x4140), __byte_perm(v[k].x, 0, 0x4342));
    *reinterpret_cast<uint2*>(&win[r * kWinWords + 2 * g]) = o;
  }
}

// One restoration tile: column j of stripe s of `plane`, PW samples wide.
template <typename T>
__device__ __forceinline__ void lr_tile(const DFrame& src, const DFrame& dst, const LrArgs& a, const int* aw,
                                        const int* ah, int enabled, int plane, int j, int s, LrSmem& sm) {
  const int ssy = plane ? src.ssy : 0;
  const int PW = a.tile_w[plane], SH = 64 >> ssy, off = 8 >> ssy;
  const int Wa = aw[plane], Ha = ah[plane];
  const DPlane& sp = src.pl[plane];
  const DPlane& dp = dst.pl[plane];
  const int Wc = sp.w, Hc = sp.h;
  const int x0 = j * PW;
  const int y0 = imax(0, s * SH - off);
  if (x0 >= Wa || y0 >= Ha) return;
  const int x1 = imin(x0 + PW, Wa), y1 = imin((s + 1) * SH - off, Ha);
  const int tid = threadIdx.x;
  const int bd = sizeof(T) == 1 ? 8 : src.bd;  // a constant for 8-bit: the rounding shifts fold

  // Which restoration unit (if any) covers this tile.
  const pf_lr_unit* u = nullptr;
  const int xf1 = imin(x1, Wc), yf1 = imin(y1, Hc);
  if (enabled && a.type[plane] != PF_LR_NONE && x0 < Wc && y0 < Hc) {
    const int us = a.unit_size[plane];
    const int ur = imin((y0 + off) / us, a.vert[plane] - 1);
    const int uc = imin(x0 / us, a.horz[plane] - 1);
    const pf_lr_unit* cand = &a.units[plane][ur * a.horz[plane] + uc];
    if (cand->type == PF_LR_WIENER || cand->type == PF_LR_SGRPROJ) u = cand;
  }
  if (!u) {
    copy_block<T>(sp, dp, x0, x1, y0, y1);
    return;
  }
  const int h = yf1 - y0, w = xf1 - x0;
  // ---- stage the (h+6) x (w+6) source window ----
  const int nominal = SH - (y0 == 0 ? off : 0);
  const bool copyAbove = y0 != 0, copyBelow = y0 + nominal < Hc;
  const int kAbove = s, kBelow = s + 1;  // boundary indices of the saved lines
  const bool words = ((reinterpret_cast<uintptr_t>(sp.ptr) | (uintptr_t)sp.stride) & (4 * sizeof(T) - 1)) == 0;
  lr_stage<T>(sm.win, x0, w, h + 6, Wc, words, [&](int r) -> const T* {
    const int yy = y0 - 3 + r;
    if (yy < y0 && copyAbove)
      return reinterpret_cast<const T*>(a.lines[plane] + (int64_t)(kAbove * 4 + imax(yy - y0 + 2, 0)) * a.line_stride[plane]);
    if (yy >= yf1 && copyBelow)
      return reinterpret_cast<const T*>(a.lines[plane] + (int64_t)(kBelow * 4 + 2 + imin(yy - yf1, 1)) * a.line_stride[plane]);
    return row_ptr<T>(sp, iclip(yy, 0, Hc - 1));
  });
  sm.xbx[tid] = c_xbx[tid];
  __syncthreads();

  // Pixels of the tile outside the cropped plane are copied through.
  if (x1 > Wc || y1 > Hc)
    for (int i = tid; i < (x1 - x0) * (y1 - y0); i += 256) {
      const int y = y0 + i / (x1 - x0), x = x0 + i % (x1 - x0);
      if (x >= Wc || y >= Hc) row_ptr<T>(dp, y)[x] = row_ptr<T>(sp, y)[x];
    }

  // Two neighbours go out as one word where the row allows it.
  uint8_t* const ob = dp.ptr + (int64_t)y0 * dp.stride + (int64_t)x0 * (int)sizeof(T);
  const int64_t os = dp.stride;
  const bool pairs = ((reinterpret_cast<uintptr_t>(ob) | (uintptr_t)os) & (2 * sizeof(T) - 1)) == 0;
  auto store = [&](int y, int x, int v0, int v1) {
    T* o = reinterpret_cast<T*>(ob + y * os) + x;
    if (pairs && x + 1 < w) {
      if constexpr (sizeof(T) == 1)
        *reinterpret_cast<uint16_t*>(o) = (uint16_t)(v0 | v1 << 8);
      else
        *reinterpret_cast<uint32_t*>(o) = (uint32_t)v0 | (uint32_t)v1 << 16;
    } else {
      o[0] = (T)v0;
      if (x + 1 < w) o[1] = (T)v1;
    }
  };
  if (u->type == PF_LR_WIENER)
    lr_wiener_window(sm, w, h, bd, u->wiener_h, u->wiener_v, PW, store);
  else
    lr_sgr_window<sizeof(T) == 1>(sm, w, h, bd, u->sgr_set, u->sgr_xqd[0], u->sgr_xqd[1], PW, store);
}

static cudaError_t lr_configure();

cudaError_t lr_upload_tables() {
  uint8_t xbx[256];
  for (int z = 0; z < 256; z++) xbx[z] = (uint8_t)(pf_sgr_x_by_xplus1[z] - 1);
  cudaError_t e = cudaMemcpyToSymbol(c_sgr_params, pf_sgr_params, sizeof(pf_sgr_params));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(c_xbx, xbx, sizeof(xbx));
  return e == cudaSuccess ? lr_configure() : e;
}

// Batched restoration: each work item is one (processing column, stripe)
// tile of one plane of one frame.  Frames without restoration get the copy
// of the CDEF output back into the frame.
struct LrTile {
  int plane, j, s;
};

__device__ __forceinline__ LrTile lr_locate(const FrameJob& J, int local) {
  int plane = 0;
  while (plane < 2 && local >= J.lr_cols[plane] * J.lr_rows[plane]) {
    local -= J.lr_cols[plane] * J.lr_rows[plane];
    plane++;
  }
  return LrTile{plane, local % J.lr_cols[plane], local / J.lr_cols[plane]};
}

__device__ __forceinline__ void lr_item(const FrameJob& J, int local, LrSmem& sm) {
  const LrTile t = lr_locate(J, local);
  if (J.io.bd == 8)
    lr_tile<uint8_t>(J.scr, J.io, J.lr, J.aw, J.ah, J.do_lr, t.plane, t.j, t.s, sm);
  else
    lr_tile<uint16_t>(J.scr, J.io, J.lr, J.aw, J.ah, J.do_lr, t.plane, t.j, t.s, sm);
}

template <bool kLoop>
__global__ void __launch_bounds__(256, 4) k_lr_batch(BatchArgs b) {
  extern __shared__ __align__(16) uint8_t lr_smem_raw[];
  LrSmem& sm = *reinterpret_cast<LrSmem*>(lr_smem_raw);
  stage_begin();
  const int* base = b.base + ST_LR * (b.n + 1);
  for_each_item<kLoop>(
      b, ST_LR,
      [&](int item) {
        const int fi = find_frame(base, b.n, item);
        lr_item(b.jobs[fi], item - base[fi], sm);
      },
      [&](int item) {
        // The tile's stripe of the CDEF output with its 3-sample halo.
        const int fi = find_frame(base, b.n, item);
        const FrameJob& J = b.jobs[fi];
        const LrTile t = lr_locate(J, item - base[fi]);
        const int ssy = t.plane ? J.io.ssy : 0;
        const int PW = J.lr.tile_w[t.plane], SH = 64 >> ssy, off = 8 >> ssy;
        const int x0 = t.j * PW, y0 = t.s * SH - off;
        if (J.io.bd == 8)
          prefetch_block<uint8_t>(J.scr.pl[t.plane], x0 - 3, x0 + PW + 3, y0 - 3, y0 + SH + 3);
        else
          prefetch_block<uint16_t>(J.scr.pl[t.plane], x0 - 3, x0 + PW + 3, y0 - 3, y0 + SH + 3);
      });
}

__global__ void __launch_bounds__(256, 4) k_lr_one(const __grid_constant__ FrameJob J) {
  extern __shared__ __align__(16) uint8_t lr_smem_raw[];
  stage_begin();
  lr_item(J, blockIdx.x, *reinterpret_cast<LrSmem*>(lr_smem_raw));
}

// The shared layout's size, on the current device.
static cudaError_t lr_configure() {
  cudaError_t e = cudaSuccess;
  auto set = [&](auto* kernel) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LrSmem));
  };
  set(k_lr_batch<true>);
  set(k_lr_batch<false>);
  set(k_lr_one);
  return e;
}

cudaError_t launch_lr(const StageLaunch& l) {
  if (l.total <= 0) return cudaSuccess;
  if (l.one) return launch_stage(k_lr_one, l.total, 256, sizeof(LrSmem), l.st, l.dependent, *l.one);
  static int wave = 0;
  if (batch_loops(l.args)) return launch_stage(k_lr_batch<true>, l.grid, 256, sizeof(LrSmem), l.st, l.dependent, l.args);
  return launch_stage(k_lr_batch<false>, l.grid, 256, sizeof(LrSmem), l.st, l.dependent,
                      with_wave(l.args, k_lr_batch<false>, 256, sizeof(LrSmem), wave));
}

// ---- encoder loop-restoration unit search ----
// encoder/restoration.go:149-210 (SearchWienerUnitU8), :216-263
// (SearchSGRProjUnitU8) and the unit loops of EncodeLoopRestorationKeyframe
// (encoder/keyframe_lossy.go:2313-2383, :2422-2453), luma of 8-bit frames.
//
// Two launches.  k_lr_search_sse: one CTA per (unit, job); job 0 measures
// the unfiltered SSE, the six horizontal-only Wiener candidates and the
// exact Wiener filter of the pick, jobs 1..4 one exact SGR preset each, into
// a table of 32-bit SSEs (a unit holds at most 95 x 95 samples, so every sum
// stays below 2^32).  When the output is wanted, each exact filter also
// stores its filtered unit in a candidate buffer ([unit][job][64 x 64]
// bytes, 10 MB at 1080p, so it stays in L2).  k_lr_search_decide: one CTA
// per unit replays the reference's decisions over the table, writes the
// unit record and copies the winner's samples (or the unfiltered ones) into
// the output plane.  Bound by integer issue and the wait for the staged rows;
// 1920x1080, by the profiler: 68 us for the measuring kernel with the source
// read byte by byte at three CTAs per SM, 53 by words, 49 with four CTAs (five
// and six: the same call time); 11.8 us for the decisions with the copy byte
// by byte, 4.4 now.

// The candidate tap sets and presets of encoder/restoration.go:166-173 and
// :235-240, in the reference's order (first strictly better wins).
__constant__ int8_t c_lrs_wiener[PF_LR_WIENER_CANDIDATES][3] = {
    {0, -3, 12}, {0, -5, 18}, {0, -2, 8}, {0, 2, 10}, {1, 4, 14}, {0, -1, 4}};
__constant__ int8_t c_lrs_sgr[PF_LR_SGR_PRESETS][3] = {{0, 8, 24}, {2, 16, 40}, {10, 0, 48}, {14, 24, 72}};

constexpr uint32_t kLrsNone = 0xffffffffu;

struct LrsSse {
  uint32_t base;
  uint32_t wiener[PF_LR_WIENER_CANDIDATES];  // horizontal approximation
  uint32_t wexact;                           // exact Wiener of the pick
  uint32_t sgr[PF_LR_SGR_PRESETS];
  int32_t wpick;
};

struct LrsArgs {
  const uint8_t* src;
  int64_t sstride;
  const uint8_t* rec;
  int64_t rstride;
  uint8_t* dst;  // null: search only
  int64_t dstride;
  int W, H, horz, vert;
  LrsSse* table;
  pf_lr_search_unit* out;
  uint8_t* cand;  // [unit][1 + PF_LR_SGR_PRESETS][64 * 64]; null: search only
};

constexpr int kLrsJobs = 1 + PF_LR_SGR_PRESETS;

__device__ __forceinline__ uint8_t* lrs_cand(const LrsArgs& a, int unit, int job) {
  return a.cand + ((size_t)unit * kLrsJobs + job) * 4096;
}

struct LrsSmem {
  LrSmem lr;
  alignas(4) uint8_t src[64 * 64];
  uint32_t red[8 * 8];
};

// tile/restoration_geometry.go:54-92 for luma units of 64.
__device__ __forceinline__ void lrs_rect(const LrsArgs& a, int col, int row, int& x0, int& y0, int& x1, int& y1) {
  x0 = col * 64;
  x1 = col + 1 == a.horz ? a.W : x0 + 64;
  y0 = row * 64;
  y1 = row + 1 == a.vert ? a.H : y0 + 64;
  if (y0 > 0) y0 -= 8;
  if (y1 < a.H) y1 -= 8;
}

// Sums N per-thread values over the CTA; every thread gets the totals.
template <int N>
__device__ __forceinline__ void lrs_block_sum(uint32_t (&v)[N], uint32_t* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < N; i++) {
    uint32_t x = v[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    if (lane == 0) red[warp * N + i] = x;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; i++) {
    uint32_t x = 0;
    for (int k = 0; k < 8; k++) x += red[k * N + i];
    v[i] = x;
  }
  __syncthreads();
}

// The unit's recon window with a 3-sample edge-clamped border (the bordered
// copy of keyframe_lossy.go:2313-2330) into sm.lr.win; the SGR table when
// `tables`; the unit's source samples into sm.src when `source`.
__device__ __forceinline__ void lrs_stage(const LrsArgs& a, LrsSmem& sm, int x0, int y0, int w, int h, bool tables,
                                          bool source) {
  const bool words = ((reinterpret_cast<uintptr_t>(a.rec) | (uintptr_t)a.rstride) & 3) == 0;
  lr_stage<uint8_t>(sm.lr.win, x0, w, h + 6, a.W, words,
                    [&](int r) { return a.rec + (int64_t)iclip(y0 - 3 + r, 0, a.H - 1) * a.rstride; });
  if (source) {
    // Four samples a load where the rows allow it (x0 is a multiple of 64).
    const bool quads = ((reinterpret_cast<uintptr_t>(a.src) | (uintptr_t)a.sstride) & 3) == 0;
    for (int i = threadIdx.x; i < h * 16; i += 256) {
      const int r = i >> 4, c = (i & 15) * 4;
      const uint8_t* p = a.src + (int64_t)(y0 + r) * a.sstride + x0 + c;
      if (quads && c + 4 <= w)
        *reinterpret_cast<uint32_t*>(&sm.src[r * 64 + c]) = *reinterpret_cast<const uint32_t*>(p);
      else
        for (int k = 0; k < 4 && c + k < w; k++) sm.src[r * 64 + c + k] = p[k];
    }
  }
  if (tables) sm.lr.xbx[threadIdx.x] = c_xbx[threadIdx.x];
  __syncthreads();
}

// The same sets as compile-time values, for the unrolled candidate loop.
__host__ __device__ constexpr int lrs_tap(int c, int k) {
  constexpr int8_t t[PF_LR_WIENER_CANDIDATES][3] = {{0, -3, 12}, {0, -5, 18}, {0, -2, 8},
                                                    {0, 2, 10},  {1, 4, 14},  {0, -1, 4}};
  return t[c][k];
}

// One candidate's horizontal-only prediction (encoder/restoration.go:181-198)
// from the symmetric pair sums p06, p15, p24 and the centre p3.
template <int C>
__device__ __forceinline__ int lrs_hpred(int p06, int p15, int p24, int p3) {
  constexpr int t0 = lrs_tap(C, 0), t1 = lrs_tap(C, 1), t2 = lrs_tap(C, 2), t3 = -2 * (t0 + t1 + t2);
  const int hs = t0 * p06 + t1 * p15 + t2 * p24 + t3 * p3;
  return iclip((hs + 64) >> 7, 0, 255);
}

template <int C>
__device__ __forceinline__ void lrs_hsse(uint32_t* acc, int s, int p06, int p15, int p24, int p3) {
  const int d = s - lrs_hpred<C>(p06, p15, p24, p3);
  acc[1 + C] += (uint32_t)(d * d);
  if constexpr (C + 1 < PF_LR_WIENER_CANDIDATES) lrs_hsse<C + 1>(acc, s, p06, p15, p24, p3);
}

// SearchWienerUnitU8's choice over the table (encoder/restoration.go:161-209).
__device__ __forceinline__ int lrs_wiener_pick(const uint32_t* cand, uint32_t base, int area) {
  int pick = -1;
  uint64_t best = base;
  if (base != 0)
    for (int c = 0; c < PF_LR_WIENER_CANDIDATES; c++)
      if ((uint64_t)cand[c] + (uint64_t)area < best) {
        best = cand[c];
        pick = c;
      }
  return pick;
}

// One exact filter's outputs of columns x and x + 1: their squared error
// against the source, and into the candidate buffer (rows of 64).
__device__ __forceinline__ uint32_t lrs_outcome(const LrsSmem& sm, uint8_t* keep, int w, int y, int x, int v0, int v1) {
  const uint32_t s = *reinterpret_cast<const uint16_t*>(&sm.src[y * 64 + x]);  // x is even
  const int d0 = (int)(s & 0xff) - v0, d1 = (int)(s >> 8) - v1;
  uint32_t e = (uint32_t)(d0 * d0);
  if (x + 1 < w) e += (uint32_t)(d1 * d1);
  if (keep) *reinterpret_cast<uint16_t*>(&keep[y * 64 + x]) = (uint16_t)(v0 | v1 << 8);  // x + 1 <= 63
  return e;
}

__global__ void __launch_bounds__(256, 4) k_lr_search_sse(LrsArgs a) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  extern __shared__ __align__(16) uint8_t lrs_smem_raw[];
  LrsSmem& sm = *reinterpret_cast<LrsSmem*>(lrs_smem_raw);
  const int unit = blockIdx.x, job = blockIdx.y;
  int x0, y0, x1, y1;
  lrs_rect(a, unit % a.horz, unit / a.horz, x0, y0, x1, y1);
  const int w = x1 - x0, h = y1 - y0;
  const bool fits = w <= 64 && h <= 64;  // restoration/wiener.go:198-200
  LrsSse& T = a.table[unit];
  const int tid = threadIdx.x;
  if (job > 0) {
    // SearchSGRProjUnitU8, one preset (encoder/restoration.go:242-261).
    const int p = job - 1;
    if (!fits) {
      if (tid == 0) T.sgr[p] = kLrsNone;
      return;
    }
    lrs_stage(a, sm, x0, y0, w, h, true, true);
    uint32_t acc[1] = {0};
    uint8_t* keep = a.cand ? lrs_cand(a, unit, job) : nullptr;
    lr_sgr_window<true>(sm.lr, w, h, 8, c_lrs_sgr[p][0], c_lrs_sgr[p][1], c_lrs_sgr[p][2], 64,
                        [&](int y, int x, int v0, int v1) { acc[0] += lrs_outcome(sm, keep, w, y, x, v0, v1); });
    lrs_block_sum(acc, sm.red);
    if (tid == 0) T.sgr[p] = acc[0];
    return;
  }
  // Job 0: SearchWienerUnitU8 (encoder/restoration.go:149-210).
  uint32_t acc[1 + PF_LR_WIENER_CANDIDATES];
#pragma unroll
  for (int i = 0; i <= PF_LR_WIENER_CANDIDATES; i++) acc[i] = 0;
  if (fits) {
    lrs_stage(a, sm, x0, y0, w, h, false, true);
    const int tx = tid & 63;
    if (tx < w)
      for (int y = tid >> 6; y < h; y += 4) {
        const uint16_t* wr = reinterpret_cast<const uint16_t*>(sm.lr.win) + (y + 3) * 2 * kWinWords + tx + 1;
        const int s = sm.src[y * 64 + tx];
        const int d0 = s - (int)wr[3];
        acc[0] += (uint32_t)(d0 * d0);
        lrs_hsse<0>(acc, s, wr[0] + wr[6], wr[1] + wr[5], wr[2] + wr[4], wr[3]);
      }
  } else {
    // Units larger than 64x64 (the last row or column of some frame sizes):
    // the search still runs on them, straight from the frame.
    for (int i = tid; i < w * h; i += 256) {
      const int y = y0 + i / w, x = x0 + i % w;
      const uint8_t* rr = a.rec + (int64_t)y * a.rstride;
      const int s = a.src[(int64_t)y * a.sstride + x];
      const int d0 = s - (int)rr[x];
      acc[0] += (uint32_t)(d0 * d0);
      int px[7];
#pragma unroll
      for (int k = 0; k < 7; k++) px[k] = rr[iclip(x + k - 3, 0, a.W - 1)];
      lrs_hsse<0>(acc, s, px[0] + px[6], px[1] + px[5], px[2] + px[4], px[3]);
    }
  }
  lrs_block_sum(acc, sm.red);
  const int pick = lrs_wiener_pick(acc + 1, acc[0], w * h);
  uint32_t ex[1] = {kLrsNone};
  if (pick >= 0 && fits) {
    // The exact filter of the pick (keyframe_lossy.go:2344-2366).
    ex[0] = 0;
    uint8_t* keep = a.cand ? lrs_cand(a, unit, 0) : nullptr;
    lr_wiener_window(sm.lr, w, h, 8, c_lrs_wiener[pick], c_lrs_wiener[pick], 64,
                     [&](int y, int x, int v0, int v1) { ex[0] += lrs_outcome(sm, keep, w, y, x, v0, v1); });
    lrs_block_sum(ex, sm.red);
  }
  if (tid == 0) {
    T.base = acc[0];
    for (int c = 0; c < PF_LR_WIENER_CANDIDATES; c++) T.wiener[c] = acc[1 + c];
    T.wexact = ex[0];
    T.wpick = pick;
  }
}

// The unit's decision (keyframe_lossy.go:2338-2382) and, with a.dst, the
// unit filtered by it (:2422-2453).
__global__ void __launch_bounds__(256) k_lr_search_decide(LrsArgs a) {
  stage_begin();
  const int unit = blockIdx.x, tid = threadIdx.x;
  int x0, y0, x1, y1;
  lrs_rect(a, unit % a.horz, unit / a.horz, x0, y0, x1, y1);
  const int w = x1 - x0, h = y1 - y0;
  const bool fits = w <= 64 && h <= 64;
  const LrsSse& T = a.table[unit];
  const uint64_t base = T.base;
  const int wpick = T.wpick;
  uint64_t best = ~0ull;
  int type = PF_LR_NONE;
  if (wpick >= 0 && fits) {
    best = T.wexact;
    type = PF_LR_WIENER;
  }
  int spick = -1;
  uint64_t sbest = fits ? base : ~0ull;
  if (fits && base != 0)
    for (int p = 0; p < PF_LR_SGR_PRESETS; p++)
      if ((uint64_t)T.sgr[p] + (uint64_t)(w * h) < sbest) {
        sbest = T.sgr[p];
        spick = p;
      }
  if (spick >= 0 && sbest < best) {
    best = sbest;
    type = PF_LR_SGRPROJ;
  }
  if (tid == 0) {
    pf_lr_search_unit r;
    memset(&r, 0, sizeof(r));
    r.x0 = x0;
    r.y0 = y0;
    r.x1 = x1;
    r.y1 = y1;
    r.base_sse = base;
    r.sse = type == PF_LR_NONE ? base : best;
    r.wiener_sse = wpick >= 0 && fits ? (uint64_t)T.wexact : ~0ull;
    r.sgr_sse = sbest;
    r.wiener_candidate = (int8_t)wpick;
    r.sgr_preset = (int8_t)spick;
    r.unit.type = (uint8_t)type;
    if (type == PF_LR_WIENER)
      for (int k = 0; k < 3; k++) r.unit.wiener_v[k] = r.unit.wiener_h[k] = c_lrs_wiener[wpick][k];
    if (type == PF_LR_SGRPROJ) {
      r.unit.sgr_set = (uint8_t)c_lrs_sgr[spick][0];
      r.unit.sgr_xqd[0] = c_lrs_sgr[spick][1];
      r.unit.sgr_xqd[1] = c_lrs_sgr[spick][2];
    }
    a.out[unit] = r;
  }
  if (!a.dst) return;
  // keyframe_lossy.go:2422-2453: the decided filter's samples, kept by the
  // measuring CTA; NONE units keep the reconstruction.
  const uint8_t* from = type == PF_LR_WIENER ? lrs_cand(a, unit, 0)
                        : type == PF_LR_SGRPROJ ? lrs_cand(a, unit, 1 + spick) : nullptr;
  // Units of up to 64x64 whose rows allow it (x0 is a multiple of 64): a word
  // of four rows a thread, all loads before the first store.
  const uint8_t* src = from ? from : a.rec + (int64_t)y0 * a.rstride + x0;
  const int64_t sstride = from ? 64 : a.rstride;
  uint8_t* dst = a.dst + (int64_t)y0 * a.dstride + x0;
  if (fits && ((reinterpret_cast<uintptr_t>(src) | (uintptr_t)sstride | reinterpret_cast<uintptr_t>(dst) |
                (uintptr_t)a.dstride) & 3) == 0) {
    const int x = (tid & 15) * 4, r = tid >> 4;
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (r + 16 * k < h && x + 4 <= w) v[k] = *reinterpret_cast<const uint32_t*>(src + (r + 16 * k) * sstride + x);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const int y = r + 16 * k;
      if (y >= h) break;
      if (x + 4 <= w)
        *reinterpret_cast<uint32_t*>(dst + y * a.dstride + x) = v[k];
      else
        for (int i = x; i < w; i++) dst[y * a.dstride + i] = src[y * sstride + i];
    }
    return;
  }
  for (int y = tid >> 5; y < h; y += 8)
    for (int x = tid & 31; x < w; x += 32) dst[(int64_t)y * a.dstride + x] = src[(int64_t)y * sstride + x];
}

static int lrs_check(const pf_frame* f, const pf_frame* ref) {
  // goav1's keyframe encoder works on 8-bit 4:2:0 pictures (SourceFrame420).
  if (f->bit_depth != 8 || f->ss_x != 1 || f->ss_y != 1 || f->mono || f->width != ref->width ||
      f->height != ref->height)
    return PF_ERR_UNSUPPORTED;
  if (f->memory != ref->memory || f->memory > PF_MEM_DEVICE) return PF_ERR_INVALID_ARG;
  const pf_plane& pl = f->plane[0];
  if (!pl.data || pl.width != ref->width || pl.height != ref->height || pl.stride < pl.width)
    return PF_ERR_SHORT_BUFFER;
  return PF_OK;
}

}  // namespace pf

void* pf_internal_search_scratch(pf_ctx* c, size_t bytes);  // pf_api.cu
int pf_internal_wait(pf_ctx* c, void* stream);  // pf_api.cu: blocking or bounded by the context's deadline
void* pf_internal_stream(pf_ctx* c);
void* pf_internal_pinned(pf_ctx* c, size_t bytes);

extern "C" int pf_lr_search(pf_ctx* ctx, const pf_frame* source, const pf_frame* recon, const pf_frame* restored,
                            pf_lr_search_unit* units, int32_t max_units) {
  using namespace pf;
  if (!ctx || !source || !recon) return PF_ERR_INVALID_ARG;
  if (recon->width <= 0 || recon->height <= 0) return PF_ERR_INVALID_ARG;
  int stt = lrs_check(recon, recon);
  if (stt == PF_OK) stt = lrs_check(source, recon);
  if (stt == PF_OK && restored) stt = lrs_check(restored, recon);
  if (stt != PF_OK) return stt;
  const int W = recon->width, H = recon->height;
  const int horz = imax((W + 32) / 64, 1), vert = imax((H + 32) / 64, 1), n = horz * vert;
  if (units && max_units < n) return PF_ERR_SHORT_BUFFER;
  const cudaStream_t st = (cudaStream_t)pf_internal_stream(ctx);
  const bool host = recon->memory == PF_MEM_HOST;
  const pf_plane &sp = source->plane[0], &rp = recon->plane[0];
  // In place (restored's luma is recon's): the unit filters read a copy.
  const bool alias = restored && restored->plane[0].data == rp.data;
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t plane = al((size_t)W * H);
  size_t off = 0;
  const size_t oTab = off;
  off += al(sizeof(LrsSse) * n);
  const size_t oOut = off;
  off += al(sizeof(pf_lr_search_unit) * n);
  const size_t oSrc = off;
  off += host ? plane : 0;
  const size_t oRec = off;
  off += host || alias ? plane : 0;
  const size_t oDst = off;
  off += host && restored ? plane : 0;
  const size_t oCand = off;
  off += restored ? (size_t)n * kLrsJobs * 4096 : 0;
  uint8_t* base = (uint8_t*)pf_internal_search_scratch(ctx, off);
  if (!base) return PF_ERR_DEVICE;
  LrsArgs a;
  a.W = W;
  a.H = H;
  a.horz = horz;
  a.vert = vert;
  a.table = (LrsSse*)(base + oTab);
  a.out = (pf_lr_search_unit*)(base + oOut);
  a.cand = restored ? base + oCand : nullptr;
  cudaError_t e = cudaSuccess;
  const cudaMemcpyKind up = host ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
  if (host) {
    a.src = base + oSrc;
    a.sstride = W;
    e = cudaMemcpy2DAsync(base + oSrc, W, sp.data, sp.stride, W, H, up, st);
  } else {
    a.src = (const uint8_t*)sp.data;
    a.sstride = sp.stride;
  }
  if (host || alias) {
    a.rec = base + oRec;
    a.rstride = W;
    if (e == cudaSuccess) e = cudaMemcpy2DAsync(base + oRec, W, rp.data, rp.stride, W, H, up, st);
  } else {
    a.rec = (const uint8_t*)rp.data;
    a.rstride = rp.stride;
  }
  a.dst = nullptr;
  a.dstride = 0;
  if (restored) {
    a.dst = host ? base + oDst : (uint8_t*)restored->plane[0].data;
    a.dstride = host ? W : restored->plane[0].stride;
  }
  if (e != cudaSuccess) return PF_ERR_DEVICE;
  static bool configured = false;
  if (!configured) {
    if (cudaFuncSetAttribute(k_lr_search_sse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(LrsSmem)) !=
        cudaSuccess)
      return PF_ERR_DEVICE;
    configured = true;
  }
  k_lr_search_sse<<<dim3(n, 1 + PF_LR_SGR_PRESETS), 256, sizeof(LrsSmem), st>>>(a);
  if (launch_stage(k_lr_search_decide, n, 256, 0, st, true, a) != cudaSuccess) return PF_ERR_DEVICE;
  e = cudaGetLastError();
  if (e == cudaSuccess && host && restored)
    e = cudaMemcpy2DAsync(restored->plane[0].data, restored->plane[0].stride, a.dst, W, W, H,
                          cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess && units)
    e = cudaMemcpyAsync(units, a.out, sizeof(pf_lr_search_unit) * n, cudaMemcpyDeviceToHost, st);
  if (e != cudaSuccess) return PF_ERR_DEVICE;
  return pf_internal_wait(ctx, st);
}

