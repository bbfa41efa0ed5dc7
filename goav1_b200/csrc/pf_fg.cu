// pf_fg.cu - film-grain synthesis and reference-frame border extension.
//
// Film grain follows goav1's publication path: internal/av1/decoder/
// postfilter_filmgrain.go:192-263 (plane activity), :516-628 (LUTs, luma then
// chroma templates, chroma planes then luma, into a display copy) and the
// filmgrain package: random.go:15-72 (LFSR, stripe seeds), luma.go:24-158 and
// chroma.go:29-241 (templates with the AR recursion), scaling.go:18-121,
// apply.go:72-343, :414-546 and blend.go:16-25 (per-32x32 block offsets drawn
// in order from each stripe's LFSR, overlap blends, noise and clipping).
//
// GPU shape: the 82x73 templates are generated by one 3-warp CTA per frame.
// The Gaussian fill is split over the CTA's 96 threads: the LFSR is linear
// over GF(2)^16, so thread k starts from M^(kL) * seed (jump matrices
// precomputed on the host) and walks its L draws; the AR filter runs as a
// wavefront over t = x + 4y (every AR input of sample (y, x) has a smaller
// t), one warp per template, rows in lanes, neighbours passed between lanes
// by shuffles.  Offsets come from one thread per 32-row stripe.  The apply
// is a thread per 4x4 samples, 64x64-sample tiles per CTA.
#include "pf_common.cuh"
#include "pf_tables.h"

namespace pf {

constexpr int kGW = 82, kGH = 73;

__device__ __forceinline__ int rpow2(int v, int bits) { return bits <= 0 ? v : (v + (1 << (bits - 1))) >> bits; }

__device__ __forceinline__ uint16_t lfsr(uint16_t& reg, int bits) {
  const uint16_t bit = ((reg >> 0) ^ (reg >> 1) ^ (reg >> 3) ^ (reg >> 12)) & 1;
  reg = (uint16_t)((reg >> 1) | (bit << 15));
  return (uint16_t)((reg >> (16 - bits)) & ((1 << bits) - 1));
}

// ---- grain templates ----
//
// Shared layout of a template while it is generated: 32 lanes x 4 padded
// rows of 128 samples.  Template row y is AR row v = y - 3 (v = -3..h-4);
// it lives in padded row 4 * (v mod 32) + floor(v / 32) + 1, column x at
// x + 4.  Lane r of the AR warp owns AR rows r, r + 32, r + 64 (rows -3..-1
// ride on lanes 29..31), so the rows a lane visits are consecutive in
// memory and its position at wavefront step t is one running address,
// 508 r + t + 132.  Samples that the recursion must pass through unchanged
// (rows 0-2, the three border columns on each side, the padding) are
// stored with kNonAr added; an AR output is a plain sample.  The stored
// value then tells each step what to do, and no step needs a bounds test.
constexpr int kTplRow = 128;
constexpr int kTplPlane = 32 * 4 * kTplRow;
constexpr int kTplCol0 = 4;
constexpr int kNonAr = 16384;  // above any grain sample (|g| <= 2048)
constexpr int kFgTemplateThreads = 96;

struct TplSmem {
  int16_t g[3][kTplPlane];  // luma, Cb, Cr
  int16_t lt[kTplPlane];    // the chroma AR's luma term, chroma layout
  int16_t gauss[2048];      // the Gaussian sequence
};

__device__ __forceinline__ int tpl_at(int y, int x) {
  const int v = y - 3;
  return (4 * (v & 31) + (v >> 5) + 1) * kTplRow + x + kTplCol0;
}

__device__ __forceinline__ int tpl_decode(int s) { return s >= kNonAr / 2 ? s - kNonAr : s; }

// AR recursion of one template (luma.go:83-158 / chroma.go:92-199 generic
// form), run by one warp as a single wavefront with no barrier: AR row v
// is at column x = t - 4v at step t, so every AR input of (v, x) from the
// rows above was finished at an earlier step.  Rows v - d at column
// x + LAG reach the lane from lane r - 1 by warp shuffles out of small
// register rings: the row directly above as that lane's output of 4 - LAG
// steps back, and the rows further up as the values that lane itself
// received 4 steps back (for LAG 3 those two are passed on as one packed
// pair of int16; for LAG 2 and 3 a pair of taps costs one __dp2a_lo).
// The filter runs in transposed form: a value arriving from the rows above
// goes straight into the partial sums of the outputs x .. x + 2*LAG it
// reaches, and the lane's own output adds its in-row products to the next
// LAG outputs' sums, so the loop-carried path is shuffle -> multiply-add ->
// shift -> clip.  The partial sums rotate through acc[] with the step and
// start from the rounding offset; the rings are whole rotations long, so
// the unrolled steps rename registers.
// The wavefront starts 4*LAG steps early so that the pass-through rows
// above the first AR row are in the rings when row 0 needs them, and may
// run a few steps past the last AR output (those steps only rewrite
// pass-through samples with their own values).  LAG is a template argument
// (coefficients in registers, unrolled taps); with LAG 0 only the luma
// term remains, one sample a lane.
template <int LAG, bool kLt>
__device__ __forceinline__ void ar_warp(int16_t* g, const int16_t* lt, const FgTemplateArgs& p, int plane, int w, int h) {
  constexpr int kTaps = 2 * LAG * (LAG + 1);  // causal neighbours before the centre
  const int lane = threadIdx.x & 31;
  const int cs = p.coeff_shift, ro = 1 << (cs - 1);
  const int gmin = -(1 << (p.bd - 1)), gmax = (1 << (p.bd - 1)) - 1;
  const int8_t* cf = p.coeffs[plane];
  if constexpr (LAG == 0) {
    if constexpr (!kLt) return;
    const int coL = cf[0], aw = w - 6;
    for (int i = lane; i < aw * (h - 3); i += 32) {
      const int o = tpl_at(3 + i / aw, 3 + i % aw);
      g[o] = (int16_t)iclip(g[o] + ((lt[o] * coL + ro) >> cs), gmin, gmax);
    }
  } else {
    constexpr int W = 2 * LAG + 1;
    constexpr int U = 2 * W;  // ring length (at least 5) and unroll
    // Per output slot j (the output j columns right of the arriving value):
    // the two farthest rows' taps as a byte pair (LAG 2 and 3) and the
    // nearest row's tap (LAG 1 and 3).
    int cp[W], c1[W], cin[LAG + 1];
#pragma unroll
    for (int j = 0; j < W; j++) {
      cp[j] = 0;
      c1[j] = 0;
      if constexpr (LAG >= 2)
        cp[j] = (int)(uint8_t)cf[2 * LAG - j] | ((int)(uint8_t)cf[W + 2 * LAG - j] << 8);
      if constexpr (LAG == 3) c1[j] = cf[2 * W + 2 * LAG - j];
      if constexpr (LAG == 1) c1[j] = cf[2 * LAG - j];
    }
#pragma unroll
    for (int m = 1; m <= LAG; m++) cin[m] = cf[LAG * W + LAG - m];
    const int coL = kLt ? cf[kTaps] : 0;
    int acc[W], ring[U], ring2[U];
#pragma unroll
    for (int j = 0; j < W; j++) acc[j] = ro;
#pragma unroll
    for (int j = 0; j < U; j++) ring[j] = ring2[j] = 0;
    const int src = (lane + 31) & 31;
    const int pos0 = 508 * lane + 132;
    // The last step finishes column w - 4 of the last AR row.
    const int tend = 4 * (h - 4) + w - 3;
    for (int t0 = -4 * LAG; t0 < tend; t0 += U) {
      int16_t* gp = g + pos0 + t0;
      const int16_t* lp = kLt ? lt + pos0 + t0 : nullptr;
#pragma unroll
      for (int k = 0; k < U; k++) {
        if constexpr (LAG == 3) {
          // (row y-3, row y-2) as a pair, then row y-1.
          const int q = __shfl_sync(0xffffffffu, ring2[(k + U - 4) % U], src);
          const int v1 = __shfl_sync(0xffffffffu, ring[(k + U - 1) % U], src);
#pragma unroll
          for (int j = W - 1; j >= 0; j--) acc[(j + k) % W] = __dp2a_lo(q, cp[j], acc[(j + k) % W]);
#pragma unroll
          for (int j = W - 1; j >= 0; j--) acc[(j + k) % W] += c1[j] * v1;
          ring2[k] = (int)__byte_perm((unsigned)q, (unsigned)v1, 0x5432);
        } else if constexpr (LAG == 2) {
          const int v1 = __shfl_sync(0xffffffffu, ring[(k + U - 2) % U], src);
          const int v2 = __shfl_sync(0xffffffffu, ring2[(k + U - 4) % U], src);
          const int pr = (int)__byte_perm((unsigned)v2, (unsigned)v1, 0x5410);
          ring2[k] = v1;
#pragma unroll
          for (int j = W - 1; j >= 0; j--) acc[(j + k) % W] = __dp2a_lo(pr, cp[j], acc[(j + k) % W]);
        } else {
          const int v1 = __shfl_sync(0xffffffffu, ring[(k + U - 3) % U], src);
#pragma unroll
          for (int j = W - 1; j >= 0; j--) acc[(j + k) % W] += c1[j] * v1;
        }
        const int g0 = gp[k];
        int s = acc[k % W];
        if constexpr (kLt) s += lp[k] * coL;
        const int o = iclip(g0 + (s >> cs), gmin, gmax);
        const int out = g0 >= kNonAr / 2 ? g0 - kNonAr : o;
        gp[k] = (int16_t)out;
        ring[k] = out;
        // Output x's in-row products for columns x + 1 .. x + LAG; its slot
        // then serves column x + W.
        acc[k % W] = ro;
#pragma unroll
        for (int m = 1; m <= LAG; m++) acc[(m + k) % W] += cin[m] * out;
      }
    }
  }
}

template <bool kLt>
__device__ __forceinline__ void ar_warp_lag(int16_t* g, const int16_t* lt, const FgTemplateArgs& p, int plane, int w, int h) {
  switch (p.lag) {
    case 0: ar_warp<0, kLt>(g, lt, p, plane, w, h); break;
    case 1: ar_warp<1, kLt>(g, lt, p, plane, w, h); break;
    case 2: ar_warp<2, kLt>(g, lt, p, plane, w, h); break;
    default: ar_warp<3, kLt>(g, lt, p, plane, w, h); break;
  }
}

// Luma term of the chroma AR (chroma.go:92-199): at each chroma AR position
// the luma grain averaged over the co-located 1, 2 or 4 samples, into lt
// (chroma layout).  The luma samples read are all AR positions, which hold
// plain values.  All threads of the CTA.
__device__ __forceinline__ void luma_term(int16_t* lt, const int16_t* luma, int sx, int sy, int w, int h) {
  const int aw = w - 6;
  for (int i = threadIdx.x; i < aw * (h - 3); i += blockDim.x) {
    const int y = 3 + i / aw, x = 3 + i % aw;
    const int lx = ((x - 3) << sx) + 3, ly = ((y - 3) << sy) + 3;
    const int a = tpl_at(ly, lx);
    int s = luma[a];
    if (sx) s += luma[a + 1];
    if (sy) {
      const int b = tpl_at(ly + 1, lx);
      s += luma[b];
      if (sx) s += luma[b + 1];
    }
    lt[tpl_at(y, x)] = (int16_t)rpow2(s, sx + sy);
  }
}

// Jump matrices: g_jump[t][k][c] = M^(k*L_t) e_c for the three template
// shapes (t = 0: 82x73, 1: 44x73, 2: 44x38), L_t = ceil(samples / 96), so
// that thread k of the CTA starts its share of the draws at draw k * L_t.
// Global memory rather than constant: every thread reads its own row.
__device__ int16_t g_gauss[2048];
__device__ uint16_t g_jump[3][kFgTemplateThreads][16];
__device__ int g_jump_len[3];

__device__ __forceinline__ uint16_t gf2_apply(const uint16_t* cols, uint16_t v) {
  uint16_t r = 0;
#pragma unroll
  for (int c = 0; c < 16; c++)
    if ((v >> c) & 1) r ^= cols[c];
  return r;
}

// Gaussian fill of one template (luma.go:32-38 / chroma.go:38-44): draw i of
// the plane's LFSR goes to sample (i / w, i % w).  All threads of the CTA,
// each walking L consecutive draws from its jumped LFSR state.
__device__ __forceinline__ void gauss_fill(int16_t* g, const int16_t* gauss, uint16_t seed, int w, int h, int shape, int shift) {
  const int L = g_jump_len[shape];
  uint16_t reg = gf2_apply(g_jump[shape][threadIdx.x], seed);
  int i = threadIdx.x * L;
  const int iend = imin(i + L, w * h);
  if (i >= iend) return;
  int y = i / w, x = i - y * w;
  int row = tpl_at(y, 0);
  for (; i < iend; i++) {
    const int v = rpow2(gauss[lfsr(reg, 11)], shift);
    const bool ar = y >= 3 && x >= 3 && x < w - 3;
    g[row + x] = (int16_t)(ar ? v : v + kNonAr);
    if (++x == w) {
      x = 0;
      row = tpl_at(++y, 0);
    }
  }
}

// One frame's templates: Gaussian fills of the three planes by the whole
// CTA, the luma AR on warp 0, the luma term, then the Cb and Cr AR side by
// side on warps 1 and 2, and the templates written out (stride 82) with
// the pass-through marks taken off.
__device__ __forceinline__ void fg_templates(const FgTemplateArgs& p, int16_t* gy, int16_t* gu, int16_t* gv, TplSmem& S) {
  const int warp = threadIdx.x >> 5;
  int16_t* outs[3] = {gy, gu, gv};
  const int cw = p.ssx ? 44 : kGW, ch = p.ssy ? 38 : kGH;
  const int cshape = p.ssx ? (p.ssy ? 2 : 1) : 0;
  {
    const int4 fill = make_int4(0x40004000, 0x40004000, 0x40004000, 0x40004000);
    static_assert(kNonAr == 0x4000, "fill pattern");
    int4* g4 = reinterpret_cast<int4*>(S.g[0]);
    for (int i = threadIdx.x; i < 3 * kTplPlane / 8; i += blockDim.x) g4[i] = fill;
    const int4* src = reinterpret_cast<const int4*>(g_gauss);
    int4* dst = reinterpret_cast<int4*>(S.gauss);
    for (int i = threadIdx.x; i < 2048 / 8; i += blockDim.x) dst[i] = src[i];
  }
  __syncthreads();
  const int shift = 12 - p.bd + p.grain_scale_shift;
  if (p.num_y_points != 0) gauss_fill(S.g[0], S.gauss, p.seed, kGW, kGH, 0, shift);
  if (p.active[1]) gauss_fill(S.g[1], S.gauss, (uint16_t)(p.seed ^ 0xb524), cw, ch, cshape, shift);
  if (p.active[2]) gauss_fill(S.g[2], S.gauss, (uint16_t)(p.seed ^ 0x49d8), cw, ch, cshape, shift);
  __syncthreads();
  if (warp == 0 && p.num_y_points != 0 && p.lag != 0) ar_warp_lag<false>(S.g[0], nullptr, p, 0, kGW, kGH);
  __syncthreads();
  const bool lumaTerm = p.num_y_points != 0;
  if (lumaTerm) {
    luma_term(S.lt, S.g[0], p.ssx, p.ssy, cw, ch);
    __syncthreads();
  }
  const bool runC = warp >= 1 && warp <= 2 && p.active[warp] && !(p.lag == 0 && p.num_y_points == 0);
  if (runC) {
    if (lumaTerm)
      ar_warp_lag<true>(S.g[warp], S.lt, p, warp, cw, ch);
    else
      ar_warp_lag<false>(S.g[warp], nullptr, p, warp, cw, ch);
  }
  __syncthreads();
  // Two samples per 32-bit store (rows of 82 samples keep pairs aligned),
  // one sample each where the plane starts on an odd one (kGrainShift).
  for (int pl = 0; pl < 3; pl++) {
    if (!outs[pl]) continue;
    if (pl && p.ssx) {
      uint32_t* o = reinterpret_cast<uint32_t*>(outs[pl]);
      for (int i = threadIdx.x; i < kGH * kGW / 2; i += blockDim.x) {
        const int y = i / (kGW / 2), x = 2 * (i - y * (kGW / 2));
        const uint32_t s = *reinterpret_cast<const uint32_t*>(&S.g[pl][tpl_at(y, x)]);
        const int lo = tpl_decode((int16_t)(s & 0xffff)), hi = tpl_decode((int16_t)(s >> 16));
        o[i] = (uint32_t)(uint16_t)lo | ((uint32_t)(uint16_t)hi << 16);
      }
    } else {
      for (int i = threadIdx.x; i < kGH * kGW; i += blockDim.x) {
        const int y = i / kGW;
        outs[pl][i] = (int16_t)tpl_decode(S.g[pl][tpl_at(y, i - y * kGW)]);
      }
    }
  }
}

// The scaling function of 10- and 12-bit samples (scaling.go:88-121) at every
// sample value: entries [0, 1 << bd) of each plane's 4,096.
__device__ __forceinline__ int scale_at(const uint8_t* lut, int index, int bd) {
  const int shift = bd - 8, x = index >> shift;
  if (x == 255) return lut[x];
  const int rem = index - (x << shift), start = lut[x], end = lut[x + 1];
  return (uint8_t)(start + rpow2((end - start) * rem, shift));
}

// Offsets of every 32x32 block: row r uses the LFSR seeded by stripe r
// (random.go:39-49), one Number(8) per block in order (apply.go:72-125).
__device__ __forceinline__ void fg_offsets_row(uint16_t seed, int r, int cols, uint8_t* out) {
  const int n = r;  // lumaLine >> 5 with lumaLine = 32 r
  uint16_t reg = seed;
  reg ^= (uint16_t)(((n * 37 + 178) & 255) << 8);
  reg ^= (uint16_t)((n * 173 + 105) & 255);
  for (int b = 0; b < cols; b++) out[r * cols + b] = (uint8_t)lfsr(reg, 8);
}

// ---- grain application ----
//
// Display = reference with grain added on the cropped area of active planes;
// every allocated sample of the display frame is written.
//
// A thread takes four adjacent columns by four rows of one plane (always
// inside one grain block): the four samples of a row move as one word, the
// block's set-up (offsets, template positions, blend weights) is shared by
// sixteen samples, and nothing else is done per sample but the scaling
// lookup, the multiply-add and one fused add-and-clamp.  10- and 12-bit
// planes look the scaling up in a table of every sample value, built once a
// frame beside the block offsets, instead of interpolating per sample.  The
// quads on a block's left edge, which blend with the block to the left, are
// gathered in warps of their own, so the others' warps never wait for that
// path.
//
// Bound by integer issue (57 % of the slots) and the wait for the grain
// behind the block offset.  us per frame: 60 x 1080p 8-bit 12.6 before (one
// column by 16 rows a thread, every sample by itself), 6.8 now, at 2.2 warp
// instructions per luma sample instead of 5.0; 8 x 4K 10-bit 62.9 and 28.8;
// one 1080p frame 25.6 and 16.  The neighbouring blocks' offsets are read
// ahead of the stores, their grains row by row through the read-only path
// (the left block's offset read row by row, too: 6.84 and 29.4; all offsets,
// and the grains by plain loads: 7.1 and 30.1).  With the last, two rows' or
// one row's loads at a time measured 7.3 and 7.8, 3 or 5 CTAs per SM 8.1 and
// 7.2.

template <typename T>
struct FgQuad;
template <>
struct FgQuad<uint8_t> {
  typedef uint32_t W;
  static __device__ __forceinline__ W load(const uint8_t* p, bool word, int n) {
    if (word) return *reinterpret_cast<const uint32_t*>(p);
    uint32_t v = 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k < n) v |= (uint32_t)p[k] << (8 * k);
    return v;
  }
  static __device__ __forceinline__ void store(uint8_t* p, W v, bool word, int n) {
    if (word) {
      *reinterpret_cast<uint32_t*>(p) = v;
      return;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k < n) p[k] = (uint8_t)(v >> (8 * k));
  }
  static __device__ __forceinline__ int get(W v, int k) { return (v >> (8 * k)) & 0xff; }
  static __device__ __forceinline__ W pack(int a, int b, int c, int d) {
    return __byte_perm(__byte_perm(a, b, 0x0040), __byte_perm(c, d, 0x0040), 0x5410);
  }
};
template <>
struct FgQuad<uint16_t> {
  typedef uint2 W;
  static __device__ __forceinline__ W load(const uint16_t* p, bool word, int n) {
    if (word) return *reinterpret_cast<const uint2*>(p);
    uint2 v = make_uint2(0, 0);
    if (n > 0) v.x = p[0];
    if (n > 1) v.x |= (uint32_t)p[1] << 16;
    if (n > 2) v.y = p[2];
    if (n > 3) v.y |= (uint32_t)p[3] << 16;
    return v;
  }
  static __device__ __forceinline__ void store(uint16_t* p, W v, bool word, int n) {
    if (word) {
      *reinterpret_cast<uint2*>(p) = v;
      return;
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (k < n) p[k] = (uint16_t)get(v, k);
  }
  static __device__ __forceinline__ int get(W v, int k) {
    const uint32_t h = k < 2 ? v.x : v.y;
    return k & 1 ? h >> 16 : h & 0xffff;
  }
  static __device__ __forceinline__ W pack(int a, int b, int c, int d) {
    return make_uint2(__byte_perm(a, b, 0x5410), __byte_perm(c, d, 0x5410));
  }
};

__device__ __forceinline__ int blend_w(int prev, int cur, int pw, int cw, int bd) {
  return iclip(rpow2(prev * pw + cur * cw, 5), -(1 << (bd - 1)), (1 << (bd - 1)) - 1);
}

// Four grains of a template row from column c: the plane's templates start
// so that unsubsampled planes' columns (always odd) fall on word boundaries
// (kGrainShift); subsampled ones are taken from three words by the parity.
template <bool kSx>
__device__ __forceinline__ uint2 grain4(const int16_t* row, int c) {
  if (!kSx) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(row + c);
    return make_uint2(__ldg(w), __ldg(w + 1));
  }
  const uint32_t* w = reinterpret_cast<const uint32_t*>(row + (c & ~1));
  const uint32_t a = __ldg(w), b = __ldg(w + 1), d = __ldg(w + 2);
  const int sh = (c & 1) * 16;
  return make_uint2(__funnelshift_r(a, b, sh), __funnelshift_r(b, d, sh));
}

__device__ __forceinline__ int grain_of(uint2 g, int k) {
  const uint32_t h = k < 2 ? g.x : g.y;
  return k & 1 ? (int)h >> 16 : (int)(int16_t)(h & 0xffff);
}

// Columns x .. x + 3, rows y0 .. y0 + 3 of one display plane (x and y0
// multiples of 4).  kLuma / kSx: the plane is luma / horizontally subsampled
// chroma.  kRows rows' loads (four, or one where words do not fit) are issued
// before their first store.  word: four
// samples of a row move as one word.
template <typename T, bool kLuma, bool kSx, int kRows>
__device__ __forceinline__ void fg_apply_quad(const DFrame& ref, const DFrame& disp, const FgArgs& a,
                                              const uint8_t* lut, int plane, int x, int y0, const bool word) {
  typedef FgQuad<T> Q;
  // Plane descriptors by value: they live in the job table in global memory,
  // which the compiler would re-read after every store.
  const DPlane sp = ref.pl[plane];
  const DPlane dp = disp.pl[plane];
  const DPlane lp = ref.pl[0];
  const int n = word ? 4 : imin(4, sp.aw - x), yend = imin(y0 + 4, sp.ah);
  const bool on = a.active[plane] && x < sp.w;
  const int sx = kSx ? 1 : 0, sy = kLuma ? 0 : ref.ssy;
  const int yclip = on ? imin(yend, sp.h) : 0;
  const uint8_t* srow = sp.ptr + (int64_t)y0 * sp.stride + (int64_t)x * (int)sizeof(T);
  uint8_t* drow = dp.ptr + (int64_t)y0 * dp.stride + (int64_t)x * (int)sizeof(T);
  if (!on) {
    typename Q::W v[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (y0 + k < yend) v[k] = Q::load(reinterpret_cast<const T*>(srow + k * sp.stride), word, n);
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (y0 + k < yend) Q::store(reinterpret_cast<T*>(drow + k * dp.stride), v[k], word, n);
    return;
  }
  const int bd = sizeof(T) == 1 ? 8 : ref.bd;  // a constant for 8-bit: the depth shifts fold
  const int bwl = 5 - sx, bhl = 5 - sy;
  const int bw = 1 << bwl, bh = 1 << bhl;
  const int row = y0 >> bhl, bcol = x >> bwl;
  const int xi = x - (bcol << bwl), yi0 = y0 - (row << bhl);
  constexpr int ovl = 2;
  const int xStart = (a.overlap && bcol > 0 && xi == 0) ? imin(sp.w - x, ovl >> sx) : 0;
  const int yStart = (a.overlap && row > 0 && yi0 == 0) ? imin(sp.h - y0, ovl >> sy) : 0;
  const uint8_t* offs = a.offsets + row * a.off_cols + bcol;
  const int16_t* gr = a.grain[plane];
  // Template column / row origins of the current, left, top and top-left blocks.
  auto gcol = [&](int offset, int bc) { return 3 + (ovl >> sx) * (3 + (offset >> 4)) + xi + bw * bc; };
  auto grow = [&](int offset, int br) { return 3 + (ovl >> sy) * (3 + (offset & 15)) + yi0 + bh * br; };
  // The offsets at once: after a store they would be read again.
  const int o00 = __ldg(offs), o10 = xStart ? __ldg(offs - 1) : 0, o01 = yStart ? __ldg(offs - a.off_cols) : 0;
  const int o11 = xStart && yStart ? __ldg(offs - a.off_cols - 1) : 0;
  const int c00 = gcol(o00, 0);
  const int16_t* g00 = gr + grow(o00, 0) * kGW;
  const int shift = a.scaling_shift, rnd = 1 << (shift - 1);
  int minV = 0, maxV = (256 << (bd - 8)) - 1;
  if (a.clip_restricted) {
    minV = 16 << (bd - 8);
    maxV = (kLuma ? 235 : (a.matrix_identity ? 235 : 240)) << (bd - 8);
  }
  const bool cfl = a.cfl, edge = x + 4 > sp.w;
  const int oddCol = a.odd_luma ? sp.w - 1 - x : -1;  // the column whose luma has no right neighbour (4 and up: another quad's)
  const int lumaMult = a.luma_mult[plane] - 128, mult = a.mult[plane] - 128;
  const int offs0 = (a.offset[plane] << (bd - 8)) - (1 << bd);
  const int top = (1 << bd) - 1;
#pragma unroll
  for (int k0 = 0; k0 < 4; k0 += kRows) {
    typename Q::W s[kRows], l[kRows][2];
    uint2 g[kRows];
#pragma unroll
    for (int r = 0; r < kRows; r++) {
      const int k = k0 + r, y = y0 + k;
      if (y < yend) s[r] = Q::load(reinterpret_cast<const T*>(srow + k * sp.stride), word, n);
      if (y < yclip) {
        g[r] = grain4<kSx>(g00 + k * kGW, c00);
        if (!kLuma) {
          // The co-located luma row; a subsampled quad's eight samples are
          // inside the 8-aligned luma allocation.
          const T* lrow = reinterpret_cast<const T*>(lp.ptr + (int64_t)(y << sy) * lp.stride) + (x << sx);
          l[r][0] = Q::load(lrow, word, kSx ? 4 : n);
          if (kSx) l[r][1] = Q::load(lrow + 4, word, 4);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kRows; r++) {
      const int k = k0 + r, y = y0 + k;
      if (y >= yend) continue;
      typename Q::W out = s[r];
      if (y < yclip) {
        int gv[4];
#pragma unroll
        for (int j = 0; j < 4; j++) gv[j] = grain_of(g[r], j);
        if (xStart | yStart) {
          // Overlap (apply.go:301-343): horizontal weights 27/17 then 17/27
          // (subsampled 23/22), vertical ones the same by row.
          if (xStart) {
            const int c10 = gcol(o10, 1), r10 = grow(o10, 0) + k;
#pragma unroll
            for (int j = 0; j < ovl; j++)
              if (j < xStart) {
                const int hpw = sx ? 23 : (j == 1 ? 17 : 27), hcw = sx ? 22 : (j == 1 ? 27 : 17);
                gv[j] = blend_w(__ldg(&gr[r10 * kGW + c10 + j]), gv[j], hpw, hcw, bd);
              }
          }
          if (k < ovl && k < yStart) {
            const int vpw = sy ? 23 : (k == 1 ? 17 : 27), vcw = sy ? 22 : (k == 1 ? 27 : 17);
            const uint2 t = grain4<kSx>(gr + (grow(o01, 1) + k) * kGW, gcol(o01, 0));
            int tv[4];
#pragma unroll
            for (int j = 0; j < 4; j++) tv[j] = grain_of(t, j);
            if (xStart) {
              const int c11 = gcol(o11, 1), r11 = grow(o11, 1) + k;
#pragma unroll
              for (int j = 0; j < ovl; j++)
                if (j < xStart) {
                  const int hpw = sx ? 23 : (j == 1 ? 17 : 27), hcw = sx ? 22 : (j == 1 ? 27 : 17);
                  tv[j] = blend_w(__ldg(&gr[r11 * kGW + c11 + j]), tv[j], hpw, hcw, bd);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; j++) gv[j] = blend_w(tv[j], gv[j], vpw, vcw, bd);
          }
        }
        int o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const int v = Q::get(s[r], j);
          int idx = v;
          if (!kLuma) {
            // chromaScalingIndex (apply.go:501-520) on the un-grained luma.
            int avg;
            if (kSx) {
              const typename Q::W& lw = l[r][j >> 1];
              const int b0 = Q::get(lw, 2 * (j & 1)), b1 = Q::get(lw, 2 * (j & 1) + 1);
              avg = (b0 + b1 + 1) >> 1;
              if (j == oddCol) avg = b0;
            } else {
              avg = Q::get(l[r][0], j);
            }
            idx = cfl ? avg : __viaddmin_s32_relu((avg * lumaMult + v * mult) >> 6, offs0, top);
          }
          if (sizeof(T) == 2) idx = imin(idx, top);
          const int noise = (int)(lut[idx] * gv[j] + rnd) >> shift;
          o[j] = __viaddmin_s32_relu(v, noise, maxV);
        }
        if (minV) {
#pragma unroll
          for (int j = 0; j < 4; j++) o[j] = imax(o[j], minV);
        }
        if (edge) {
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (x + j >= sp.w) o[j] = Q::get(s[r], j);
        }
        out = Q::pack(o[0], o[1], o[2], o[3]);
      }
      Q::store(reinterpret_cast<T*>(drow + k * dp.stride), out, word, n);
    }
  }
}

// frame/buffer.go:339-400: replicate the last visible column into the padding
// columns of every visible row, then the last visible row into padding rows.
template <typename T>
__device__ __forceinline__ void extend_px(const DFrame& f, int plane, int x, int y) {
  const DPlane& p = f.pl[plane];
  if (x >= p.aw || y >= p.ah) return;
  if (x < p.w && y < p.h) return;
  const int h = imin(p.h, p.ah);
  row_ptr<T>(p, y)[x] = row_ptr<T>(p, imin(y, h - 1))[imin(x, p.w - 1)];
}

// ---- batched kernels ----

__device__ __forceinline__ void fg_templates_item(const FrameJob& J, TplSmem& S) {
  fg_templates(J.fgt, J.fg.grain[0], J.fg.grain[1], J.fg.grain[2], S);
}

__global__ void __launch_bounds__(kFgTemplateThreads) k_fg_templates_batch(BatchArgs b) {
  extern __shared__ __align__(16) unsigned char s_tpl[];
  TplSmem& S = *reinterpret_cast<TplSmem*>(s_tpl);
  const int* base = b.base + ST_FG_TEMPLATES * (b.n + 1);
  for_each_item(b, ST_FG_TEMPLATES, [&](int item) { fg_templates_item(b.jobs[find_frame(base, b.n, item)], S); });
}

__global__ void __launch_bounds__(kFgTemplateThreads) k_fg_templates_one(const __grid_constant__ FrameJob J) {
  extern __shared__ __align__(16) unsigned char s_tpl[];
  fg_templates_item(J, *reinterpret_cast<TplSmem*>(s_tpl));
}

__device__ __forceinline__ void fg_offsets_item(const FrameJob& J, int local) {
  if (J.io.bd > 8) {
    // The first items of a frame of more than 8 bits build its scaling
    // tables, 256 entries each.
    const int per = 1 << (J.io.bd - 8);
    if (local < 3 * per) {
      const int pl = local / per, i0 = (local - pl * per) * 256;
      for (int i = threadIdx.x; i < 256; i += 64)
        J.fg.scale[pl * kFgScaleLen + i0 + i] = (uint8_t)scale_at(J.fg.lut[pl], i0 + i, J.io.bd);
      return;
    }
    local -= 3 * per;
  }
  const int r = local * 64 + threadIdx.x;
  if (r < J.fg.off_rows) fg_offsets_row(J.fgt.seed, r, J.fg.off_cols, const_cast<uint8_t*>(J.fg.offsets));
}

__global__ void __launch_bounds__(64) k_fg_offsets_batch(BatchArgs b) {
  const int* base = b.base + ST_FG_OFFSETS * (b.n + 1);
  for_each_item(b, ST_FG_OFFSETS, [&](int item) {
    const int fi = find_frame(base, b.n, item);
    fg_offsets_item(b.jobs[fi], item - base[fi]);
  });
}

__global__ void __launch_bounds__(64) k_fg_offsets_one(const __grid_constant__ FrameJob J) {
  fg_offsets_item(J, blockIdx.x);
}

// Display frame: 64x64-sample tiles of each plane, 256 threads of four
// columns by four rows.  The plane's scaling table is staged in shared memory
// per tile.
struct FgTile {
  int plane, tx, ty;
};

__device__ __forceinline__ FgTile fg_locate(const FrameJob& J, int local) {
  int plane = 0;
  while (plane < 2 && local >= J.fg_tx[plane] * J.fg_ty[plane]) {
    local -= J.fg_tx[plane] * J.fg_ty[plane];
    plane++;
  }
  return FgTile{plane, local % J.fg_tx[plane], local / J.fg_tx[plane]};
}

// A quad of a plane whose rows are not on word boundaries, or one that
// reaches past the allocated width.
template <typename T, bool kLuma, bool kSx>
__device__ __noinline__ void fg_apply_any(const FrameJob* J, const uint8_t* lut, int plane, int x, int y0) {
  fg_apply_quad<T, kLuma, kSx, 1>(J->io, J->disp, J->fg, lut, plane, x, y0, false);
}

template <typename T, bool kLuma, bool kSx>
__device__ __forceinline__ void fg_apply_plane(const FrameJob& J, const uint8_t* lut, int plane, int x, int y0) {
  const DPlane &sp = J.io.pl[plane], &dp = J.disp.pl[plane], &lp = J.io.pl[0];
  if (x >= sp.aw || y0 >= sp.ah) return;
  if (x + 4 <= sp.aw &&
      ((reinterpret_cast<uintptr_t>(sp.ptr) | (uintptr_t)sp.stride | reinterpret_cast<uintptr_t>(dp.ptr) |
        (uintptr_t)dp.stride | reinterpret_cast<uintptr_t>(lp.ptr) | (uintptr_t)lp.stride) &
       (4 * sizeof(T) - 1)) == 0)
    fg_apply_quad<T, kLuma, kSx, 4>(J.io, J.disp, J.fg, lut, plane, x, y0, true);
  else
    fg_apply_any<T, kLuma, kSx>(&J, lut, plane, x, y0);
}

template <typename T>
__device__ __forceinline__ void fg_tile(const FrameJob& J, const FgTile& t, uint8_t* lut) {
  const int tid = threadIdx.x;
  if (sizeof(T) == 1) {
    lut[tid] = J.fg.lut[t.plane][tid];
  } else if (J.fg.active[t.plane]) {
    const uint4* src = reinterpret_cast<const uint4*>(J.fg.scale + t.plane * kFgScaleLen);
    if (tid < 1 << (J.io.bd - 4)) reinterpret_cast<uint4*>(lut)[tid] = src[tid];
  }
  __syncthreads();
  // Quads of the tile: first those inside their blocks, four rows at a
  // time, then (the last one or two warps) those on a block's left edge.
  const bool sx = t.plane && J.io.ssx;
  const int per = sx ? 12 : 14;  // inside quads a row: 3 of 4 or 7 of 8
  int q, rg;
  if (tid < per * 16) {
    rg = sx ? tid / 12 : tid / 14;
    const int i = tid - rg * per;
    q = sx ? i + i / 3 + 1 : i + i / 7 + 1;
  } else {
    const int i = tid - per * 16;
    rg = sx ? i >> 2 : i >> 1;
    q = sx ? (i & 3) * 4 : (i & 1) * 8;
  }
  const int x = t.tx * 64 + 4 * q, y0 = t.ty * 64 + 4 * rg;
  if (t.plane == 0)
    fg_apply_plane<T, true, false>(J, lut, 0, x, y0);
  else if (sx)
    fg_apply_plane<T, false, true>(J, lut, t.plane, x, y0);
  else
    fg_apply_plane<T, false, false>(J, lut, t.plane, x, y0);
}

template <bool kLoop>
__global__ void __launch_bounds__(256, 4) k_fg_apply_batch(BatchArgs b) {
  __shared__ __align__(16) uint8_t s_lut[kFgScaleLen];
  stage_begin();
  const int* base = b.base + ST_FG_APPLY * (b.n + 1);
  for_each_item<kLoop>(
      b, ST_FG_APPLY,
      [&](int item) {
        const int fi = find_frame(base, b.n, item);
        const FrameJob& J = b.jobs[fi];
        const FgTile t = fg_locate(J, item - base[fi]);
        if (J.io.bd == 8)
          fg_tile<uint8_t>(J, t, s_lut);
        else
          fg_tile<uint16_t>(J, t, s_lut);
        if (kLoop) __syncthreads();  // the table is rewritten by the next tile
      },
      [&](int item) {
        // The tile of the filtered frame (the grain's input).
        const int fi = find_frame(base, b.n, item);
        const FrameJob& J = b.jobs[fi];
        const FgTile t = fg_locate(J, item - base[fi]);
        const int x0 = t.tx * 64, y0 = t.ty * 64;
        if (J.io.bd == 8)
          prefetch_block<uint8_t>(J.io.pl[t.plane], x0, x0 + 64, y0, y0 + 64);
        else
          prefetch_block<uint16_t>(J.io.pl[t.plane], x0, x0 + 64, y0, y0 + 64);
      });
}

__global__ void __launch_bounds__(256, 4) k_fg_apply_one(const __grid_constant__ FrameJob J) {
  __shared__ __align__(16) uint8_t s_lut[kFgScaleLen];
  stage_begin();
  const FgTile t = fg_locate(J, blockIdx.x);
  if (J.io.bd == 8)
    fg_tile<uint8_t>(J, t, s_lut);
  else
    fg_tile<uint16_t>(J, t, s_lut);
}

// Border extension: 64x4-sample tiles of the right strip [w, aw) x [0, h)
// then of the bottom strip [0, aw) x [h, ah), per plane.
__device__ __forceinline__ void extend_item(const FrameJob& J, int local) {
  for (int plane = 0; plane < 3; plane++) {
    const int nr = J.ext_r[plane][0] * J.ext_r[plane][1], nb = J.ext_b[plane][0] * J.ext_b[plane][1];
    if (local >= nr + nb) {
      local -= nr + nb;
      continue;
    }
    const DPlane& p = J.io.pl[plane];
    int x, y;
    if (local < nr) {
      x = p.w + (local % J.ext_r[plane][0]) * 64 + (threadIdx.x & 63);
      y = (local / J.ext_r[plane][0]) * 4 + (threadIdx.x >> 6);
      if (y >= p.h) return;
    } else {
      local -= nr;
      x = (local % J.ext_b[plane][0]) * 64 + (threadIdx.x & 63);
      y = p.h + (local / J.ext_b[plane][0]) * 4 + (threadIdx.x >> 6);
    }
    if (J.io.bd == 8)
      extend_px<uint8_t>(J.io, plane, x, y);
    else
      extend_px<uint16_t>(J.io, plane, x, y);
    return;
  }
}

__global__ void __launch_bounds__(256) k_extend_batch(BatchArgs b) {
  stage_begin();
  const int* base = b.base + ST_EXTEND * (b.n + 1);
  for_each_item(b, ST_EXTEND, [&](int item) {
    const int fi = find_frame(base, b.n, item);
    extend_item(b.jobs[fi], item - base[fi]);
  });
}

__global__ void __launch_bounds__(256) k_extend_one(const __grid_constant__ FrameJob J) {
  stage_begin();
  extend_item(J, blockIdx.x);
}

// LFSR step as a GF(2)^16 map, for the host-side jump tables.
static uint16_t lfsr_step_host(uint16_t reg) {
  const uint16_t bit = ((reg >> 0) ^ (reg >> 1) ^ (reg >> 3) ^ (reg >> 12)) & 1;
  return (uint16_t)((reg >> 1) | (bit << 15));
}

static cudaError_t fg_configure();

cudaError_t fg_upload_tables() {
  static_assert(sizeof(pf_gaussian_sequence) == sizeof(g_gauss), "Gaussian sequence length");
  cudaError_t e = cudaMemcpyToSymbol(g_gauss, pf_gaussian_sequence, sizeof(pf_gaussian_sequence));
  if (e != cudaSuccess) return e;
  uint16_t jump[3][kFgTemplateThreads][16];
  int lens[3];
  const int samples[3] = {82 * 73, 44 * 73, 44 * 38};
  for (int t = 0; t < 3; t++) {
    const int L = (samples[t] + kFgTemplateThreads - 1) / kFgTemplateThreads;
    lens[t] = L;
    uint16_t cols[16];
    for (int c = 0; c < 16; c++) cols[c] = (uint16_t)(1u << c);
    for (int k = 0; k < kFgTemplateThreads; k++) {
      for (int c = 0; c < 16; c++) jump[t][k][c] = cols[c];
      for (int c = 0; c < 16; c++)
        for (int s = 0; s < L; s++) cols[c] = lfsr_step_host(cols[c]);
    }
  }
  e = cudaMemcpyToSymbol(g_jump, jump, sizeof(jump));
  if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_jump_len, lens, sizeof(lens));
  if (e == cudaSuccess) e = fg_configure();
  return e;
}

static cudaError_t fg_configure() {
  // The templates' shared layout is above the default 48 KB.
  cudaError_t e = cudaFuncSetAttribute(k_fg_templates_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TplSmem));
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_fg_templates_one, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TplSmem));
  return e;
}

cudaError_t launch_fg_templates(const StageLaunch& l) {
  if (l.total <= 0) return cudaSuccess;
  if (l.one)
    return launch_stage(k_fg_templates_one, l.total, kFgTemplateThreads, sizeof(TplSmem), l.st, false, *l.one);
  return launch_stage(k_fg_templates_batch, l.grid, kFgTemplateThreads, sizeof(TplSmem), l.st, false, l.args);
}

cudaError_t launch_fg_offsets(const StageLaunch& l) {
  if (l.total <= 0) return cudaSuccess;
  if (l.one) return launch_stage(k_fg_offsets_one, l.total, 64, 0, l.st, false, *l.one);
  return launch_stage(k_fg_offsets_batch, l.grid, 64, 0, l.st, false, l.args);
}

cudaError_t launch_fg_apply(const StageLaunch& l) {
  if (l.total <= 0) return cudaSuccess;
  if (l.one) return launch_stage(k_fg_apply_one, l.total, 256, 0, l.st, l.dependent, *l.one);
  static int wave = 0;
  if (batch_loops(l.args)) return launch_stage(k_fg_apply_batch<true>, l.grid, 256, 0, l.st, l.dependent, l.args);
  return launch_stage(k_fg_apply_batch<false>, l.grid, 256, 0, l.st, l.dependent,
                      with_wave(l.args, k_fg_apply_batch<false>, 256, 0, wave));
}

cudaError_t launch_extend(const StageLaunch& l) {
  if (l.total <= 0) return cudaSuccess;
  if (l.one) return launch_stage(k_extend_one, l.total, 256, 0, l.st, l.dependent, *l.one);
  return launch_stage(k_extend_batch, l.grid, 256, 0, l.st, l.dependent, l.args);
}

}  // namespace pf
