// pf_cdef.cu - CDEF on the GPU, one CTA per 64x64 filter unit (all planes).
//
// Semantics follow goav1's snapshot walk: internal/av1/decoder/
// postfilter_cdef.go:525-710 (applyCDEFPostFilterRows), :936-1035
// (unitStrength, applySnapshot), :1041-1047 (luma direction gate),
// :1101-1249 (VeryLarge halo fill and the row/column replicate quirk of
// frameWorkCopyCDEFInput), :1390-1412 (MI-aligned plane extent), :1544-1561
// (block list from the noskip word); and the kernels cdef/direction.go:37-79,
// :432-501, cdef/filter.go:79-169, :231-241, :396-543, :603-633.
//
// The kernel reads the deblocked frame (never written here) and writes every
// sample of the unit's MI-aligned extent to the output frame, filtered or
// copied, so the output is a pure function of the pre-CDEF frame exactly as
// in the reference's immutable-snapshot walk.  It also saves, straight from
// the pre-CDEF input, the four rows around each loop-restoration stripe
// boundary that falls inside the unit (tile/restoration_boundary.go:192-255):
// the boundary-line save is fused into the CDEF pass instead of a separate
// frame sweep.
//
// Bound by instruction issue (72 % of the slots at 32 warps per SM; the
// half-rate fp16 and integer pipes are both half busy, DRAM 3 %).  Hence the
// packed pairs of pf_cdef_dev.cuh (7 instructions a tap for two samples,
// where one sample's constrain() from a shared-memory table took 5 with two
// shared reads) and the three 4:2:0 planes staged and filtered in one pass.
// Per frame, 60 x 1080p 8-bit: 22.4 us before, 12.0 now (5.6 of it the taps,
// 1.5 the directions, 1.0 the staging); 8 x 4K 10-bit: 103.2 and 49.4; one
// 1080p frame alone: 44.8 and 22.3.  64 registers and 4 CTAs per SM: 48 (5
// CTAs, with spills) and 80 (3 CTAs) measured 4 % slower.
#include "pf_cdef_dev.cuh"

namespace pf {

// How a unit's samples are staged and filtered: fp16 pairs (8 bits, 10-bit
// words of at most 10 bits), packed 16-bit integers (words of at most 12
// bits), one by one in 32-bit integers.
enum CdefForm { kPairs, kInts, kWide };

// What a luma block's filter needs, made once per block: the primary tap's
// constants (PairTap) and flags: bit 31 filtered, bit 4 odd strength (weights 3, 3
// instead of 4, 2), low bits the direction.
struct CdefBlk {
  PairTap pri;
  uint32_t flags;
};

// Pitch of a 4:2:0 chroma unit's 32 + 8 words; other chroma units are staged
// where luma was, with its pitch.
constexpr int kPC = 40;

struct CdefSmem {
  alignas(16) uint32_t y[kPH * kPW];
  alignas(16) uint32_t c[2][36 * kPC];
  alignas(16) int32_t cost[64 * 8];
  alignas(16) CdefBlk blk[64];
  int2 ofs[2][12];  // direction tap offsets in words (cdef/filter.go:53-66), pitch kPW and kPC
  uint8_t dir[64];
};

// Four samples of a row as they lie in memory.
template <typename T>
struct Quad;
template <>
struct Quad<uint8_t> {
  typedef uint32_t W;
  static __device__ __forceinline__ W zero() { return 0; }
  static __device__ __forceinline__ W load(const uint8_t* p, bool words) {
    if (words) return *reinterpret_cast<const uint32_t*>(p);
    return p[0] | (uint32_t)p[1] << 8 | (uint32_t)p[2] << 16 | (uint32_t)p[3] << 24;
  }
  // Column k's samples of two rows as a pair of plain integers.
  template <int k>
  static __device__ __forceinline__ uint32_t pair(W a, W b) {
    return __byte_perm(a, b, 0x0400 + 0x0101 * k) & 0x00ff00ffu;
  }
  static __device__ __forceinline__ uint32_t bits(W) { return 0; }
};
template <>
struct Quad<uint16_t> {
  typedef uint2 W;
  static __device__ __forceinline__ W zero() { return make_uint2(0, 0); }
  static __device__ __forceinline__ W load(const uint16_t* p, bool words) {
    if (words) return *reinterpret_cast<const uint2*>(p);
    return make_uint2(p[0] | (uint32_t)p[1] << 16, p[2] | (uint32_t)p[3] << 16);
  }
  template <int k>
  static __device__ __forceinline__ uint32_t pair(W a, W b) {
    return __byte_perm(k < 2 ? a.x : a.y, k < 2 ? b.x : b.y, k & 1 ? 0x7632 : 0x5410);
  }
  static __device__ __forceinline__ uint32_t bits(W a) { return a.x | a.y; }
};

// One plane of a unit: where its samples are and what of them there is.
struct CdefPlane {
  const uint8_t* src;
  int64_t stride;
  int x, y, w, h;  // the unit in the plane
  int Wa, Ha;      // the plane's MI-aligned extent
  bool words;      // rows on 4-sample boundaries
  bool inside;     // the whole halo is frame data
};

__device__ __forceinline__ CdefPlane cdef_plane(const DPlane& p, int bytes, int x, int y, int wmax, int hmax, int Wa,
                                                int Ha) {
  CdefPlane q;
  q.src = p.ptr;
  q.stride = p.stride;
  q.x = x;
  q.y = y;
  q.w = imin(wmax, Wa - x);
  q.h = imin(hmax, Ha - y);
  q.Wa = Wa;
  q.Ha = Ha;
  q.words = ((reinterpret_cast<uintptr_t>(p.ptr) | (uintptr_t)p.stride) & (4 * bytes - 1)) == 0;
  q.inside = x >= 4 && x + q.w + 4 <= Wa && y >= 2 && y + q.h + 3 <= Ha;
  return q;
}

// Staging of a unit with its 2-row / 4-column halo as pair words
// (frameWorkFillCDEFInputSentinels / frameWorkCopyCDEFInput; planes end on
// 4-sample boundaries and the taps reach two samples, so the reference's row
// and column replication past a plane's end is never read).  A task is four
// columns (group cg, from the unit's column -4) of two word rows (2d,
// 2d + 1): three 4-sample loads, eight words.  Loads and stores are apart so
// that a thread's tasks are all in flight together.
// kIn: the unit's whole halo is frame data in rows on 4-sample boundaries.
template <typename T, bool kIn>
__device__ __forceinline__ void stage_load(const CdefPlane& p, const uint8_t* src, int d, int cg,
                                           typename Quad<T>::W (&v)[3]) {
  const int x = p.x - 4 + 4 * cg, y = p.y - 2 + 2 * d;
  const uint8_t* s = src + (int64_t)y * p.stride + (int64_t)x * (int)sizeof(T);
  const bool cin = x >= 0 && x < p.Wa;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    if (!kIn) v[j] = Quad<T>::zero();
    if (kIn || (cin && y + j >= 0 && y + j < p.Ha))
      v[j] = Quad<T>::load(reinterpret_cast<const T*>(s + j * p.stride), kIn || p.words);
  }
}

// Pairs as biased fp16 values, the other forms as plain integers.
template <typename T, bool kIn, CdefForm kForm, int kPitch>
__device__ __forceinline__ void stage_store(const CdefPlane& p, int d, int cg, const typename Quad<T>::W (&v)[3],
                                            uint32_t* buf) {
  constexpr uint32_t kBias = kForm == kPairs ? kPairBias : 0u, kNone = kForm == kPairs ? kPairNone : kPairRawNone;
  uint32_t* o = buf + 2 * d * kPitch + 4 * cg;
#pragma unroll
  for (int j = 0; j < 2; j++) {
    uint4 w = make_uint4(Quad<T>::template pair<0>(v[j], v[j + 1]) | kBias,
                         Quad<T>::template pair<1>(v[j], v[j + 1]) | kBias,
                         Quad<T>::template pair<2>(v[j], v[j + 1]) | kBias,
                         Quad<T>::template pair<3>(v[j], v[j + 1]) | kBias);
    if (!kIn) {
      const int x = p.x - 4 + 4 * cg, y = p.y - 2 + 2 * d + j;
      const bool cin = x >= 0 && x < p.Wa;
      const uint32_t keep =
          (cin && y >= 0 && y < p.Ha ? 0xffffu : 0u) | (cin && y + 1 >= 0 && y + 1 < p.Ha ? 0xffff0000u : 0u);
      const uint32_t fill = kNone & ~keep;
      w = make_uint4((w.x & keep) | fill, (w.y & keep) | fill, (w.z & keep) | fill, (w.w & keep) | fill);
    }
    *reinterpret_cast<uint4*>(o + j * kPitch) = w;
  }
}

// Bits that no sample of the form has.
template <typename T, CdefForm kForm>
__device__ __forceinline__ uint32_t stage_over(const typename Quad<T>::W (&v)[3]) {
  constexpr uint32_t kOver = kForm == kPairs ? 0xfc00fc00u : kForm == kInts ? 0xf000f000u : 0u;
  return (Quad<T>::bits(v[0]) | Quad<T>::bits(v[1]) | Quad<T>::bits(v[2])) & kOver;
}

// One plane's tasks one by one, any unit.
template <typename T, CdefForm kForm, int kPitch>
__device__ __forceinline__ uint32_t stage_any(const CdefPlane& p, const uint8_t* src, uint32_t* buf) {
  const int cgs = (p.w + 8) >> 2;
  const uint32_t inv = (65536u + (uint32_t)cgs - 1) / (uint32_t)cgs;  // i / cgs for i < 612
  const int total = cgs * ((p.h + 4) >> 1);
  uint32_t over = 0;
#pragma unroll 1
  for (int i = threadIdx.x; i < total; i += 256) {
    typename Quad<T>::W t[3];
    const int d = (int)((i * inv) >> 16), cg = i - d * cgs;
    stage_load<T, false>(p, src, d, cg, t);
    over |= stage_over<T, kForm>(t);
    stage_store<T, false, kForm, kPitch>(p, d, cg, t, buf);
  }
  return over;
}

// The three planes of a 4:2:0 unit.  Luma's 18 x 34 tasks fill two rounds of
// the CTA and warps 0-3 of the third; 2 x (10 x 18) chroma tasks follow on
// warps 4-7 and in a fourth.  All of a thread's loads are in flight together.
// kIn: a whole 64x64 unit with its halo inside the frame.
template <typename T, bool kIn, CdefForm kForm>
__device__ __forceinline__ uint32_t stage_420(const CdefPlane& P, const CdefPlane& Q, const uint8_t* vsrc, bool y,
                                              bool c, CdefSmem& sm) {
  const int tid = threadIdx.x;
  const bool c2 = tid >= 128;  // the third round is chroma's
  typename Quad<T>::W t[4][3];
  int d[4], cg[4], i[4];
  bool on[4];
  uint32_t over = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const bool chroma = k == 3 || (k == 2 && c2);
    i[k] = chroma ? (k == 2 ? tid - 128 : tid + 128) : tid + 256 * k;
    const bool second = chroma && i[k] >= 180;
    const int j = i[k] - (second ? 180 : 0);
    d[k] = chroma ? j / 10 : j / 18;
    cg[k] = j - (chroma ? 10 : 18) * d[k];
    on[k] = i[k] < (chroma ? 360 : 612);
    if (!kIn) {
      const CdefPlane& p = chroma ? Q : P;
      on[k] = on[k] && (chroma ? c : y) && 4 * cg[k] < p.w + 8 && 2 * d[k] < p.h + 4;
    }
    if (on[k]) {
      if (chroma)
        stage_load<T, kIn>(Q, second ? vsrc : Q.src, d[k], cg[k], t[k]);
      else
        stage_load<T, kIn>(P, P.src, d[k], cg[k], t[k]);
    }
  }
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (!on[k]) continue;
    over |= stage_over<T, kForm>(t[k]);
    if (k == 3 || (k == 2 && c2))
      stage_store<T, kIn, kForm, kPC>(Q, d[k], cg[k], t[k], sm.c[i[k] >= 180]);
    else
      stage_store<T, kIn, kForm, kPW>(P, d[k], cg[k], t[k], sm.y);
  }
  return over;
}

// Filters a run of `rows` rows (whole blocks of kBh) of one column, two rows
// at a time, so that a block's parameters are read once per block.  c: the
// run's first word; o: its first output sample; blk(k): the run's k-th
// block's parameters.
template <typename T, CdefForm kForm, bool kPri, bool kSec, int kBh, class B>
__device__ __forceinline__ void filter_run(const uint32_t* c, int pitch, const int2* ofs, uint8_t* o, int64_t os,
                                           int rows, const PairTap& st, B blk) {
#pragma unroll 1
  for (int k = 0; k * kBh < rows; k++) {
    const CdefBlk b = blk(k);
    const int dir = b.flags & 7;
    const bool filt = b.flags >> 31, odd = b.flags & 16;
    const int2 po = ofs[dir + 2], s0 = ofs[dir + 4], s1 = ofs[dir];
    const __half2 w0 = __float2half2_rn(odd ? 3.f : 4.f), w1 = __float2half2_rn(odd ? 3.f : 2.f);
#pragma unroll 1
    for (int y = 0; y < kBh; y += 2, c += 2 * pitch, o += 2 * os) {
      uint32_t v = c[0];
      if (filt) {
        if (kForm == kPairs) {
          v = pair_filter<kPri, kSec>(c, b.pri, w0, w1, st, po, s0, s1);
        } else if (kForm == kInts) {
          v = pair_filter_ints<kPri, kSec>(c, b.pri, odd ? 3 : 4, odd ? 3 : 2, st, po, s0, s1);
        } else {
          v = pair_filter_wide<kPri, kSec>(c, b.pri, odd ? 3 : 4, odd ? 3 : 2, st, po, s0, s1);
        }
      }
      if (sizeof(T) == 2 && kForm == kPairs) v &= 0x03ff03ffu;
      *reinterpret_cast<T*>(o) = (T)v;
      *reinterpret_cast<T*>(o + os) = (T)(v >> 16);
    }
  }
}

template <CdefForm kForm>
__device__ __forceinline__ PairTap cdef_tap(int thr, int shift) {
  return kForm == kPairs ? pair_tap(thr, shift) : kForm == kInts ? pair_tap_ints(thr, shift) : pair_tap_wide(thr, shift);
}

template <typename T, CdefForm kForm, int kBh, class B>
__device__ __forceinline__ void filter_plane(const uint32_t* c, int pitch, const int2* ofs, uint8_t* o, int64_t os,
                                             int rows, int pri, int sec, int damping, B blk) {
  const PairTap st = cdef_tap<kForm>(sec, constrain_shift(sec, damping));
  if (pri && sec)
    filter_run<T, kForm, true, true, kBh>(c, pitch, ofs, o, os, rows, st, blk);
  else if (pri)
    filter_run<T, kForm, true, false, kBh>(c, pitch, ofs, o, os, rows, st, blk);
  else
    filter_run<T, kForm, false, true, kBh>(c, pitch, ofs, o, os, rows, st, blk);
}

// The four rows b-2 .. b+1 around the restoration stripe boundary
// b = k*SH - off (k >= 1) that lies inside the unit (stripes are as high as
// units, so a unit of row ur has the one of k = ur + 1), saved from the
// pre-CDEF samples (tile/restoration_boundary.go:192-255): from the staged
// words (`staged` points at the unit's first one) or, where the plane was not
// staged, from the frame.  Thread `t` of a group saves sample t of the
// 4 x (64 >> xdec).
template <typename T>
__device__ __forceinline__ void cdef_save_lines(const CdefArgs& a, const DPlane& ip, const CdefPlane& p, int plane,
                                                int xdec, int ydec, int ur, const uint32_t* staged, int pitch,
                                                uint32_t mask, int t) {
  const int Hc = ip.h;
  const int k = ur + 1, b = (k << (6 - ydec)) - (8 >> ydec);
  const int j = t >> (6 - xdec), c = t & ((64 >> xdec) - 1);
  const int y = b - 2 + j, x = p.x + c;
  if (b < Hc && j < 4 && y < imin(p.y + p.h, Hc) && c < p.w && x < ip.w) {
    const T v = staged ? (T)(staged[(y - p.y) * pitch + c] & mask) : row_ptr<T>(ip, y)[x];
    uint8_t* line = a.lines[plane] + (int64_t)(k * 4 + j) * a.line_stride[plane];
    reinterpret_cast<T*>(line)[x] = v;
    if (j == 2 && b + 1 >= Hc) reinterpret_cast<T*>(line + a.line_stride[plane])[x] = v;
  }
}

// One 64x64 filter unit (uc, ur) of all planes.  4:2:0 units (k420) stage the
// three planes at once and go through the steps together: one wait for the
// frame's samples and four barriers a unit, where plane after plane took
// three waits and thirteen barriers, which is what a unit of few
// instructions spends its time on.  Other layouts' chroma is as large as
// luma or half of it and takes luma's place in shared memory, plane by
// plane.  Starts at plane `plane` (0 for k420) and returns 3, or the plane it
// stopped at, before writing it, because a sample there has more bits than the
// form takes; the next form goes on from that plane.
template <typename T, CdefForm kForm, bool k420>
__device__ __forceinline__ int cdef_unit(const FrameJob& J, int uc, int ur, int plane, CdefSmem& sm) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const CdefArgs& a = J.cdef;
  const int ssx = k420 ? 1 : J.io.ssx, ssy = k420 ? 1 : J.io.ssy;
  const int coeffShift = sizeof(T) == 1 ? 0 : (kForm == kPairs ? 2 : J.io.bd - 8);
  constexpr uint32_t kSample = kForm == kPairs ? 0x3ffu : 0xffffu;
  if (tid < 24) sm.ofs[tid / 12][tid % 12] = make_int2(pair_off(tid % 12, 0, tid < 12 ? kPW : kPC),
                                                       pair_off(tid % 12, 1, tid < 12 ? kPW : kPC));
  // ---- what the unit filters, postfilter_cdef.go:936-956 ----
  // The index map is only present when CDEF filters; the copy-only pass (CDEF
  // off, loop restoration on) reads no side information.
  int ystr = 0, uvstr = 0;
  uint64_t listed = 0;
  if (a.filter) {
    const int mapOff = ur * a.index_stride + uc;
    const int rd = a.read[mapOff], idx = a.index[mapOff];
    uint64_t word = ~0ull;
    if (a.noskip) {
      const uint8_t* w = a.noskip + (size_t)(ur * a.ucols + uc) * 8;
      if ((reinterpret_cast<uintptr_t>(w) & 7) == 0) {
        word = *reinterpret_cast<const uint64_t*>(w);
      } else {
        word = 0;
#pragma unroll
        for (int i = 0; i < 8; i++) word |= (uint64_t)w[i] << (8 * i);
      }
    }
    if (rd && idx < a.strength_count) {
      ystr = a.y_strength[idx];
      uvstr = a.uv_strength[idx];
      // The unit's 8x8 blocks inside the MI-aligned plane (the same in every plane).
      const int bcols = imin(8, (J.aw[0] - uc * 64) >> 3), brows = imin(8, (J.ah[0] - ur * 64) >> 3);
      const uint64_t cols = 0x0101010101010101ull * ((1u << bcols) - 1);
      listed = word & cols & (brows == 8 ? ~0ull : (1ull << (8 * brows)) - 1);
    }
  }
  const bool chromaPri = a.chroma_filtering && (uvstr >> 2) != 0;
  const bool actY = listed && a.plane_process[0] && (ystr || chromaPri);
  const bool actC = listed && a.plane_process[1] && uvstr;
  const bool needDir = actY && ((ystr >> 2) || chromaPri);
  const int nplanes = J.io.mono ? 1 : 3;
  for (; plane < nplanes; plane += k420 ? 3 : 1) {
    const int p1 = k420 ? nplanes : plane + 1;  // this pass: planes [plane, p1)
    // ---- stage ----
    uint32_t over = 0;
    CdefPlane P, Q;  // luma (or the one plane of the pass); k420: chroma
    const int xd = plane ? ssx : 0, yd = plane ? ssy : 0;
    const bool actP = plane ? actC : actY;
    P = cdef_plane(J.io.pl[plane], sizeof(T), (uc * 64) >> xd, (ur * 64) >> yd, 64 >> xd, 64 >> yd, J.aw[plane],
                   J.ah[plane]);
    if (P.w <= 0 || P.h <= 0) continue;
    if (k420) {
      Q = cdef_plane(J.io.pl[1], sizeof(T), uc * 32, ur * 32, 32, 32, J.aw[1], J.ah[1]);
      const uint8_t* const vsrc = J.io.pl[2].ptr;
      Q.words &= ((reinterpret_cast<uintptr_t>(vsrc) | (uintptr_t)J.io.pl[2].stride) & (4 * sizeof(T) - 1)) == 0;
      Q.words &= J.io.pl[2].stride == Q.stride;
      if (P.inside && P.words && Q.inside && Q.words && P.w == 64 && P.h == 64 && actY && actC) {
        over = stage_420<T, true, kForm>(P, Q, vsrc, true, true, sm);
      } else if (J.io.pl[2].stride == Q.stride) {
        over = stage_420<T, false, kForm>(P, Q, vsrc, actY, actC, sm);
      } else {
        if (actY) over |= stage_any<T, kForm, kPW>(P, P.src, sm.y);
        if (actC) {
          over |= stage_any<T, kForm, kPC>(Q, Q.src, sm.c[0]);
          CdefPlane V = Q;
          V.stride = J.io.pl[2].stride;
          over |= stage_any<T, kForm, kPC>(V, vsrc, sm.c[1]);
        }
      }
    } else if (actP) {
      over = stage_any<T, kForm, kPW>(P, P.src, sm.y);
    }
    if (sizeof(T) == 1 || kForm == kWide)
      __syncthreads();
    else if (__syncthreads_or((int)(over != 0)))
      return plane;
    // ---- luma direction search on listed blocks ----
    if (plane == 0 && needDir) {
      // A pair of warps takes two directions of the 64 blocks, so a warp
      // runs one code without divergence.
      const int b = tid & 63;
      const uint32_t* blk = &sm.y[(2 + (b >> 3) * 8) * kPW + kPX + (b & 7) * 8];
      if (!((listed >> b) & 1)) {
      } else if (kForm == kWide) {
        for (int d = tid >> 6; d < 8; d += 4) sm.cost[b * 8 + d] = dir_cost_wide_any(d, blk, coeffShift);
      } else {
        dir_costs_vert(tid >> 6, blk, kForm == kInts ? coeffShift : (sizeof(T) == 1 ? 0 : 2),
                       kForm == kInts ? (0xffffu >> coeffShift) * 0x10001u : 0x00ff00ffu, &sm.cost[b * 8]);
      }
      __syncthreads();
    }
    // ---- block parameters (cdef/filter.go:490-543): the adjusted luma
    // strength, the direction (0 when the primary strength is zero) ----
    int ypri = ystr >> 2, ysec = ystr & 3, cpri = uvstr >> 2, csec = uvstr & 3;
    ypri <<= coeffShift;
    cpri <<= coeffShift;
    ysec = (ysec + (ysec == 3)) << coeffShift;
    csec = (csec + (csec == 3)) << coeffShift;
    const int ydamp = a.damping + coeffShift, cdamp = ydamp - 1;
    if (plane == 0 && actY && tid < 64 && ((listed >> tid) & 1)) {
      int best = 0, var = 0;
      if (needDir) {
        const int4 c0 = *reinterpret_cast<const int4*>(&sm.cost[tid * 8]);
        const int4 c1 = *reinterpret_cast<const int4*>(&sm.cost[tid * 8 + 4]);
        const int32_t c[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
        int32_t top = c[0], across = c[4];  // the best direction's cost and that across it
#pragma unroll
        for (int d = 1; d < 8; d++)
          if (c[d] > top) {
            best = d;
            top = c[d];
            across = c[(d + 4) & 7];
          }
        var = (top - across) >> 10;
      }
      sm.dir[tid] = (uint8_t)best;
      // lumaAdjust holds whenever ypri is not zero: needDir does then.
      const int strength = ypri ? adjust_strength(ypri, var) : 0;
      CdefBlk blk;
      blk.pri = cdef_tap<kForm>(strength, constrain_shift(strength, ydamp));
      blk.flags = (strength | ysec ? 1u << 31 : 0u) | (((strength >> coeffShift) & 1) << 4) | (ypri ? best : 0);
      sm.blk[tid] = blk;
    } else if (!k420 && plane == 1 && actC && cpri && ssx != ssy && tid < 64 && ((listed >> tid) & 1)) {
      // cdef/filter.go:614-633: U converts the shared grid in place (V reuses
      // it): {7, 0, 2, 4, 5, 6, 6, 6} (4:2:2), {1, 2, 2, 2, 3, 4, 6, 0}
      // (4:4:0), four bits an entry.
      sm.dir[tid] = (uint8_t)(((ssx ? 0x66654207u : 0x06432221u) >> (4 * sm.dir[tid])) & 15);
    }
    __syncthreads();
    // ---- filter ----
    // The descriptors of the output in registers: they sit in the job table,
    // which the compiler would re-read after every store.
    if (plane == 0) {
      if (actY && ystr) {
        uint8_t* const ob = J.scr.pl[0].ptr;
        const int64_t os = J.scr.pl[0].stride;
        const int tx = tid & 63, ya = (tid >> 6) * 16, rows = imin(16, P.h - ya);
        if (tx < P.w && rows > 0)
          filter_plane<T, kForm, 8>(&sm.y[(2 + ya) * kPW + kPX + tx], kPW, sm.ofs[0],
                                   ob + (int64_t)(P.y + ya) * os + (int64_t)(P.x + tx) * (int)sizeof(T), os, rows, ypri,
                                   ysec, ydamp, [&](int k) {
                                     const int b = ((ya >> 3) + k) * 8 + (tx >> 3);
                                     CdefBlk r = sm.blk[b];
                                     if (!((listed >> b) & 1)) r.flags = 0;
                                     return r;
                                   });
      } else {
        copy_block<T>(J.io.pl[0], J.scr.pl[0], P.x, P.x + P.w, P.y, P.y + P.h);
      }
    }
    if (k420 ? nplanes > 1 : plane > 0) {
      CdefBlk cb;
      cb.pri = cdef_tap<kForm>(cpri, constrain_shift(cpri, cdamp));
      cb.flags = 1u << 31 | (((cpri >> coeffShift) & 1) << 4);
      auto chroma_blk = [&](int b) {
        CdefBlk r = cb;
        r.flags = (listed >> b) & 1 ? cb.flags | (cpri ? sm.dir[b] : 0) : 0;
        return r;
      };
      if (k420) {
        // Warps 0-3 take U, 4-7 V: 32 columns by 8 rows (two blocks) each.
        const int pl = 1 + (warp >> 2);
        uint8_t* const ob = J.scr.pl[pl].ptr;
        const int64_t os = J.scr.pl[pl].stride;
        const int ya = (warp & 3) * 8, rows = imin(8, Q.h - ya);
        if (!actC) {
          copy_block<T>(J.io.pl[1], J.scr.pl[1], Q.x, Q.x + Q.w, Q.y, Q.y + Q.h);
          copy_block<T>(J.io.pl[2], J.scr.pl[2], Q.x, Q.x + Q.w, Q.y, Q.y + Q.h);
        } else if (lane < Q.w && rows > 0) {
          filter_plane<T, kForm, 4>(&sm.c[pl - 1][(2 + ya) * kPC + kPX + lane], kPC, sm.ofs[1],
                                   ob + (int64_t)(Q.y + ya) * os + (int64_t)(Q.x + lane) * (int)sizeof(T), os, rows,
                                   cpri, csec, cdamp,
                                   [&](int k) { return chroma_blk(((ya >> 2) + k) * 8 + (lane >> 2)); });
        }
      } else if (!actC) {
        copy_block<T>(J.io.pl[plane], J.scr.pl[plane], P.x, P.x + P.w, P.y, P.y + P.h);
      } else {
        uint8_t* const ob = J.scr.pl[plane].ptr;
        const int64_t os = J.scr.pl[plane].stride;
        const int lw = 6 - ssx, tx = tid & ((1 << lw) - 1), rpt = (64 >> ssy) >> (8 - lw);
        const int ya = (tid >> lw) * rpt, rows = imin(rpt, P.h - ya);
        const uint32_t* c = &sm.y[(2 + ya) * kPW + kPX + tx];
        uint8_t* o = ob + (int64_t)(P.y + ya) * os + (int64_t)(P.x + tx) * (int)sizeof(T);
        if (tx < P.w && rows > 0) {
          auto at = [&](int k) { return chroma_blk(((ya >> (3 - ssy)) + k) * 8 + (tx >> (3 - ssx))); };
          if (ssy)
            filter_plane<T, kForm, 4>(c, kPW, sm.ofs[0], o, os, rows, cpri, csec, cdamp, at);
          else
            filter_plane<T, kForm, 8>(c, kPW, sm.ofs[0], o, os, rows, cpri, csec, cdamp, at);
        }
      }
    }
    // ---- fused loop-restoration boundary-line save ----
    if (k420) {
      if (a.save_lines[0])
        cdef_save_lines<T>(a, J.io.pl[0], P, 0, 0, 0, ur, actY ? &sm.y[2 * kPW + kPX] : nullptr, kPW, kSample, tid);
      if (nplanes > 1) {
        const int pl = 1 + (tid >> 7);
        if (a.save_lines[pl])
          cdef_save_lines<T>(a, J.io.pl[pl], Q, pl, 1, 1, ur, actC ? &sm.c[pl - 1][2 * kPC + kPX] : nullptr, kPC, kSample,
                             tid & 127);
      }
    } else if (a.save_lines[plane]) {
      cdef_save_lines<T>(a, J.io.pl[plane], P, plane, xd, yd, ur, actP ? &sm.y[2 * kPW + kPX] : nullptr, kPW, kSample, tid);
    }
    if (p1 < nplanes) __syncthreads();  // the next plane restages sm.y
  }
  return 3;
}

// The unit from plane `plane` on, with samples staged as integers: 12-bit
// frames, and 10-bit ones that hold longer samples.
template <CdefForm kForm>
__device__ __noinline__ int cdef_unit_ints(const FrameJob* J, int uc, int ur, int plane, CdefSmem* sm) {
  if (J->io.ssx && J->io.ssy) return cdef_unit<uint16_t, kForm, true>(*J, uc, ur, plane, *sm);
  return cdef_unit<uint16_t, kForm, false>(*J, uc, ur, plane, *sm);
}

// 4:2:2, 4:4:4 and 4:4:0.
template <typename T>
__device__ __noinline__ int cdef_unit_planes(const FrameJob* J, int uc, int ur, CdefSmem* sm) {
  return cdef_unit<T, kPairs, false>(*J, uc, ur, 0, *sm);
}

__device__ __forceinline__ void cdef_item(const FrameJob& J, int local, CdefSmem& sm) {
  const int uc = local % J.cdef.ucols, ur = local / J.cdef.ucols;
  const bool c420 = J.io.ssx && J.io.ssy;
  if (J.io.bd == 8) {
    if (c420)
      cdef_unit<uint8_t, kPairs, true>(J, uc, ur, 0, sm);
    else
      cdef_unit_planes<uint8_t>(&J, uc, ur, &sm);
  } else {
    int from = 0;
    if (J.io.bd == 10)
      from = c420 ? cdef_unit<uint16_t, kPairs, true>(J, uc, ur, 0, sm) : cdef_unit_planes<uint16_t>(&J, uc, ur, &sm);
    if (from < 3) from = cdef_unit_ints<kInts>(&J, uc, ur, from, &sm);
    if (from < 3) cdef_unit_ints<kWide>(&J, uc, ur, from, &sm);
  }
}

// Batched CDEF: each work item is one 64x64 unit of one frame.
template <bool kLoop>
__global__ void __launch_bounds__(256, 4) k_cdef_batch(BatchArgs b) {
  __shared__ CdefSmem sm;
  stage_begin();
  const int* base = b.base + ST_CDEF * (b.n + 1);
  for_each_item<kLoop>(
      b, ST_CDEF,
      [&](int item) {
        const int fi = find_frame(base, b.n, item);
        cdef_item(b.jobs[fi], item - base[fi], sm);
      },
      [&](int item) {
        // Every plane's unit with its 8-column / 2-row halo.
        const int fi = find_frame(base, b.n, item);
        const FrameJob& J = b.jobs[fi];
        const int local = item - base[fi];
        const int uc = local % J.cdef.ucols, ur = local / J.cdef.ucols;
        for (int plane = 0; plane < (J.io.mono ? 1 : 3); plane++) {
          const int xdec = plane ? J.io.ssx : 0, ydec = plane ? J.io.ssy : 0;
          const int x = (uc * 64) >> xdec, y = (ur * 64) >> ydec;
          if (J.io.bd == 8)
            prefetch_block<uint8_t>(J.io.pl[plane], x - 8, x + (64 >> xdec) + 8, y - 2, y + (64 >> ydec) + 2);
          else
            prefetch_block<uint16_t>(J.io.pl[plane], x - 8, x + (64 >> xdec) + 8, y - 2, y + (64 >> ydec) + 2);
        }
      });
}

__global__ void __launch_bounds__(256, 4) k_cdef_one(const __grid_constant__ FrameJob J) {
  __shared__ CdefSmem sm;
  stage_begin();
  cdef_item(J, blockIdx.x, sm);
}

cudaError_t launch_cdef(const StageLaunch& l) {
  if (l.total <= 0) return cudaSuccess;
  if (l.one) return launch_stage(k_cdef_one, l.total, 256, 0, l.st, l.dependent, *l.one);
  static int wave = 0;
  if (batch_loops(l.args)) return launch_stage(k_cdef_batch<true>, l.grid, 256, 0, l.st, l.dependent, l.args);
  return launch_stage(k_cdef_batch<false>, l.grid, 256, 0, l.st, l.dependent,
                      with_wave(l.args, k_cdef_batch<false>, 256, 0, wave));
}

}  // namespace pf
