// pf_search.cu - the encoder's CDEF strength search on the GPU.
//
// Follows goav1's cdefSearcher (internal/av1/encoder/cdef_search.go) over a
// trial list: level 1's (:98-110: all 64 packed strengths in the svtPfGI
// order, chroma the same list, row subsampling 1) for pf_cdef_search and the
// learned search, any level's for pf_cdef_search_ex (chroma trials the level
// does not measure, luma rows every subsamplingFactor-th with the SSE scaled
// back).  Trial indices past the list hold kNotATrial, which no selection
// step picks, so the selection over all 64 indices equals finish's over the
// list (:892-899: endGI = len(filterMap)):
//   k_cdef_search   a cluster of three CTAs per 64x64 filter block: the noskip
//                   8x8 list (computeCDEFList, :410-447), the VeryLarge-padded
//                   input (loadCDEFInput, :479-506), luma directions from the
//                   reconstruction, then for each tested trial the SSE of the
//                   filtered block against the source (searchRow, :649-745;
//                   FilterBlocksU8SubsampledTrusted with row step 1,
//                   cdef/filter_search.go:20-74).  An untested trial gets the
//                   reference's untested-chroma figure (cdefDefaultMSEUV*64,
//                   :669-672) in both planes.
//   k_sel_greedy    finish (:886-945): jointStrengthSearchDual /
//                   searchOneDual (:780-869) for one nb = 1 << cluster index,
//                   all 5*nb greedy and refinement steps inside one launch.
//                   The CTAs of a thread-block cluster each own a slice of
//                   the filter blocks (SSE rows in shared memory), compute
//                   partial savings sav[j][k] = sum_i max(0, best_i -
//                   m0[i][j] - m1[i][k]) (the reference's form), and hand
//                   them to the CTA that reduces the pair through
//                   distributed shared memory.  The refinement ends once nb
//                   steps in a row have changed nothing (no later one can).
//                   Bound by the barriers of a step, two of the cluster
//                   among them, hence maxima by warp reductions of one
//                   key and one thread's bookkeeping a step; 1080p: 303 us
//                   with all 40 steps of 8 presets run, 127 ended early, 85
//                   now; the learned search's 8 steps 62 and 42 (1,024
//                   threads a CTA instead of 512: 152 and 75).  Of a step's
//                   cycles the partial savings took 4,800 of 11,500 block by
//                   block (two at a time now, chroma rows negated), handing
//                   them over 2,600 (9,000 as 64-bit sums of eight
//                   neighbouring pairs a thread).
//   k_sel_finish    the RD choice of nb and the per-block preset index.
#include <cooperative_groups.h>
#include <string.h>

#include <vector>

#include "pf_cdef_dev.cuh"
#include "pf_search.cuh"

namespace cg = cooperative_groups;

namespace pf {

// ---- the trial search ----
//
// One cluster of three CTAs per 64x64 filter block: rank 0 the block's upper
// 32 luma rows, rank 1 the lower ones, rank 2 both chroma planes, which is
// the same number of samples each.  A warp takes 32 columns by 8 rows: a lane
// has one column as four pair words (pf_cdef_dev.cuh).
//
// What a trial's filter adds to a sample is the sum of a part that depends
// only on the primary strength (4 taps) and one that depends only on the
// secondary strength (8 taps), and the clamp range depends on neither.  So
// the 64 trials of a block need 15 primary sums and 3 secondary ones (and 3
// more with the direction that a zero primary strength implies) a sample, 108
// taps instead of 64 x 12, and the rest of a trial is one addition, the
// rounding, the clamp and the squared error of four samples at a time.
// Bound by the packed instructions themselves.  1080p: all 64 luma and 64
// chroma trials 107 us, trial by trial with constrain() tables about 1,500;
// the learned search's few trials a block 54 us, then 178.
//
// What a sample does not count for is settled once, before the trials: an
// unlisted block's, a skipped row's (subsampled search) has its clamp range,
// source and reconstruction set to the sample itself, so that every trial's
// error there is 0; one below or right of the crop, which the reference
// stages as VeryLarge and whose filtered 8-bit value is 0
// (cdef/filter_u8.go:151), has the range {-3}, whose low byte is 0.

constexpr int kSrchTab = 14;  // entries of a luma primary strength: zero variance, adjust index 0..12

struct SearchSmem {
  alignas(16) uint32_t w[36 * kPW];  // 36 rows of half a luma unit, or two chroma units (pitch kSrchPC)
  alignas(16) uint4 pri[16 * kSrchTab];  // PairTap; bit 0 odd strength, bit 1 zero strength
  alignas(16) uint4 sec[3];
  alignas(16) int32_t cost[64 * 8];
  uint32_t tested[2];  // strengths that some tested trial has (bit: packed strength)
  uint32_t sse[64];    // by packed strength
  int2 ofs[12];
  uint8_t dir[64];
  int8_t ai[64];  // adjustStrength index, -1 for zero variance
};
constexpr int kSrchPC = 40;
static_assert(2 * 36 * kSrchPC <= 36 * kPW, "chroma units fit the luma buffer");

// Stages pair words (four columns from x, two word rows from y) of a plane:
// frame samples inside the crop, absent ones outside it (loadCDEFInput,
// cdef_search.go:479-506).
__device__ __forceinline__ void search_stage(const DPlane& p, bool inside, int x, int y, uint32_t* o, int pitch) {
  uint32_t v[3], ok[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const uint8_t* r = p.ptr + (int64_t)(y + j) * p.stride + x;
    if (inside) {
      v[j] = *reinterpret_cast<const uint32_t*>(r);
    } else {
      v[j] = 0;
      ok[j] = 0;
      if (y + j >= 0 && y + j < p.h)
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (x + k >= 0 && x + k < p.w) {
            v[j] |= (uint32_t)r[k] << (8 * k);
            ok[j] |= 1u << k;
          }
    }
  }
#pragma unroll
  for (int j = 0; j < 2; j++) {
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
      w[k] = (__byte_perm(v[j], v[j + 1], 0x0400 + 0x0101 * k) & 0x00ff00ffu) | kPairBias;
      if (!inside) {
        const uint32_t keep = ((ok[j] >> k) & 1 ? 0xffffu : 0u) | ((ok[j + 1] >> k) & 1 ? 0xffff0000u : 0u);
        w[k] = (w[k] & keep) | (kPairNone & ~keep);
      }
    }
    *reinterpret_cast<uint4*>(o + j * pitch) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// The secondary sum of one pair at one strength from its eight differences
// (0..3: weight 2, 4..7: weight 1).
__device__ __forceinline__ __half2 search_sec(const __half2 (&d)[8], const uint4& c) {
  const PairTap t{c.x, c.y, c.z};
  const __half2 n = __hadd2(__hadd2(pair_constrain(d[0], t), pair_constrain(d[1], t)),
                            __hadd2(pair_constrain(d[2], t), pair_constrain(d[3], t)));
  const __half2 f = __hadd2(__hadd2(pair_constrain(d[4], t), pair_constrain(d[5], t)),
                            __hadd2(pair_constrain(d[6], t), pair_constrain(d[7], t)));
  return __hfma2(n, __float2half2_rn(2.f), f);
}

__device__ __forceinline__ uint32_t search_y(__half2 x, __half2 sum, uint32_t lo, uint32_t hi) {
  return __vminu2(__vmaxu2(h2_bits(pair_round(x, sum)), lo), hi);
}

// Adds the squared errors of the eight samples of two quads: ys, the four
// pairs' outcomes (8-bit samples in their low bytes), against the sources.
__device__ __forceinline__ uint32_t search_err(uint32_t y4, uint32_t s4, uint32_t acc) {
  const uint32_t d = __vabsdiffu4(y4, s4);
  return __dp4a(d, d, acc);
}

__global__ void __cluster_dims__(3, 1, 1) __launch_bounds__(256, 3) k_cdef_search(SearchArgs a) {
  stage_begin();
  __shared__ SearchSmem sm;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int fb = blockIdx.x / 3, rank = blockIdx.x - 3 * fb;
  const bool chroma = rank == 2;
  const int fbr = fb / a.nhfb, fbc = fb - fbr * a.nhfb;
  const int nfb = a.nhfb * a.nvfb;
  uint64_t* const m = a.mse + (size_t)(chroma ? nfb + fb : fb) * 64;
  const uint64_t listed = fb_listed(a, fb, 16 * fbr, 16 * fbc);
  const int count = a.trials.count;
  if (listed == 0) {
    // The whole cluster leaves before any barrier.
    if (tid < 64 && rank != 1) m[tid] = tid < count ? 0 : (uint64_t)kNotATrial;
    if (tid == 0 && rank == 0) a.skip[fb] = 1;
    return;
  }
  if (tid == 0 && rank == 0) a.skip[fb] = 0;
  const uint64_t listMask = count >= 64 ? ~0ull : (1ull << count) - 1;
  const uint64_t mask = a.tmask ? a.tmask[2 * fb + (chroma ? 1 : 0)] : (chroma ? a.trials.uvMask : listMask);
  // ---- stage, strengths, tap constants ----
  if (tid < 2) sm.tested[tid] = 0;
  if (tid < 64) sm.sse[tid] = 0;
  if (tid < 12) sm.ofs[tid] = make_int2(pair_off(tid, 0, chroma ? kSrchPC : kPW), pair_off(tid, 1, chroma ? kSrchPC : kPW));
  const int damping = chroma ? a.damping - 1 : a.damping;
  if (tid < 16 * kSrchTab) {
    const int p = tid / kSrchTab, e = tid - p * kSrchTab;
    const int strength = chroma ? p : (e == 0 ? 0 : (p * (3 + e) + 8) >> 4);
    const PairTap t = pair_tap(strength, constrain_shift(strength, damping));
    sm.pri[tid] = make_uint4(t.k, t.m, t.o, (uint32_t)(strength & 1) | (strength == 0 ? 2u : 0u));
  } else if (tid < 16 * kSrchTab + 3) {
    const int s = 1 << (tid - 16 * kSrchTab);
    const PairTap t = pair_tap(s, constrain_shift(s, damping));
    sm.sec[tid - 16 * kSrchTab] = make_uint4(t.k, t.m, t.o, 0);
  }
  if (!chroma) {
    const DPlane& rp = a.rec.pl[0];
    const int x = 64 * fbc - 4, y = 64 * fbr + 32 * rank - 2;
    const bool in = x >= 0 && x + 72 <= rp.w && y >= 0 && y + 37 <= rp.h &&
                    ((reinterpret_cast<uintptr_t>(rp.ptr) | (uintptr_t)rp.stride) & 3) == 0;
    for (int i = tid; i < 18 * 18; i += 256) {
      const int d = i / 18, cg4 = i - 18 * d;
      search_stage(rp, in, x + 4 * cg4, y + 2 * d, &sm.w[2 * d * kPW + 4 * cg4], kPW);
    }
  } else {
    for (int i = tid; i < 2 * 180; i += 256) {
      const int pl = i >= 180, j = i - (pl ? 180 : 0), d = j / 10, cg4 = j - 10 * d;
      const DPlane& rp = a.rec.pl[1 + pl];
      const int x = 32 * fbc - 4, y = 32 * fbr - 2;
      const bool in = x >= 0 && x + 40 <= rp.w && y >= 0 && y + 37 <= rp.h &&
                      ((reinterpret_cast<uintptr_t>(rp.ptr) | (uintptr_t)rp.stride) & 3) == 0;
      search_stage(rp, in, x + 4 * cg4, y + 2 * d, &sm.w[(pl * 36 + 2 * d) * kSrchPC + 4 * cg4], kSrchPC);
    }
  }
  __syncthreads();
  if (tid < 64 && ((mask >> tid) & 1)) {
    const int s = chroma ? a.trials.uv[tid] : a.trials.y[tid];
    atomicOr(&sm.tested[s >> 5], 1u << (s & 31));
  }
  // ---- luma directions of the listed blocks, from the reconstruction ----
  if (a.dirs) {
    // Found by the features kernel (same arithmetic).
    if (tid < 64 && ((listed >> tid) & 1)) {
      sm.dir[tid] = a.dirs[(size_t)fb * 64 + tid];
      sm.ai[tid] = a.ais[(size_t)fb * 64 + tid];
    }
    cl.sync();  // rank 0's sums are cleared before rank 1 can add to them
  } else {
    if (!chroma) {
      const DPlane& rp = a.rec.pl[0];
      const int x0 = 64 * fbc, y0 = 64 * fbr;
      const bool whole = x0 + 64 <= rp.w && y0 + 32 * rank + 32 <= rp.h;
      if (whole) {
        // A warp has two directions of the half's 32 blocks.
        const int b = rank * 32 + lane;
        if (warp < 4 && ((listed >> b) & 1))
          dir_costs_vert(warp, &sm.w[(2 + (lane >> 3) * 8) * kPW + kPX + (lane & 7) * 8], 0, 0x00ff00ffu,
                         &sm.cost[b * 8]);
      } else {
        // Blocks past the crop take their directions from the padding too.
        const int b = rank * 32 + lane;
        if ((listed >> b) & 1)
          sm.cost[b * 8 + warp] =
              dir_cost8_dev(warp, rp.ptr + (int64_t)(y0 + (b >> 3) * 8) * rp.stride + x0 + (b & 7) * 8, rp.stride);
      }
      __syncthreads();
      const int b = rank * 32 + tid;
      if (tid < 32 && ((listed >> b) & 1)) {
        int best = 0;
        int32_t bc = sm.cost[b * 8];
        for (int d = 1; d < 8; d++)
          if (sm.cost[b * 8 + d] > bc) {
            best = d;
            bc = sm.cost[b * 8 + d];
          }
        const int32_t var = (bc - sm.cost[b * 8 + ((best + 4) & 7)]) >> 10;
        sm.dir[b] = (uint8_t)best;
        int ai = -1;
        if (var != 0) {
          ai = 0;
          const int32_t v = var >> 6;
          if (v) ai = imin(31 - __clz(v), 12);
        }
        sm.ai[b] = (int8_t)ai;
      }
    }
    cl.sync();
    // The chroma CTA takes the directions from the two luma ones.
    if (chroma && tid < 64) sm.dir[tid] = cl.map_shared_rank(&sm.dir[0], tid >> 5)[tid];
    cl.sync();  // and they stay until it has
  }
  // ---- trials ----
  const uint64_t tested = sm.tested[0] | (uint64_t)sm.tested[1] << 32;
  if (tested) {
    const int pl = chroma ? 1 + (warp >> 2) : 0;
    const int pitch = chroma ? kSrchPC : kPW;
    // The lane's column and first row in the unit, and its word there.
    const int col = chroma ? lane : 32 * (warp & 1) + lane;
    const int row = chroma ? 8 * (warp & 3) : 32 * rank + 8 * (warp >> 1);
    const uint32_t* c = chroma ? &sm.w[((pl - 1) * 36 + 2 + row) * kSrchPC + kPX + col]
                               : &sm.w[(2 + row - 32 * rank) * kPW + kPX + col];
    const DPlane& sp = a.src.pl[pl];
    const int64_t at = (int64_t)((chroma ? 32 * fbr : 64 * fbr) + row);
    const int px = (chroma ? 32 * fbc : 64 * fbc) + col;
    // Per quad (four rows): its block, source and reconstruction samples; per
    // pair: the sample, the clamp range.
    int dir[2];
    uint32_t s4[2], r4[2], x[4], lo[4], hi[4], fix[4];
#pragma unroll
    for (int q = 0; q < 2; q++) {
      const int b = chroma ? ((row >> 2) + q) * 8 + (col >> 2) : (row >> 3) * 8 + (col >> 3);
      const bool on = (listed >> b) & 1;
      dir[q] = on ? sm.dir[b] : 0;
      // Rows that count: every ss-th of a luma block, all of a chroma one.
      uint32_t rows = on ? 0xffffffffu : 0u;
      if (!chroma && a.trials.ss > 1)
#pragma unroll
        for (int k = 0; k < 4; k++)
          if ((4 * q + k) % a.trials.ss) rows &= ~(0xffu << (8 * k));
      x[2 * q] = c[4 * q * pitch];
      x[2 * q + 1] = c[(4 * q + 2) * pitch];
      const uint32_t x4 = __byte_perm(x[2 * q], x[2 * q + 1], 0x6420);
      s4[q] = r4[q] = x4;
      if (on) {
        uint32_t s = 0;
        const uint8_t* sr = sp.ptr + (at + 4 * q) * sp.stride + px;
#pragma unroll
        for (int k = 0; k < 4; k++) s |= (uint32_t)sr[k * sp.stride] << (8 * k);
        s4[q] = (s & rows) | (x4 & ~rows);
      }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uint32_t xv = x[2 * q + h], rb = rows >> (16 * h);
        // Halves whose outcome is the sample itself whatever the trial:
        // those that do not count, and absent ones.
        uint32_t f = (rb & 1 ? 0u : 0xffffu) | (rb & 0x100 ? 0u : 0xffff0000u);
        if ((xv & 0xffffu) == (kPairNone & 0xffffu)) f |= 0xffffu;
        if ((xv >> 16) == (kPairNone >> 16)) f |= 0xffff0000u;
        fix[2 * q + h] = f;
      }
      if (on && ((fix[2 * q] | fix[2 * q + 1]) & (((x[2 * q] | x[2 * q + 1]) & 0x80008000u) >> 15)) != 0) {
        // Absent samples that count: the unfiltered trial measures the
        // reconstruction's padding.
        const DPlane& rp = a.rec.pl[pl];
        const uint8_t* rr = rp.ptr + (at + 4 * q) * rp.stride + px;
        uint32_t r = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) r |= (uint32_t)rr[k * rp.stride] << (8 * k);
        r4[q] = (r & rows) | (x4 & ~rows);
      }
    }
    auto put = [&](int strength, uint32_t e) {
      e = __reduce_add_sync(0xffffffffu, e);
      if (lane == 0) atomicAdd(&sm.sse[strength], e);
    };
    auto taps8 = [&](int j, const int2& s0, const int2& s1, uint32_t (&t)[8]) {
      const uint32_t* w = c + 2 * j * pitch;
      t[0] = w[s0.x], t[1] = w[-s0.x], t[2] = w[s1.x], t[3] = w[-s1.x];
      t[4] = w[s0.y], t[5] = w[-s0.y], t[6] = w[s1.y], t[7] = w[-s1.y];
    };
    // Primary strength 0: direction 0 whatever the block's, no clamp.
    if (tested & 1) put(0, search_err(r4[1], s4[1], search_err(r4[0], s4[0], 0)));
    if (tested & 14) {
      const int2 s0 = sm.ofs[4], s1 = sm.ofs[0];
      uint32_t y[3][4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        uint32_t t[8];
        __half2 d[8];
        taps8(j, s0, s1, t);
#pragma unroll
        for (int k = 0; k < 8; k++) d[k] = __hsub2(bits_h2(t[k]), bits_h2(x[j]));
        const uint32_t l = (fix[j] & x[j]) | (~fix[j] & 0x3c003c00u), h = (fix[j] & x[j]) | (~fix[j] & 0x3cff3cffu);
#pragma unroll
        for (int s = 0; s < 3; s++)
          if ((tested >> (s + 1)) & 1) y[s][j] = search_y(bits_h2(x[j]), search_sec(d, sm.sec[s]), l, h);
      }
#pragma unroll
      for (int s = 0; s < 3; s++)
        if ((tested >> (s + 1)) & 1)
          put(s + 1, search_err(__byte_perm(y[s][2], y[s][3], 0x6420), s4[1],
                                search_err(__byte_perm(y[s][0], y[s][1], 0x6420), s4[0], 0)));
    }
    if (tested >> 4) {
      // Some primary strength: the differences of its taps, the secondary
      // sums that any trial needs, the clamp range.
      __half2 d[4][4], sec[3][4];
      const uint64_t any = tested >> 4;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int2 po = sm.ofs[dir[j >> 1] + 2], s0 = sm.ofs[dir[j >> 1] + 4], s1 = sm.ofs[dir[j >> 1]];
        const uint32_t* w = c + 2 * j * pitch;
        const uint32_t p[4] = {w[po.x], w[-po.x], w[po.y], w[-po.y]};
        uint32_t t[8];
        taps8(j, s0, s1, t);
        uint32_t l = x[j], h = x[j];
        __half2 e[8];
#pragma unroll
        for (int k = 0; k < 4; k++) d[j][k] = __hsub2(bits_h2(p[k]), bits_h2(x[j]));
#pragma unroll
        for (int k = 0; k < 8; k++) e[k] = __hsub2(bits_h2(t[k]), bits_h2(x[j]));
        l = __vimin3_u16x2(__vimin3_u16x2(l, p[0], p[1]), p[2], p[3]);
        h = __vimax3_s16x2(__vimax3_s16x2(h, p[0], p[1]), p[2], p[3]);
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          l = __vimin3_u16x2(l, t[k], t[k + 1]);
          h = __vimax3_s16x2(h, t[k], t[k + 1]);
        }
        lo[j] = (l & ~fix[j]) | (x[j] & fix[j]);
        hi[j] = (h & ~fix[j]) | (x[j] & fix[j]);
#pragma unroll
        for (int s = 0; s < 3; s++) {
          sec[s][j] = __float2half2_rn(0.f);
          if (any & (0x1111111111111111ull << (s + 1))) sec[s][j] = search_sec(e, sm.sec[s]);
        }
      }
      const int e0 = chroma ? 0 : ((listed >> ((row >> 3) * 8 + (col >> 3))) & 1 ? sm.ai[(row >> 3) * 8 + (col >> 3)] + 1 : 0);
#pragma unroll 1
      for (int p = 1; p < 16; p++) {
        const uint32_t t4 = (uint32_t)(tested >> (4 * p)) & 15u;
        if (t4 == 0) continue;
        const uint4 k = sm.pri[p * kSrchTab + e0];
        const PairTap pt{k.x, k.y, k.z};
        const __half2 w0 = bits_h2(k.w & 1 ? 0x42004200u : 0x44004400u), w1 = bits_h2(k.w & 1 ? 0x42004200u : 0x40004000u);
        __half2 sum[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          sum[j] = __hmul2(w0, __hadd2(pair_constrain(d[j][0], pt), pair_constrain(d[j][1], pt)));
          sum[j] = __hfma2(w1, __hadd2(pair_constrain(d[j][2], pt), pair_constrain(d[j][3], pt)), sum[j]);
        }
        if (t4 & 1) {
          uint32_t y[4], e = 0;
#pragma unroll
          for (int j = 0; j < 4; j++) y[j] = search_y(bits_h2(x[j]), sum[j], lo[j], hi[j]);
#pragma unroll
          for (int q = 0; q < 2; q++) {
            const uint32_t y4 = __byte_perm(y[2 * q], y[2 * q + 1], 0x6420);
            e = search_err(k.w & 2 ? r4[q] : y4, s4[q], e);  // a zero strength leaves the block unfiltered
          }
          put(4 * p, e);
        }
#pragma unroll
        for (int s = 0; s < 3; s++)
          if (t4 & (2u << s)) {
            uint32_t y[4];
#pragma unroll
            for (int j = 0; j < 4; j++) y[j] = search_y(bits_h2(x[j]), __hadd2(sum[j], sec[s][j]), lo[j], hi[j]);
            put(4 * p + s + 1, search_err(__byte_perm(y[2], y[3], 0x6420), s4[1],
                                          search_err(__byte_perm(y[0], y[1], 0x6420), s4[0], 0)));
          }
      }
    }
  }
  __syncthreads();
  // ---- the table: rank 0 has luma's sums (rank 1 adds its own), rank 2 chroma's ----
  if (rank == 1 && tid < 64 && ((tested >> tid) & 1)) atomicAdd(&cl.map_shared_rank(&sm.sse[0], 0)[tid], sm.sse[tid]);
  cl.sync();
  if (rank != 1 && tid < 64) {
    uint64_t v;
    if (tid >= count)
      v = kNotATrial;
    else if ((mask >> tid) & 1)
      // A subsampled luma SSE is scaled back by the row step (searchRow, :722-734).
      v = (uint64_t)sm.sse[chroma ? a.trials.uv[tid] : a.trials.y[tid]] * (uint64_t)(chroma ? 1 : a.trials.ss);
    else
      v = (uint64_t)kUntestedMSE;
    m[tid] = v;
  }
}

// ---- greedy preset selection (finish) ----

struct SelShared {
  // Partial savings of this CTA's slice of the pairs, a row from each CTA of
  // the cluster (first pick: this CTA's column sums).
  alignas(16) unsigned long long part[4096];
  int narrow[kSelMaxCluster];  // whether a CTA's partial savings fit 32 bits
  unsigned long long cand[2][kSelMaxCluster];
  unsigned long long tot[kSelMaxCluster];  // rank 0's: every CTA's part of the total
  unsigned long long red[kSelThreads / 32];
  int wsum[kSelThreads / 32];
  int lev0[8], lev1[8];
  int done;
};

// A pair's saving with the pair's number below it, turned: the largest key is
// the first maximum.  A sum over the blocks (at most 2^16 of less than 2^31)
// is below kSelSumMax, so what it lacks of that serves for the first minimum.
constexpr unsigned long long kSelSumMax = 1ull << 50;
__device__ __forceinline__ unsigned long long sel_key(unsigned long long saving, int pair) {
  return saving << 12 | (unsigned long long)(4095 - pair);
}

// The warp's largest key, by its upper and then its lower word.
__device__ __forceinline__ unsigned long long warp_max(unsigned long long v) {
  const uint32_t hi = (uint32_t)(v >> 32), top = __reduce_max_sync(~0u, hi);
  return (unsigned long long)top << 32 | __reduce_max_sync(~0u, hi == top ? (uint32_t)v : 0u);
}

// The non-skip filter blocks in order (computeCDEFList's non-empty units):
// a ballot per warp and a running base; returns their count.  All threads
// of the block call it; `wsum` is one int per warp of scratch.
__device__ int compact_blocks(const uint8_t* skip, int nfb, int* list, int* wsum) {
  const int t = threadIdx.x, nw = blockDim.x >> 5;
  int base = 0;
  for (int b0 = 0; b0 < nfb; b0 += blockDim.x) {
    const int fb = b0 + t;
    const bool keep = fb < nfb && !skip[fb];
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    __syncthreads();  // the previous chunk of blocks is done with wsum
    if ((t & 31) == 0) wsum[t >> 5] = __popc(m);
    __syncthreads();
    int off = base;
    for (int w = 0; w < (t >> 5); w++) off += wsum[w];
    off += __popc(m & ((1u << (t & 31)) - 1));
    if (keep) list[off] = fb;
    for (int w = 0; w < nw; w++) base += wsum[w];
  }
  __syncthreads();
  return base;
}

// One cluster per configuration nb = 1 << (blockIdx.x / cluster size); the
// cluster size (16, or 8 where a 16-CTA cluster cannot be placed) is read at
// run time.  kRows: the filter blocks' SSE rows (as 32-bit values; an 8-bit
// 64x64 block's SSE is below 2^28) are copied into shared memory, chroma's
// negated.
template <bool kRows>
__global__ void __launch_bounds__(kSelThreads) k_sel_greedy(SelArgs a) {
  stage_begin();
  extern __shared__ __align__(16) unsigned char smem[];
  SelShared& S = *reinterpret_cast<SelShared*>(smem);
  int* s_sb = reinterpret_cast<int*>(smem + sizeof(SelShared));  // [nfb] non-skip blocks
  uint32_t* s_best = reinterpret_cast<uint32_t*>(s_sb + ((a.nfb + 3) & ~3));
  uint32_t* s_min1 = s_best + a.cap;
  // [cap][128] when kRows, on 16 bytes (the pool is, and sel_smem_bytes leaves room).
  uint32_t* s_rows = s_min1 + a.cap;
  s_rows += (4 - (((unsigned char*)s_rows - smem) >> 2 & 3)) & 3;
  cg::cluster_group cl = cg::this_cluster();
  const int CS = (int)cl.num_blocks();
  const int rank = (int)cl.block_rank();
  const int cfg = blockIdx.x / CS;
  const int nb = 1 << cfg;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int n = compact_blocks(a.skip, a.nfb, s_sb, S.wsum);
  SelOut* out = a.out;
  if (n == 0) {
    if (rank == 0 && t == 0) {
      for (int g = 0; g < 8; g++) out->lev0[cfg][g] = out->lev1[cfg][g] = 0;
      out->tot[cfg] = 0;
    }
    return;
  }
  const int per = (n + CS - 1) / CS;
  const int i0 = imin(n, rank * per), i1 = imin(n, i0 + per), cnt = i1 - i0;
  const int pairs = 4096 / CS;
  const uint64_t* M0 = a.mse;
  const uint64_t* M1 = a.mse + (size_t)a.nfb * 64;
  auto row = [&](int il, int pl, int j) -> uint32_t {
    if (kRows) return pl ? 0u - s_rows[il * 128 + 64 + j] : s_rows[il * 128 + j];
    const int fb = s_sb[i0 + il];
    return (uint32_t)(pl ? M1 : M0)[(size_t)fb * 64 + j];
  };
  if (kRows)
    for (int e = t; e < cnt * 128; e += kSelThreads) {
      const int il = e >> 7, pl = (e >> 6) & 1, j = e & 63;
      const int fb = s_sb[i0 + il];
      const uint32_t v = (uint32_t)(pl ? M1 : M0)[(size_t)fb * 64 + j];
      s_rows[e] = pl ? 0u - v : v;  // chroma's negated: a term of the savings as it stands
    }
  __syncthreads();
  unsigned long long most = 0;
  for (int il = warp; il < cnt; il += kSelThreads / 32) {
    const uint32_t a0 = row(il, 1, lane), a1 = row(il, 1, lane + 32);
    const uint32_t m = __reduce_min_sync(~0u, min(a0, a1));
    if (lane == 0) s_min1[il] = m;
    // No block saves more than its largest SSEs (places past the trial list
    // hold 2^31 - 1 and are never picked).
    auto held = [](uint32_t v) { return v == kNotATrial ? 0u : v; };
    most += __reduce_max_sync(~0u, max(held(a0), held(a1)));
    most += __reduce_max_sync(~0u, max(held(row(il, 0, lane)), held(row(il, 0, lane + 32))));
  }
  if (lane == 0) S.red[warp] = most;
  if (t < 8) S.lev0[t] = S.lev1[t] = 0;
  __syncthreads();
  if (t < CS) {
    most = 0;
    for (int i = 0; i < kSelThreads / 32; i++) most += S.red[i];
  }
  const int steps = a.refine ? 5 * nb : nb;
  int same = 0, drop0 = 0, drop1 = 0;  // thread 0's: refinement steps in a row that took back the pick they had dropped
  for (int k = 0; k < steps; k++) {
    const int nbCur = k < nb ? k : nb - 1;
    const int par = k & 1;
    if (nbCur == 0) {
      // First pick: the luma and chroma strengths with the least total SSE.
      if (t < 128) {
        unsigned long long s = 0;
        for (int il = 0; il < cnt; il++) s += row(il, t >> 6, t & 63);
        S.part[t] = s;
      }
      cl.sync();  // (the first: every CTA of the cluster has started)
      if (t < CS) cl.map_shared_rank(&S, t)->narrow[rank] = most < 1ull << 32;
      if (t < 128) {
        unsigned long long s0 = 0, s1 = 0, s2 = 0, s3 = 0;
        for (int r = 0; r < CS; r += 4) {
          s0 += cl.map_shared_rank(&S.part[0], r)[t];
          s1 += cl.map_shared_rank(&S.part[0], r + 1)[t];
          s2 += cl.map_shared_rank(&S.part[0], r + 2)[t];
          s3 += cl.map_shared_rank(&S.part[0], r + 3)[t];
        }
        const unsigned long long sum = (s0 + s1) + (s2 + s3);
        // The first minimum of each plane's 64 sums, two warps a plane.
        const unsigned long long best = warp_max(sel_key(kSelSumMax - sum, t & 63));
        if (lane == 0) S.red[warp] = best;
      }
      __syncthreads();
      if (t == 0) {
        S.lev0[0] = 4095 - (int)(max(S.red[0], S.red[1]) & 4095);
        S.lev1[0] = 4095 - (int)(max(S.red[2], S.red[3]) & 4095);
      }
      cl.sync();  // every CTA has read the others' column sums
    } else {
      // best_i over the strengths selected so far.
      for (int il = t; il < cnt; il += kSelThreads) {
        uint32_t best = row(il, 0, S.lev0[0]) + row(il, 1, S.lev1[0]);
        for (int g = 1; g < nbCur; g++) best = min(best, row(il, 0, S.lev0[g]) + row(il, 1, S.lev1[g]));
        s_best[il] = best;
      }
      __syncthreads();
      // Partial savings of this CTA's blocks: thread t owns (j, k) for the
      // strengths k = 32 m + 4 (t & 7) + 0..3, so that eight neighbours' sums
      // are 128 bytes of a row when they are handed over.  A block saves
      // below 2^29, so eight blocks sum exactly in 32 bits before joining the
      // 64-bit totals; all of them do where the CTA's narrow flag says so.
      const bool narrow = S.narrow[rank];
      const int j = t >> 3, k0 = (t & 7) * 4;
      unsigned long long acc[8];
      uint32_t acc32[8];
#pragma unroll
      for (int q = 0; q < 8; q++) acc[q] = acc32[q] = 0;
      for (int il0 = 0; il0 < cnt; il0 += 8) {
        const int il1 = imin(cnt, il0 + 8);
        for (int il = il0; il < il1; il += 2) {
          // Two blocks a pass (the odd last one twice, the second time with
          // nothing left to save).
          const int ih = imin(il + 1, cnt - 1);
          const uint32_t b0 = s_best[il], b1 = s_best[ih], a0 = row(il, 0, j), a1 = row(ih, 0, j);
          const bool on0 = a0 + s_min1[il] < b0, on1 = ih > il && a1 + s_min1[ih] < b1;
          if (!on0 && !on1) continue;  // no k can save anything
          // Saved so far without chroma.  Both are below 2^30 where on and a
          // sentinel is 2^31 - 1, so no difference can overflow.
          const int rem0 = on0 ? (int)(b0 - a0) : 0, rem1 = on1 ? (int)(b1 - a1) : 0;
          uint32_t v0[8], v1[8];
          auto load = [&](int i, uint32_t (&v)[8]) {
            if (kRows) {
#pragma unroll
              for (int m = 0; m < 2; m++) {
                const uint4 x = *reinterpret_cast<const uint4*>(&s_rows[i * 128 + 64 + 32 * m + k0]);
                v[4 * m] = x.x, v[4 * m + 1] = x.y, v[4 * m + 2] = x.z, v[4 * m + 3] = x.w;
              }
            } else {
#pragma unroll
              for (int q = 0; q < 8; q++) v[q] = 0u - row(i, 1, 32 * (q >> 2) + k0 + (q & 3));
            }
          };
          load(il, v0);
          load(ih, v1);
#pragma unroll
          for (int q = 0; q < 8; q++)
            acc32[q] += (uint32_t)__viaddmax_s32((int)v0[q], rem0, 0) + (uint32_t)__viaddmax_s32((int)v1[q], rem1, 0);
        }
        if (narrow) continue;
#pragma unroll
        for (int q = 0; q < 8; q++) {
          acc[q] += acc32[q];
          acc32[q] = 0;
        }
      }
      // Each CTA reduces a slice of the pairs: the eight sums go straight
      // into their slice's CTA (rows of one sender each), so that only the
      // barrier is waited for and every read after it is local.
      {
        const int e0 = j * 64 + k0, to = e0 / pairs;
        unsigned long long* d = cl.map_shared_rank(&S.part[0], to) + rank * pairs;  // the sender's row
        const int at = e0 - to * pairs;
        if (narrow) {
          uint32_t* d32 = reinterpret_cast<uint32_t*>(d) + at;
#pragma unroll
          for (int m = 0; m < 2; m++)
            *reinterpret_cast<uint4*>(d32 + 32 * m) =
                make_uint4(acc32[4 * m], acc32[4 * m + 1], acc32[4 * m + 2], acc32[4 * m + 3]);
        } else {
#pragma unroll
          for (int q = 0; q < 8; q += 2)
            *reinterpret_cast<ulonglong2*>(d + at + 32 * (q >> 2) + (q & 3)) = make_ulonglong2(acc[q], acc[q + 1]);
        }
      }
      cl.sync();
      // First maximum wins.  Two neighbouring threads share a pair.
      unsigned long long key = 0;
      for (int e2 = t; e2 < 2 * pairs; e2 += kSelThreads) {
        const int e = e2 >> 1, r0 = (e2 & 1) * (CS >> 1);
        unsigned long long sum = 0;
#pragma unroll
        for (int r = 0; r < kSelMaxCluster / 2; r++)
          if (r < (CS >> 1)) {
            const unsigned long long* from = &S.part[(r0 + r) * pairs];
            sum += S.narrow[r0 + r] ? reinterpret_cast<const uint32_t*>(from)[e] : from[e];
          }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        key = max(key, sel_key(sum, rank * pairs + e));
      }
      key = warp_max(key);
      if (lane == 0) S.red[warp] = key;
      __syncthreads();
      if (warp == 0) {
        key = warp_max(lane < kSelThreads / 32 ? S.red[lane] : 0);
        // Lane r hands this CTA's candidate to rank r (alternate steps use
        // alternate places).
        if (lane < CS) cl.map_shared_rank(&S, lane)->cand[par][rank] = key;
      }
      cl.sync();
      if (warp == 0) {
        key = warp_max(lane < CS ? S.cand[par][lane] : 0);
        if (lane == 0) {
          const int i = 4095 - (int)(key & 4095);
          S.lev0[nbCur] = i >> 6;
          S.lev1[nbCur] = i & 63;
        }
      }
    }
    if (t == 0) {
      // A pick depends only on the set of the other nb - 1, so once nb steps
      // in a row have taken back what they dropped, every later one does: the
      // remaining steps only turn the list, which is then done at once.
      if (k >= nb) same = S.lev0[nb - 1] == drop0 && S.lev1[nb - 1] == drop1 ? same + 1 : 0;
      const int turn = same == nb ? (steps - 1 - k) % nb : 1;
      // Refinement passes drop the oldest pick (jointStrengthSearchDual).
      if (k + 1 >= nb && k + 1 < steps) {
        drop0 = S.lev0[0];
        drop1 = S.lev1[0];
        for (int q = 0; q < turn; q++) {
          const int l0 = S.lev0[0], l1 = S.lev1[0];
          for (int g = 0; g < nb - 1; g++) {
            S.lev0[g] = S.lev0[g + 1];
            S.lev1[g] = S.lev1[g + 1];
          }
          S.lev0[nb - 1] = l0;
          S.lev1[nb - 1] = l1;
        }
      }
      S.done = same == nb;
    }
    __syncthreads();
    if (S.done) break;
  }
  // The total SSE with the picks.
  unsigned long long tot = 0;
  for (int il = t; il < cnt; il += kSelThreads) {
    uint32_t best = row(il, 0, S.lev0[0]) + row(il, 1, S.lev1[0]);
    for (int g = 1; g < nb; g++) best = min(best, row(il, 0, S.lev0[g]) + row(il, 1, S.lev1[g]));
    tot += best;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  if (lane == 0) S.red[warp] = tot;
  __syncthreads();
  if (t == 0) {
    tot = 0;
    for (int i = 0; i < kSelThreads / 32; i++) tot += S.red[i];
    cl.map_shared_rank(&S, 0)->tot[rank] = tot;
  }
  cl.sync();
  if (rank == 0 && t == 0) {
    for (int g = 0; g < 8; g++) {
      out->lev0[cfg][g] = g < nb ? S.lev0[g] : 0;
      out->lev1[cfg][g] = g < nb ? S.lev1[g] : 0;
    }
    tot = 0;
    for (int r = 0; r < CS; r++) tot += S.tot[r];
    out->tot[cfg] = tot;
  }
}

// RD choice of nb (finish, :914-931) and the per-block preset index.
__global__ void __launch_bounds__(256) k_sel_finish(SelArgs a, int maxCfg, unsigned long long lambda, uint8_t* fbIndex,
                                                    FinishOut* fo) {
  stage_begin();
  __shared__ int s_best, s_n;
  const SelOut* st = a.out;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  {
    int c = 0;
    for (int fb = threadIdx.x; fb < a.nfb; fb += blockDim.x) c += !a.skip[fb];
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(&s_n, c);
  }
  __syncthreads();
  const int n = s_n;
  if (threadIdx.x == 0) {
    unsigned long long bestTot = 1ull << 63;
    int best = 0;
    for (int c = 0; c <= maxCfg; c++) {
      const int nb = 1 << c;
      const long long rate = (long long)(n * c + nb * 6 * 2) << 9;
      const unsigned long long cost =
          (unsigned long long)((rate * (long long)lambda + (1 << 8)) >> 9) + ((st->tot[c] * 16ull) << 7);
      if (cost < bestTot) {
        bestTot = cost;
        best = c;
      }
    }
    s_best = best;
    if (blockIdx.x == 0) {
      fo->bits = best;
      fo->cost = bestTot;
      for (int j = 0; j < (1 << best); j++) {
        fo->ys[j] = st->lev0[best][j];
        fo->uvs[j] = a.uvFromY ? st->lev0[best][j] : st->lev1[best][j];
      }
    }
  }
  __syncthreads();
  const int c = s_best, nb = 1 << c;
  const uint64_t* M0 = a.mse;
  const uint64_t* M1 = a.mse + (size_t)a.nfb * 64;
  for (int fb = blockIdx.x * blockDim.x + threadIdx.x; fb < a.nfb; fb += gridDim.x * blockDim.x) {
    if (a.skip[fb]) {
      fbIndex[fb] = 0;
      continue;
    }
    int bg = 0;
    unsigned long long bm = 1ull << 63;
    for (int g = 0; g < nb; g++) {
      const int uvg = a.uvFromY ? st->lev0[c][g] : st->lev1[c][g];
      const unsigned long long v = M0[(size_t)fb * 64 + st->lev0[c][g]] + M1[(size_t)fb * 64 + uvg];
      if (v < bm) {
        bg = g;
        bm = v;
      }
    }
    fbIndex[fb] = (uint8_t)bg;
  }
}

size_t sel_smem_bytes(int nfb, bool rows) {
  const int cap = (nfb + kSelMinCluster - 1) / kSelMinCluster;
  return sizeof(SelShared) + (size_t)((nfb + 3) & ~3) * 4 + (size_t)cap * 8 + (rows ? (size_t)cap * 512 + 16 : 0);
}

cudaError_t launch_search(const SearchArgs& a, cudaStream_t st) {
  // After the mask kernel (tmask) the CTAs are placed while that one drains.
  return launch_stage(k_cdef_search, 3 * a.nhfb * a.nvfb, 256, 0, st, a.tmask != nullptr, a);
}

// Launches k_sel_greedy with 16-CTA clusters when the device can place one
// with this much shared memory, else with 8-CTA clusters.  Not as a
// programmatic dependent: its clusters, placed while the search drains, took
// the exhaustive 1080p call from 260 to 300 us.
template <bool kRows>
static cudaError_t launch_greedy(const SelArgs& s, int maxCfg, size_t bytes, cudaStream_t st) {
  const void* fn = (const void*)k_sel_greedy<kRows>;
  // The attributes and the cluster size are settled once per device and
  // shared-memory size (host queries cost more than the short launches).
  static thread_local int lastDev = -1;
  static thread_local size_t lastBytes = 0;
  static thread_local int lastCs = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev == lastDev && bytes <= lastBytes && lastCs) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = lastCs;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(lastCs * (maxCfg + 1));
    cfg.blockDim = dim3(kSelThreads);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_sel_greedy<kRows>, s);
  }
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kSelThreads);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int cs = kSelMaxCluster;
  for (; cs > kSelMinCluster; cs >>= 1) {
    attr[0].val.clusterDim.x = cs;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(cs * (maxCfg + 1));
    int nclusters = 0;
    if (cudaOccupancyMaxActiveClusters(&nclusters, fn, &cfg) == cudaSuccess && nclusters >= 1) break;
    cudaGetLastError();  // a refused query leaves no sticky error
  }
  attr[0].val.clusterDim.x = cs;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(cs * (maxCfg + 1));
  e = cudaLaunchKernelEx(&cfg, k_sel_greedy<kRows>, s);
  if (e == cudaSuccess) {
    lastDev = dev;
    lastBytes = bytes;
    lastCs = cs;
  }
  return e;
}

cudaError_t launch_select(SelArgs s, int maxCfg, unsigned long long lambda, uint8_t* fbIndex, FinishOut* fo,
                          cudaStream_t st) {
  s.cap = (s.nfb + kSelMinCluster - 1) / kSelMinCluster;
  const bool rows = sel_smem_bytes(s.nfb, true) <= kSelMaxSmem;
  const size_t bytes = sel_smem_bytes(s.nfb, rows);
  if (bytes > kSelMaxSmem) return cudaErrorInvalidValue;
  const cudaError_t e = rows ? launch_greedy<true>(s, maxCfg, bytes, st) : launch_greedy<false>(s, maxCfg, bytes, st);
  if (e != cudaSuccess) return e;
  return launch_stage(k_sel_finish, imax(1, (s.nfb + 255) / 256), 256, 0, st, true, s, maxCfg, lambda, fbIndex, fo);
}

}  // namespace pf

using namespace pf;

// ---------------------------------------------------------------------------
// Host side: the search entry points.  Scratch comes from a cache the context
// keeps (grown, never shrunk); host frames are staged like pf_frame_apply's.

void* pf_internal_search_scratch(pf_ctx* c, size_t bytes);  // pf_api.cu
void* pf_internal_stream(pf_ctx* c);
cudaEvent_t* pf_internal_events(pf_ctx* c);  // pf_api.cu: null unless the context times stages
void* pf_internal_pinned(pf_ctx* c, size_t bytes);
void* pf_internal_fork(pf_ctx* c);  // pf_api.cu
bool pf_internal_join(pf_ctx* c);
bool pf_internal_bounded(const pf_ctx* c);
void* pf_internal_cached_upload(pf_ctx* c, const void* host, size_t bytes, size_t extra, cudaStream_t st,
                                int* changed);
int pf_internal_wait(pf_ctx* c, void* stream);  // pf_api.cu: blocking or bounded by the context's deadline

static void* stage_frame(const pf_frame* f, void* dst, int64_t* strides, cudaStream_t st, cudaError_t* e) {
  size_t off = 0;
  for (int p = 0; p < 3; p++) {
    strides[p] = ((int64_t)f->plane[p].alloc_width + 255) & ~(int64_t)255;
    off += (size_t)strides[p] * f->plane[p].alloc_height;
  }
  if (!dst) return (void*)off;
  uint8_t* base = (uint8_t*)dst;
  for (int p = 0; p < 3 && *e == cudaSuccess; p++) {
    *e = cudaMemcpy2DAsync(base, strides[p], f->plane[p].data, f->plane[p].stride, f->plane[p].alloc_width,
                           f->plane[p].alloc_height, cudaMemcpyHostToDevice, st);
    base += (size_t)strides[p] * f->plane[p].alloc_height;
  }
  return dst;
}

static DFrame search_dframe(const pf_frame* f, uint8_t* const* ptrs, const int64_t* strides) {
  DFrame d;
  memset(&d, 0, sizeof(d));
  d.width = f->width;
  d.height = f->height;
  d.bd = 8;
  d.ssx = d.ssy = 1;
  for (int p = 0; p < 3; p++) {
    d.pl[p].ptr = ptrs[p];
    d.pl[p].stride = strides[p];
    d.pl[p].w = f->plane[p].width;
    d.pl[p].h = f->plane[p].height;
    d.pl[p].aw = f->plane[p].alloc_width;
    d.pl[p].ah = f->plane[p].alloc_height;
  }
  return d;
}

// Validation, staging and scratch shared by the search entry points.
// Scratch: [staged src | staged rec | noskip | mse | skip | SelOut |
//           FinishOut | fbIndex | caller's extra bytes].
struct Staged {
  SearchArgs a;
  SelArgs s;
  uint8_t* idx;
  FinishOut* fo;
  uint8_t* extra;
  uint8_t* pin;  // page-locked staging: noskip words up, then the results down, then the SSE table
  int nfb, maxCfg;
  cudaStream_t st;
  pf_ctx* ctx;
};

static int check_search_frame(const pf_frame* f, const pf_frame* recon) {
  // goav1's searcher works on 8-bit 4:2:0 pictures (SourceFrame420).
  if (f->bit_depth != 8 || f->ss_x != 1 || f->ss_y != 1 || f->mono || f->width != recon->width ||
      f->height != recon->height)
    return PF_ERR_UNSUPPORTED;
  if (f->memory != recon->memory || f->memory > PF_MEM_DEVICE) return PF_ERR_INVALID_ARG;
  for (int p = 0; p < 3; p++) {
    const int w = p ? (recon->width + 1) >> 1 : recon->width, h = p ? (recon->height + 1) >> 1 : recon->height;
    const int aw8 = ((recon->width + 7) & ~7) >> (p ? 1 : 0), ah8 = ((recon->height + 7) & ~7) >> (p ? 1 : 0);
    const pf_plane& pl = f->plane[p];
    if (!pl.data || pl.width != w || pl.height != h || pl.alloc_width < aw8 || pl.alloc_height < ah8 ||
        pl.stride < pl.alloc_width)
      return PF_ERR_SHORT_BUFFER;
  }
  return PF_OK;
}

static void level1_trials(TrialList* t);

// source may be null (features only: the source is never read).  table: the
// SSE table will be wanted.
static int stage_search(pf_ctx* ctx, const pf_frame* source, const pf_frame* recon, const uint8_t* noskip,
                        int damping, int maxCfg, size_t extra, bool table, Staged* S) {
  int stt = check_search_frame(recon, recon);
  if (stt == PF_OK && source) stt = check_search_frame(source, recon);
  if (stt != PF_OK) return stt;
  if (damping < 3 || damping > 6) return PF_ERR_INVALID_CDEF;
  const int miCols = ((recon->width + 7) >> 3) << 1, miRows = ((recon->height + 7) >> 3) << 1;
  const int nhfb = (miCols + 15) / 16, nvfb = (miRows + 15) / 16, nfb = nhfb * nvfb;
  if (sel_smem_bytes(nfb, false) > kSelMaxSmem) return PF_ERR_UNSUPPORTED;
  const cudaStream_t st = (cudaStream_t)pf_internal_stream(ctx);
  const bool host = recon->memory == PF_MEM_HOST;
  int64_t sS[3] = {0, 0, 0}, rS[3];
  cudaError_t e = cudaSuccess;
  const size_t srcBytes = host && source ? (size_t)stage_frame(source, nullptr, sS, st, &e) : 0;
  const size_t recBytes = host ? (size_t)stage_frame(recon, nullptr, rS, st, &e) : 0;
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  size_t off = 0;
  const size_t oSrc = off; off += al(srcBytes);
  const size_t oRec = off; off += al(recBytes);
  const size_t oNs = off; off += al((size_t)nfb * 8);
  const size_t oMse = off; off += al((size_t)2 * nfb * 64 * 8);
  const size_t oSkip = off; off += al(nfb);
  const size_t oSel = off; off += al(sizeof(SelOut));
  const size_t oFin = off; off += al(sizeof(FinishOut));
  const size_t oIdx = off; off += al(nfb);
  const size_t oExtra = off; off += al(extra);
  uint8_t* base = (uint8_t*)pf_internal_search_scratch(ctx, off);
  if (!base) return PF_ERR_DEVICE;
  uint8_t* sp[3] = {nullptr, nullptr, nullptr};
  uint8_t* rpp[3];
  if (host) {
    if (source) stage_frame(source, base + oSrc, sS, st, &e);
    stage_frame(recon, base + oRec, rS, st, &e);
    size_t o1 = 0, o2 = 0;
    for (int p = 0; p < 3; p++) {
      if (source) {
        sp[p] = base + oSrc + o1;
        o1 += (size_t)sS[p] * source->plane[p].alloc_height;
      }
      rpp[p] = base + oRec + o2;
      o2 += (size_t)rS[p] * recon->plane[p].alloc_height;
    }
  } else {
    for (int p = 0; p < 3; p++) {
      if (source) {
        sp[p] = (uint8_t*)source->plane[p].data;
        sS[p] = source->plane[p].stride;
      }
      rpp[p] = (uint8_t*)recon->plane[p].data;
      rS[p] = recon->plane[p].stride;
    }
  }
  // The noskip words may live in host or device memory: copy them into the
  // scratch either way; host words go through page-locked staging so the
  // copy does not hold the host.
  // One page-locked block for the call (requested once, so it never moves
  // while a copy is queued): the noskip words, the selection results, the SSE
  // table.
  uint8_t* pin = (uint8_t*)pf_internal_pinned(ctx, al((size_t)nfb * 8) + al(sizeof(FinishOut)) + al(nfb) +
                                                       (table ? (size_t)2 * nfb * 64 * 8 : 0));
  if (!pin) return PF_ERR_DEVICE;
  S->pin = pin;
  const uint8_t* ns = nullptr;
  if (noskip && e == cudaSuccess) {
    cudaPointerAttributes at;
    const bool dev = cudaPointerGetAttributes(&at, noskip) == cudaSuccess &&
                     (at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged);
    cudaGetLastError();
    if (dev) {
      e = cudaMemcpyAsync(base + oNs, noskip, (size_t)nfb * 8, cudaMemcpyDeviceToDevice, st);
    } else {
      memcpy(pin, noskip, (size_t)nfb * 8);
      e = cudaMemcpyAsync(base + oNs, pin, (size_t)nfb * 8, cudaMemcpyHostToDevice, st);
    }
    ns = base + oNs;
  }
  if (e != cudaSuccess) return PF_ERR_DEVICE;
  SearchArgs& a = S->a;
  a.src = source ? search_dframe(source, sp, sS) : search_dframe(recon, rpp, rS);
  a.rec = search_dframe(recon, rpp, rS);
  a.noskip = ns;
  a.tmask = nullptr;
  a.miCols = miCols;
  a.miRows = miRows;
  a.nhfb = nhfb;
  a.nvfb = nvfb;
  a.damping = damping;
  a.mse = (uint64_t*)(base + oMse);
  a.skip = base + oSkip;
  a.dirs = nullptr;
  a.ais = nullptr;
  level1_trials(&a.trials);
  SelArgs& s = S->s;
  s.mse = a.mse;
  s.skip = a.skip;
  s.nfb = nfb;
  s.cap = 0;
  s.refine = 1;
  s.uvFromY = 0;
  s.out = (SelOut*)(base + oSel);
  S->idx = base + oIdx;
  S->fo = (FinishOut*)(base + oFin);
  S->extra = base + oExtra;
  S->nfb = nfb;
  S->maxCfg = maxCfg;
  S->st = st;
  S->ctx = ctx;
  return PF_OK;
}

// The level-1 list (cdef_search.go:98-110).
static void level1_trials(TrialList* t) {
  memset(t, 0, sizeof(*t));
  for (int g = 0; g < 64; g++) t->y[g] = t->uv[g] = (int8_t)trial_strength(g);
  t->uvMask = ~0ull;
  t->count = 64;
  t->ss = 1;
}

static int search_damping(const pf_cdef_search_params* params) {
  return params->damping ? params->damping : 3 + (params->qindex >> 6);
}

static int search_max_cfg(const pf_cdef_search_params* params) {
  return params->max_presets >= 8 ? 3 : params->max_presets >= 4 ? 2 : params->max_presets >= 2 ? 1 : 0;
}

// Search (with S.a.tmask already set by the caller, or null), selection,
// results to the host.
static int search_finish(Staged& S, const pf_cdef_search_params* params, uint64_t* mse_out, uint8_t* fb_index_out,
                         pf_cdef_search_result* result, cudaEvent_t* ev = nullptr) {
  const cudaStream_t st = S.st;
  if (launch_search(S.a, st) != cudaSuccess) return PF_ERR_DEVICE;
  if (ev && cudaEventRecord(ev[3], st) != cudaSuccess) return PF_ERR_DEVICE;
  // The small results come back through the page-locked block (a pageable
  // destination would make each copy a staged, synchronous one).  So does
  // the SSE table (522 KB at 1080p, 58 us of the call as a pageable copy at
  // its end): on the second stream and on to the caller beside the selection,
  // which does not write it.
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  uint8_t* pfo = S.pin + al((size_t)S.nfb * 8);
  uint8_t* pidx = pfo + al(sizeof(FinishOut));
  uint8_t* ptab = pidx + al(S.nfb);
  const size_t tab = (size_t)2 * S.nfb * 64 * 8;
  cudaStream_t side = nullptr;
  if (mse_out) {
    side = (cudaStream_t)pf_internal_fork(S.ctx);
    if (!side || cudaMemcpyAsync(ptab, S.a.mse, tab, cudaMemcpyDeviceToHost, side) != cudaSuccess) return PF_ERR_DEVICE;
  }
  if (launch_select(S.s, S.maxCfg, (unsigned long long)params->lambda, S.idx, S.fo, st) != cudaSuccess)
    return PF_ERR_DEVICE;
  if (ev && cudaEventRecord(ev[4], st) != cudaSuccess) return PF_ERR_DEVICE;
  if (cudaMemcpyAsync(pfo, S.fo, sizeof(FinishOut), cudaMemcpyDeviceToHost, st) != cudaSuccess) return PF_ERR_DEVICE;
  if (fb_index_out && cudaMemcpyAsync(pidx, S.idx, S.nfb, cudaMemcpyDeviceToHost, st) != cudaSuccess)
    return PF_ERR_DEVICE;
  if (mse_out && !pf_internal_join(S.ctx)) return PF_ERR_DEVICE;
  // A context with a deadline waits once, for both streams.
  const bool early = mse_out && !pf_internal_bounded(S.ctx);
  if (early) {
    const int w = pf_internal_wait(S.ctx, side);
    if (w != PF_OK) return w;
    memcpy(mse_out, ptab, tab);
  }
  const int w = pf_internal_wait(S.ctx, st);
  if (w != PF_OK) return w;
  if (mse_out && !early) memcpy(mse_out, ptab, tab);
  FinishOut fo;
  memcpy(&fo, pfo, sizeof(fo));
  if (fb_index_out) memcpy(fb_index_out, pidx, S.nfb);
  if (result) {
    memset(result, 0, sizeof(*result));
    result->bits = (uint8_t)fo.bits;
    result->strength_count = (uint8_t)(1 << fo.bits);
    // Presets map back through the luma list, chroma's too (finish,
    // cdef_search.go:937-940).
    for (int j = 0; j < (1 << fo.bits); j++) {
      result->y_strength[j] = (uint8_t)S.a.trials.y[fo.ys[j]];
      result->uv_strength[j] = (uint8_t)S.a.trials.y[fo.uvs[j]];
    }
    result->cost = (double)fo.cost;
  }
  return PF_OK;
}

extern "C" int pf_cdef_search(pf_ctx* ctx, const pf_frame* source, const pf_frame* recon, const uint8_t* noskip,
                              const pf_cdef_search_params* params, uint64_t* mse_out, uint8_t* fb_index_out,
                              pf_cdef_search_result* result) {
  if (!ctx || !source || !recon || !params) return PF_ERR_INVALID_ARG;
  Staged S;
  const int stt = stage_search(ctx, source, recon, noskip, search_damping(params), search_max_cfg(params), 0, mse_out != nullptr, &S);
  if (stt != PF_OK) return stt;
  return search_finish(S, params, mse_out, fb_index_out, result);
}

extern "C" int pf_cdef_search_ex(pf_ctx* ctx, const pf_frame* source, const pf_frame* recon, const uint8_t* noskip,
                                 const pf_cdef_search_params* params, const pf_cdef_search_ctrls* ctrls,
                                 uint64_t* mse_out, uint8_t* fb_index_out, pf_cdef_search_result* result) {
  if (!ctx || !source || !recon || !params || !ctrls) return PF_ERR_INVALID_ARG;
  if (ctrls->count < 1 || ctrls->count > PF_CDEF_MAX_TRIALS || ctrls->subsampling < 1) return PF_ERR_INVALID_ARG;
  TrialList t;
  memset(&t, 0, sizeof(t));
  for (int g = 0; g < ctrls->count; g++) {
    if (ctrls->y[g] < 0 || ctrls->y[g] > 63 || ctrls->uv[g] < -1 || ctrls->uv[g] > 63) return PF_ERR_INVALID_CDEF;
    t.y[g] = ctrls->y[g];
    t.uv[g] = ctrls->uv[g];
    if (ctrls->uv[g] >= 0) t.uvMask |= 1ull << g;
  }
  t.count = ctrls->count;
  t.ss = ctrls->subsampling < 4 ? ctrls->subsampling : 4;  // BLOCK_8X8 caps the luma step (searchRow, :694-699)
  Staged S;
  const int stt = stage_search(ctx, source, recon, noskip, search_damping(params), search_max_cfg(params), 0, mse_out != nullptr, &S);
  if (stt != PF_OK) return stt;
  S.a.trials = t;
  S.s.uvFromY = ctrls->uv_from_y ? 1 : 0;
  return search_finish(S, params, mse_out, fb_index_out, result);
}

// ---------------------------------------------------------------------------
// Search controls per level and the picture plan (host logic).

extern "C" int pf_cdef_search_level_rtc(int32_t islice, int32_t screen) {
  // svtRTCCDEFSearchLevel (cdef_search.go:208-221).
  if (islice) return 5;
  return screen ? 7 : 8;
}

namespace {
// One level's controls: first- and second-pass luma and chroma lists and the
// flags updateOnRefInfo and the plan read (svtCDEFSearchCtrls,
// cdef_search.go:55-70, filled as setSVTCDEFSearchControls does, :72-202).
struct LevelCtrls {
  bool enabled = false, useRef = false, bestRef = false, skipDetector = false, uvFromY = false;
  int first = 0, second = 0, ss = 1;
  int8_t fs1[64] = {}, fs2[64] = {}, uv1[64] = {}, uv2[64] = {};
  int predY = 0;
};

// The first-pass primaries of levels 1-8 (indices into svtPfGI, p * 4).
const int8_t* level_primaries(int level, int* n) {
  static const int8_t l1[16] = {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15};
  static const int8_t l2[12] = {0, 1, 2, 4, 5, 6, 8, 9, 10, 12, 13, 14};
  static const int8_t l3[5] = {0, 4, 8, 12, 15};
  static const int8_t l45[3] = {0, 7, 15};
  static const int8_t l678[2] = {0, 15};
  switch (level) {
    case 1: *n = 16; return l1;
    case 2: *n = 12; return l2;
    case 3: *n = 5; return l3;
    case 4:
    case 5: *n = 3; return l45;
    default: *n = 2; return l678;
  }
}

LevelCtrls level_ctrls(int level, bool isBase, bool notHighest) {
  LevelCtrls c;
  c.enabled = true;
  int n;
  const int8_t* pri = level_primaries(level, &n);
  c.first = n;
  for (int i = 0; i < n; i++) c.fs1[i] = c.uv1[i] = (int8_t)(4 * pri[i]);
  if (level <= 4) {
    // Second pass: each first-pass strength's three secondaries.
    c.second = 3 * n;
    for (int i = 0; i < n; i++)
      for (int j = 1; j < 4; j++) c.fs2[3 * i + j - 1] = (int8_t)(c.fs1[i] + j);
    for (int i = 0; i < c.second; i++) c.uv2[i] = level == 1 ? c.fs2[i] : (int8_t)-1;
    return c;
  }
  // Levels 5-8: secondary 2 of each first-pass strength, chroma untested there.
  c.second = n;
  for (int i = 0; i < n; i++) {
    c.fs2[i] = (int8_t)(c.fs1[i] + 2);
    c.uv2[i] = -1;
  }
  if (level == 5) {
    c.bestRef = !notHighest;
    return c;
  }
  if (level == 8) c.uv1[0] = c.uv1[1] = -1;
  c.uv1[2] = -1;
  c.ss = 4;
  if (level == 6) c.bestRef = !notHighest;
  if (level == 7) {
    c.useRef = !notHighest;
    c.bestRef = !isBase;
    c.skipDetector = !isBase;
  }
  if (level == 8) {
    c.useRef = !isBase;
    c.bestRef = !isBase;
    c.uvFromY = true;
    for (int i = 0; i < c.first; i++) c.uv1[i] = -1;
    for (int i = 0; i < c.second; i++) c.uv2[i] = -1;
  }
  return c;
}

// updateOnRefInfo (cdef_search.go:237-272): false when CDEF turns off.
bool on_ref_info(LevelCtrls& c, const pf_cdef_ref_strengths& ref) {
  if (c.useRef) {
    int lo = 63, hi = 0;
    for (int i = 0; i < ref.count; i++) {
      lo = ref.y[i] < lo ? ref.y[i] : lo;
      hi = ref.y[i] > hi ? ref.y[i] : hi;
    }
    c.predY = (lo + hi) / 2 < 63 ? (lo + hi) / 2 : 63;
    c.first = c.second = 0;
    return c.predY != 0;
  }
  if (c.bestRef) {
    c.first = 1;
    c.second = 0;
    if ((int8_t)ref.y[0] != c.fs1[0]) c.fs1[c.first++] = (int8_t)ref.y[0];
    if ((int8_t)ref.uv[0] == c.uv1[0]) c.uv1[0] = c.uv1[1] = -1;
    return c.first != 1;
  }
  return true;
}
}  // namespace

extern "C" int pf_cdef_plan_picture(int32_t level, int32_t islice, int32_t is_base, int32_t not_highest_layer,
                                    const pf_cdef_ref_strengths* ref, int32_t ref_skip_percent, pf_cdef_plan* plan) {
  if (!plan) return PF_ERR_INVALID_ARG;
  if (level == 9) return PF_ERR_UNSUPPORTED;
  if (level < 0 || level > 9) return PF_ERR_INVALID_ARG;
  memset(plan, 0, sizeof(*plan));
  if (level == 0) return PF_OK;
  LevelCtrls c = level_ctrls(level, is_base != 0, not_highest_layer != 0);
  bool on = c.enabled;
  // planSVTCDEF (cdef_frame.go:34-54): on inter pictures, the skip detector,
  // else the reference's strengths.
  if (!islice) {
    if (ref_skip_percent > 75 && c.skipDetector) {
      on = false;
    } else if (c.useRef || c.bestRef) {
      if (!ref || ref->count < 1 || ref->count > 8) return PF_ERR_INVALID_ARG;
      on = on_ref_info(c, *ref);
    }
  }
  plan->on = on;
  plan->search = on && !c.useRef;
  if (on && c.useRef) plan->y_strength = (uint8_t)c.predY;  // predUVF is 0
  pf_cdef_search_ctrls& t = plan->ctrls;
  t.count = c.first + c.second;
  for (int g = 0; g < t.count; g++) {
    t.y[g] = g < c.first ? c.fs1[g] : c.fs2[g - c.first];
    t.uv[g] = g < c.first ? c.uv1[g] : c.uv2[g - c.first];
  }
  t.subsampling = c.ss;
  t.uv_from_y = c.uvFromY;
  return PF_OK;
}

// Host or device bytes into a host vector.
static bool read_small(const uint8_t* p, size_t n, std::vector<uint8_t>* out) {
  out->resize(n);
  cudaPointerAttributes at;
  const bool dev = cudaPointerGetAttributes(&at, p) == cudaSuccess &&
                   (at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged);
  cudaGetLastError();
  if (!dev) {
    memcpy(out->data(), p, n);
    return true;
  }
  return cudaMemcpy(out->data(), p, n, cudaMemcpyDeviceToHost) == cudaSuccess;
}

extern "C" int pf_cdef_apply(pf_ctx* ctx, const pf_frame* recon, const uint8_t* noskip,
                             const pf_cdef_search_params* params, const pf_cdef_search_result* result,
                             const uint8_t* fb_index) {
  if (!ctx || !recon || !params || !result) return PF_ERR_INVALID_ARG;
  const int stt = check_search_frame(recon, recon);
  if (stt != PF_OK) return stt;
  if (result->bits > 3) return PF_ERR_INVALID_CDEF;
  const int count = 1 << result->bits;
  // cdef_apply.go:262-271: nothing to do when every strength is zero.
  bool zero = true;
  for (int i = 0; i < count; i++)
    if (result->y_strength[i] || result->uv_strength[i]) zero = false;
  if (zero) return PF_OK;
  const int ucols = (recon->width + 63) / 64, urows = (recon->height + 63) / 64, n = ucols * urows;
  std::vector<uint8_t> ns, idx, read(n, 1), index(n, 0);
  if (noskip && !read_small(noskip, (size_t)n * 8, &ns)) return PF_ERR_DEVICE;
  if (fb_index && !read_small(fb_index, n, &idx)) return PF_ERR_DEVICE;
  // cdef_apply.go:202-235 (markFromLoopFilterMap, noskip-grid branch): a
  // unit is coded, with its searched index, when an in-frame 8x8 block of it
  // carries residual.
  const int cols8 = (recon->width + 7) >> 3, rows8 = (recon->height + 7) >> 3;
  for (int uy = 0; uy < urows; uy++)
    for (int ux = 0; ux < ucols; ux++) {
      const int u = uy * ucols + ux;
      if (noskip) {
        uint64_t inFrame = 0, word = 0;
        for (int by = 0; by < 8 && uy * 8 + by < rows8; by++)
          for (int bx = 0; bx < 8 && ux * 8 + bx < cols8; bx++) inFrame |= 1ull << (by * 8 + bx);
        for (int b = 0; b < 8; b++) word |= (uint64_t)ns[(size_t)u * 8 + b] << (8 * b);
        read[u] = (word & inFrame) != 0;
      }
      index[u] = read[u] && fb_index ? idx[u] : 0;
    }
  pf_frame_side side;
  memset(&side, 0, sizeof(side));
  side.stages = PF_STAGE_CDEF;
  side.side_memory = PF_MEM_HOST;
  pf_cdef& c = side.cdef;
  c.damping = (uint8_t)search_damping(params);
  c.bits = result->bits;
  c.strength_count = (uint8_t)count;
  memcpy(c.y_strength, result->y_strength, 8);
  memcpy(c.uv_strength, result->uv_strength, 8);
  c.index = index.data();
  c.read = read.data();
  c.index_stride = ucols;
  c.index_rows = urows;
  c.noskip = noskip ? ns.data() : nullptr;
  const int r = pf_frame_apply(ctx, recon, &side, nullptr, nullptr);
  if (r != PF_OK) return r;
  return pf_sync(ctx);
}

extern "C" int pf_cdef_features(pf_ctx* ctx, const pf_frame* recon, const uint8_t* noskip, int32_t qindex,
                                int32_t damping, float* features) {
  if (!ctx || !recon || !features) return PF_ERR_INVALID_ARG;
  if (qindex < 0 || qindex > 255) return PF_ERR_INVALID_ARG;
  const int dmp = damping ? damping : 3 + (qindex >> 6);
  Staged S;
  const int miCols = ((recon->width + 7) >> 3) << 1, miRows = ((recon->height + 7) >> 3) << 1;
  const int nfb = ((miCols + 15) / 16) * ((miRows + 15) / 16);
  const size_t xBytes = (size_t)nfb * PF_MLP_FEATURES * sizeof(float);
  const int stt = stage_search(ctx, nullptr, recon, noskip, dmp, 0, xBytes, false, &S);
  if (stt != PF_OK) return stt;
  float* X = (float*)S.extra;
  if (launch_features(S.a, qindex, X, true, S.st) != cudaSuccess) return PF_ERR_DEVICE;
  if (cudaMemcpyAsync(features, X, xBytes, cudaMemcpyDeviceToHost, S.st) != cudaSuccess) return PF_ERR_DEVICE;
  return pf_internal_wait(ctx, S.st);
}

extern "C" int pf_cdef_search_learned(pf_ctx* ctx, const pf_frame* source, const pf_frame* recon,
                                      const uint8_t* noskip, const pf_cdef_search_params* params,
                                      const pf_cdef_mlp* model, float threshold, int32_t candidates,
                                      int32_t flags, uint64_t* mse_out, uint8_t* fb_index_out,
                                      pf_cdef_search_result* result, pf_cdef_learned_stats* stats) {
  if (!ctx || !source || !recon || !params || !model) return PF_ERR_INVALID_ARG;
  if (flags & ~PF_LEARNED_REFINE) return PF_ERR_INVALID_ARG;
  if (candidates < 1 || candidates > 8 || !(threshold >= 0.f)) return PF_ERR_INVALID_ARG;
  if (params->qindex < 0 || params->qindex > 255) return PF_ERR_INVALID_ARG;
  const int miCols = ((recon->width + 7) >> 3) << 1, miRows = ((recon->height + 7) >> 3) << 1;
  const int nfb = ((miCols + 15) / 16) * ((miRows + 15) / 16);
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t xBytes = al((size_t)nfb * PF_MLP_FEATURES * sizeof(float));
  const size_t mBytes = al((size_t)nfb * 2 * sizeof(uint64_t));
  const size_t dBytes = al((size_t)nfb * 128);
  Staged S;
  const int stt = stage_search(ctx, source, recon, noskip, search_damping(params), search_max_cfg(params),
                               xBytes + mBytes + dBytes, mse_out != nullptr, &S);
  if (stt != PF_OK) return stt;
  float* X = (float*)S.extra;
  uint64_t* masks = (uint64_t*)(S.extra + xBytes);
  int changed = 0;
  uint8_t* mbase = (uint8_t*)pf_internal_cached_upload(ctx, model, sizeof(pf_cdef_mlp), mlp_expanded_bytes(), S.st,
                                                       &changed);
  if (!mbase) return PF_ERR_DEVICE;
  const pf_cdef_mlp* dmodel = (const pf_cdef_mlp*)mbase;
  float* W = (float*)(mbase + ((sizeof(pf_cdef_mlp) + 255) & ~(size_t)255));
  S.a.dirs = S.extra + xBytes + mBytes;
  S.a.ais = (int8_t*)(S.extra + xBytes + mBytes + (size_t)nfb * 64);
  // With stage timing on: events around features, network, trial search
  // and selection (read into stats->stage_ms).
  cudaEvent_t* ev = stats ? pf_internal_events(ctx) : nullptr;
  if (ev && cudaEventRecord(ev[0], S.st) != cudaSuccess) return PF_ERR_DEVICE;
  if (launch_features(S.a, params->qindex, X, false, S.st) != cudaSuccess) return PF_ERR_DEVICE;
  if (ev && cudaEventRecord(ev[1], S.st) != cudaSuccess) return PF_ERR_DEVICE;
  if (launch_mlp_masks(dmodel, W, changed != 0, X, nfb, threshold, candidates, masks, S.st) != cudaSuccess)
    return PF_ERR_DEVICE;
  if (ev && cudaEventRecord(ev[2], S.st) != cudaSuccess) return PF_ERR_DEVICE;
  S.a.tmask = masks;
  S.s.refine = (flags & PF_LEARNED_REFINE) ? 1 : 0;
  const int r = search_finish(S, params, mse_out, fb_index_out, result, ev);
  if (r != PF_OK) return r;
  // The statistics are read back after the search (no host wait between the
  // network and the search it steers).
  if (stats) {
    std::vector<uint64_t> hm((size_t)nfb * 2);
    std::vector<uint8_t> skip(nfb);
    if (cudaMemcpy(hm.data(), masks, (size_t)nfb * 16, cudaMemcpyDeviceToHost) != cudaSuccess ||
        cudaMemcpy(skip.data(), S.a.skip, nfb, cudaMemcpyDeviceToHost) != cudaSuccess)
      return PF_ERR_DEVICE;
    memset(stats, 0, sizeof(*stats));
    for (int i = 0; i < 4; i++) {
      float ms = -1.f;
      if (ev && cudaEventElapsedTime(&ms, ev[i], ev[i + 1]) != cudaSuccess) {
        ms = -1.f;
        (void)cudaGetLastError();
      }
      stats->stage_ms[i] = ev ? ms : -1.f;
    }
    for (int fb = 0; fb < nfb; fb++) {
      if (skip[fb]) continue;
      stats->blocks++;
      const int c0 = __builtin_popcountll(hm[2 * fb]), c1 = __builtin_popcountll(hm[2 * fb + 1]);
      if (c0 == 64) stats->fallback_luma++;
      if (c1 == 64) stats->fallback_chroma++;
      stats->trials_luma += c0;
      stats->trials_chroma += c1;
    }
  }
  return PF_OK;
}
