// pf_superres.cu - AV1 super-resolution upscaling on the GPU.
//
// superres.UpscalePlaneCoded (internal/av1/superres/superres.go:40-107) as
// the decoder runs it between CDEF and loop restoration
// (internal/av1/decoder/postfilter_superres.go:206-283): each plane's coded
// samples, read over the MI-aligned span (the columns past the crop are the
// genuine coded samples, not a clamp of the last cropped column), are
// resampled to the upscaled width with the normative 8-tap, 64-phase filter;
// the step and initial phase come from the cropped coded width
// (av1_get_upscale_convolve_step / get_upscale_convolve_x0 as restated there).
// The restoration stripe-boundary rows of a super-resolved frame
// (tile/restoration_boundary.go:257-406, SaveRestorationBoundaryLinesFromFramePlaneSuperRes)
// are the same resampling of the deblocked coded rows b-2 .. b+1 around each
// stripe boundary b, into the rows the restoration kernel reads (k*4 + j for
// boundary k; when row b+1 is past the plane, row b stands in for it, as
// finishRestorationBoundaryLines does).
//
// A CTA makes 256 output columns of up to 8 rows: the rows' source samples
// are staged in shared memory as floats (their edge already clamped), and a
// thread reads its column's eight taps once for all rows.  Samples times taps
// add up to at most 65535 * 216 < 2^24, so fp32 holds every sum exactly; its
// multiply-adds run at twice the rate of 32-bit integer ones.  Bound by
// instruction issue (83 % of the slots at 59 warps per SM), the eight shared
// reads a sample among them.  Several frames go in one launch.  8 frames of
// 1920x1080 8-bit 4:2:0: 63 us, and 11 for the boundary rows; with a launch a
// frame, a row a CTA and the taps read anew for every sample 8 x 20 and 8 x 8.7.
#include <string.h>

#include "pf_common.cuh"
#include "pf_superres.cuh"
#include "pf_tables.h"

namespace pf {

constexpr int kSrScaleBits = 14, kSrExtraBits = kSrScaleBits - 6;
constexpr int kSrCols = 256, kSrRows = 8;
constexpr int kSrSpan = kSrCols + 8;  // source columns of a row: the step is below one column

// The filter as floats, filled by superres_upload_tables.
__device__ float g_sr_filter[64][8];

cudaError_t superres_upload_tables() {
  float f[64][8];
  for (int p = 0; p < 64; p++)
    for (int k = 0; k < 8; k++) f[p][k] = (float)pf_superres_filter[p][k];
  return cudaMemcpyToSymbol(g_sr_filter, f, sizeof(f));
}

struct SrPlane {
  const uint8_t* src;
  uint8_t* dst;
  int64_t sstride, dstride;
  int srcWidth, dstWidth, rows, step, x0;
  int cols, bands;  // column chunks; row bands (frames) or stripe boundaries (lines)
  int sh, off;      // stripe height and offset (lines)
};

constexpr int kSrFrames = 8;  // frames of one launch (their planes travel as kernel arguments)
struct SrArgs {
  SrPlane pl[kSrFrames][3];
  int base[kSrFrames * 3 + 1];  // prefix of the planes' CTAs
  uint8_t deep[kSrFrames], maxv_bits[kSrFrames];
  int lines;
};

template <typename T>
__device__ __forceinline__ void sr_tile(const SrPlane& q, bool lines, int cc, int band, int maxv, float* s_src) {
  const int tid = threadIdx.x;
  const int xa = cc * kSrCols;
  // superres.go:78-107 (upscaleRowPureGo): output x reads source columns
  // px - 3 .. px + 4.
  const int first = (-(1 << kSrScaleBits) + q.x0 + xa * q.step) >> kSrScaleBits;
  const int last = q.srcWidth - 1;
  // Row r's source row and destination, or no row.
  const int b = lines ? (band + 1) * q.sh - q.off : 0;
  const int nrows = lines ? 4 : kSrRows;
  auto src_row = [&](int r) { return lines ? b - 2 + r : band * kSrRows + r; };
  auto has = [&](int r) { return r < nrows && src_row(r) < q.rows && (!lines || b < q.rows); };
  // A warp stages a row.
  static_assert(kSrRows == 8, "a row for each of the 8 warps");
  const int wr = tid >> 5, lane = tid & 31;
  if (has(wr)) {
    const T* row = reinterpret_cast<const T*>(q.src + (int64_t)src_row(wr) * q.sstride);
    const int s0 = first - 3 + lane;
    float* d = s_src + wr * kSrSpan + lane;
    constexpr int kSteps = (kSrSpan + 31) / 32;
    const bool in = first - 3 >= 0 && first - 3 + 32 * kSteps - 1 <= last;
    int v[kSteps];
#pragma unroll
    for (int k = 0; k < kSteps; k++) v[k] = row[in ? s0 + 32 * k : iclip(s0 + 32 * k, 0, last)];
#pragma unroll
    for (int k = 0; k < kSteps; k++)
      if (32 * k + 31 < kSrSpan || lane + 32 * k < kSrSpan) d[32 * k] = (float)v[k];
  }
  __syncthreads();
  const int x = xa + tid;
  if (x >= q.dstWidth) return;
  const int srcX = -(1 << kSrScaleBits) + q.x0 + x * q.step;
  const int at = (srcX >> kSrScaleBits) - first;
  const float4* f = reinterpret_cast<const float4*>(g_sr_filter[(srcX & ((1 << kSrScaleBits) - 1)) >> kSrExtraBits]);
  const float4 t0 = __ldg(&f[0]), t1 = __ldg(&f[1]);
  uint8_t* d = q.dst + (int64_t)(lines ? (band + 1) * 4 : band * kSrRows) * q.dstride + (int64_t)x * (int)sizeof(T);
  const float* s = s_src + at;
#pragma unroll 4
  for (int r = 0; r < nrows; r++, s += kSrSpan, d += q.dstride) {
    if (!has(r)) break;  // rows end together
    float sum = s[0] * t0.x;
    sum = fmaf(s[1], t0.y, sum);
    sum = fmaf(s[2], t0.z, sum);
    sum = fmaf(s[3], t0.w, sum);
    sum = fmaf(s[4], t1.x, sum);
    sum = fmaf(s[5], t1.y, sum);
    sum = fmaf(s[6], t1.z, sum);
    sum = fmaf(s[7], t1.w, sum);
    const T v = (T)iclip((__float2int_rn(sum) + 64) >> 7, 0, maxv);
    *reinterpret_cast<T*>(d) = v;
    if (lines && r == 2 && b + 1 >= q.rows) *reinterpret_cast<T*>(d + q.dstride) = v;
  }
}

__global__ void __launch_bounds__(256) k_superres(const __grid_constant__ SrArgs a) {
  __shared__ float s_src[kSrRows * kSrSpan];
  int p = 0;
  while ((int)blockIdx.x >= a.base[p + 1]) p++;
  const int f = p / 3, i = blockIdx.x - a.base[p];
  const SrPlane& q = a.pl[f][p - 3 * f];
  const int band = i / q.cols, cc = i - band * q.cols;
  const int maxv = (1 << a.maxv_bits[f]) - 1;
  if (a.deep[f])
    sr_tile<uint16_t>(q, a.lines, cc, band, maxv, s_src);
  else
    sr_tile<uint8_t>(q, a.lines, cc, band, maxv, s_src);
}

// Step and initial phase of one plane (superres.go:45-51).
static void sr_phase(int coded, int dst, int* step, int* x0) {
  const int s = ((coded << kSrScaleBits) + dst / 2) / dst;
  const int err = dst * s - (coded << kSrScaleBits);
  int x = ((-((dst - coded) << (kSrScaleBits - 1))) + dst / 2) / dst;
  x += (1 << (kSrExtraBits - 1)) - err / 2;
  *step = s;
  *x0 = x & ((1 << kSrScaleBits) - 1);
}

cudaError_t launch_superres(const SrFrame* frames, int n, bool lines, cudaStream_t st) {
  for (int at = 0; at < n; at += kSrFrames) {
    SrArgs a;
    memset(&a, 0, sizeof(a));
    const int frames_here = imin(kSrFrames, n - at);
    a.lines = lines;
    int total = 0;
    for (int i = 0; i < kSrFrames; i++)
      for (int p = 0; p < 3; p++) {
        a.base[3 * i + p] = total;
        if (i >= frames_here) continue;
        const SrFrame& F = frames[at + i];
        const pf_frame* c = F.coded;
        a.deep[i] = c->bit_depth > 8;
        a.maxv_bits[i] = c->bit_depth;
        if (p >= (c->mono ? 1 : 3) || (lines && F.boundaries[p] <= 1)) continue;
        const int sx = p ? c->ss_x : 0, sy = p ? c->ss_y : 0;
        SrPlane& q = a.pl[i][p];
        q.src = F.src[p];
        q.sstride = F.sstride[p];
        q.dst = F.dst[p];
        q.dstride = F.dstride[p];
        q.srcWidth = ((c->width + 7) & ~7) >> sx;  // the MI-aligned span the decoder reads
        q.dstWidth = (F.up_width + sx) >> sx;
        q.rows = (c->height + sy) >> sy;
        sr_phase((c->width + sx) >> sx, q.dstWidth, &q.step, &q.x0);
        q.cols = (q.dstWidth + kSrCols - 1) / kSrCols;
        q.sh = 64 >> sy;
        q.off = 8 >> sy;
        // Boundary slot 0 is the frame's top, which has none.
        q.bands = lines ? F.boundaries[p] - 1 : (q.rows + kSrRows - 1) / kSrRows;
        total += q.cols * q.bands;
      }
    a.base[kSrFrames * 3] = total;
    if (total == 0) continue;
    k_superres<<<total, 256, 0, st>>>(a);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace pf

void* pf_internal_search_scratch(pf_ctx* c, size_t bytes);  // pf_api.cu
int pf_internal_wait(pf_ctx* c, void* stream);  // pf_api.cu: blocking or bounded by the context's deadline
void* pf_internal_stream(pf_ctx* c);

// pf_superres_upscale takes coded spans of at most this many samples (its
// frames are at most 16384 wide and a coded frame of a bitstream at most
// 8/9 of that).
constexpr int kSrMaxSpan = 14600;

extern "C" int pf_superres_upscale(pf_ctx* ctx, const pf_frame* coded, const pf_frame* upscaled) {
  using namespace pf;
  if (!ctx || !coded || !upscaled) return PF_ERR_INVALID_ARG;
  if (coded->memory > PF_MEM_DEVICE || coded->memory != upscaled->memory) return PF_ERR_INVALID_ARG;
  if (coded->bit_depth != 8 && coded->bit_depth != 10 && coded->bit_depth != 12) return PF_ERR_INVALID_FORMAT;
  if (coded->bit_depth != upscaled->bit_depth || coded->ss_x != upscaled->ss_x || coded->ss_y != upscaled->ss_y ||
      coded->mono != upscaled->mono || coded->height != upscaled->height || coded->width <= 0 ||
      coded->height <= 0 || upscaled->width <= coded->width || upscaled->width > 16384)
    return PF_ERR_INVALID_FORMAT;
  const int bps = coded->bit_depth > 8 ? 2 : 1;
  const int nplanes = coded->mono ? 1 : 3;
  int aw[3], dw[3], rows[3];
  size_t hostBytes = 0;
  for (int p = 0; p < nplanes; p++) {
    const int sx = p ? coded->ss_x : 0, sy = p ? coded->ss_y : 0;
    const int cw = (coded->width + sx) >> sx;
    aw[p] = ((coded->width + 7) & ~7) >> sx;  // the MI-aligned span the decoder reads
    dw[p] = (upscaled->width + sx) >> sx;
    rows[p] = (coded->height + sy) >> sy;
    const pf_plane &sp = coded->plane[p], &dp = upscaled->plane[p];
    if (!sp.data || !dp.data || sp.width != cw || sp.height != rows[p] || sp.alloc_width < aw[p] ||
        sp.alloc_height < rows[p] || sp.stride < (int64_t)sp.alloc_width * bps || dp.width != dw[p] ||
        dp.height != rows[p] || dp.alloc_width < dw[p] || dp.alloc_height < rows[p] ||
        dp.stride < (int64_t)dp.alloc_width * bps)
      return PF_ERR_SHORT_BUFFER;
    hostBytes += ((size_t)aw[p] * bps + 255) / 256 * 256 * rows[p] + ((size_t)dw[p] * bps + 255) / 256 * 256 * rows[p];
  }
  const bool host = coded->memory == PF_MEM_HOST;
  const cudaStream_t st = (cudaStream_t)pf_internal_stream(ctx);
  uint8_t* scratch = nullptr;
  if (host) {
    scratch = (uint8_t*)pf_internal_search_scratch(ctx, hostBytes + 256);
    if (!scratch) return PF_ERR_DEVICE;
  }
  SrFrame f;
  memset(&f, 0, sizeof(f));
  f.coded = coded;
  f.up_width = upscaled->width;
  size_t off = 0;
  cudaError_t e = cudaSuccess;
  for (int p = 0; p < nplanes; p++) {
    const pf_plane &sp = coded->plane[p], &dp = upscaled->plane[p];
    if (host) {
      const int64_t ss = ((int64_t)aw[p] * bps + 255) / 256 * 256, ds = ((int64_t)dw[p] * bps + 255) / 256 * 256;
      f.src[p] = scratch + off;
      f.sstride[p] = ss;
      off += (size_t)ss * rows[p];
      f.dst[p] = scratch + off;
      f.dstride[p] = ds;
      off += (size_t)ds * rows[p];
      if (e == cudaSuccess)
        e = cudaMemcpy2DAsync((void*)f.src[p], ss, sp.data, sp.stride, (size_t)aw[p] * bps, rows[p],
                              cudaMemcpyHostToDevice, st);
    } else {
      f.src[p] = (const uint8_t*)sp.data;
      f.sstride[p] = sp.stride;
      f.dst[p] = (uint8_t*)dp.data;
      f.dstride[p] = dp.stride;
    }
  }
  if (e != cudaSuccess) return PF_ERR_DEVICE;
  if (aw[0] > kSrMaxSpan) return PF_ERR_INVALID_FORMAT;
  e = launch_superres(&f, 1, false, st);
  if (host)
    for (int p = 0; p < nplanes && e == cudaSuccess; p++)
      e = cudaMemcpy2DAsync(upscaled->plane[p].data, upscaled->plane[p].stride, f.dst[p], f.dstride[p],
                            (size_t)dw[p] * bps, rows[p], cudaMemcpyDeviceToHost, st);
  if (e != cudaSuccess) return PF_ERR_DEVICE;
  return pf_internal_wait(ctx, st);
}
