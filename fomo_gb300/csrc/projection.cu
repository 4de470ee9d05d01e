// Projection render (fomo-c/src/fomo-projection.cpp:17-193): every data point
// adds its emission to the image pixel nearest its projection -- no line of
// sight is marched.  Per view: j = round((x' - minx)(nx - 1) / (maxx - minx)),
// i = round((y' - miny)(ny - 1) / (maxy - miny)) with x', y' the point rotated
// in FP64 exactly as for the extents (nn:83-85, the same operand order, so the
// pixel of every point is the reference's); a spectroscopic point adds
// eps * 2^(-(2 (lambda - shift) / w)^2) (= eps exp(-4 ln2 (dl / w)^2), :134)
// to the lambda bins of its pixel, an imaging point adds eps.  The view's
// path-length (and DN pixel-area) scale of :161-191 is applied to each
// contribution.  Contributions of points that share a pixel are summed with
// FP32 atomics, so the order of the sum -- like the reference's `omp atomic`
// -- is not fixed.
//
// Spectroscopy of many points goes by pixel: each point's pixel is found and
// counted, the points are listed by pixel (a counting sort of their positions), and
// one warp per pixel sums its points' profiles in registers and writes its spectrum
// once (SpectralBins).  The direct kernel below adds every point's bins to the cube
// with atomics, 268 million of them for 2M points x 4 lines x 32 bins at 256 x 256
// pixels: the render took 969 us, 845 with the pixels from FP32 (pixel_of), and
// takes 276 by pixel.  kProjListed, points x lines x windows: the direct kernel
// against the list at 0.11M points, 1 line 86 / 106 us, 4 lines of 2 windows 137 /
// 112 (96 x 96), 147 / 148 (256 x 256); 0.5M points, 1 line of 2 windows 146 / 146,
// 4 lines 307 / 183; 2M points, 1 line 322 / 204.  A warp per pixel also has to be
// worth it: by pixel from 4 points a pixel on for one line, 3 for more.  2M points
// at 0.5, 1, 2, 3, 6 points a pixel, the direct kernel / the list: 1 line of 64 bins
// 490 / 1069, 424 / 662, 392 / 426, 380 / 343, 366 / 254; 4 lines of 64 bins 1565 /
// 2877, 1303 / 1672, 1176 / 984, 1139 / 741, 1102 / 488; 0.5M points, 4 lines of 128
// bins 804 / 1782, 662 / 1056, 577 / 640, 552 / 489, 533 / 339.  Imaging adds one
// float per point and line and keeps the direct kernel.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "fomo_device.cuh"
#include "fomo_internal.h"
#include "spectral_bins.cuh"

namespace fomo {

namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kProjThreads = 256;
constexpr int64_t kProjListed = 900000;  // points x lines x windows from which a projection goes by pixel

// The pixel of point q (x, y, z): std::round, halves away from zero (:124, :126).
// x', y' lie within the extents, so it is in the image; a degenerate extent (max ==
// min) gives NaN in the reference: see the range check of the callers.
__device__ __noinline__ int2 pixel_f64(const ViewDesc* V, float4 q) {
  const double cb = V->rcb, sb = V->rsb, cl = V->cl, sl = V->sl;
  const double minx = V->minx, miny = V->miny;
  const double dxr = __dsub_rn(V->maxx, minx), dyr = __dsub_rn(V->maxy, miny);
  const double gx = q.x, gy = q.y, gz = q.z;
  const double xa = __dsub_rn(__dsub_rn(__dmul_rn(__dmul_rn(gx, cb), cl), __dmul_rn(__dmul_rn(gy, cb), sl)),
                              __dmul_rn(gz, sb));
  const double ya = __dadd_rn(__dmul_rn(gx, sl), __dmul_rn(gy, cl));
  return make_int2((int)round(__ddiv_rn(__dmul_rn(__dsub_rn(xa, minx), (double)(V->nx - 1)), dxr)),
                   (int)round(__ddiv_rn(__dmul_rn(__dsub_rn(ya, miny), (double)(V->ny - 1)), dyr)));
}

// What pixel_of takes from a view: the rotation's rows and the scales in FP32.
struct PixelMap {
  float ax, ay, az, bx, by, minx, miny, kx, ky;
  __device__ __forceinline__ explicit PixelMap(const ViewDesc* V) {
    ax = (float)(V->rcb * V->cl);
    ay = (float)(-V->rcb * V->sl);
    az = (float)-V->rsb;
    bx = (float)V->sl;
    by = (float)V->cl;
    minx = (float)V->minx;
    miny = (float)V->miny;
    kx = (float)((double)(V->nx - 1) / (V->maxx - V->minx));
    ky = (float)((double)(V->ny - 1) / (V->maxy - V->miny));
  }
};

// The pixel of a point, from FP32 where that is far enough from a pixel's border.  FP32
// (with FMAs) errs by at most 5 roundings of the products' sum in x' and of the
// extent's end, scaled to pixels, and 4 of the pixel coordinate itself; 8 are
// allowed for each.  Two in a thousand points take FP64 (1/64 of the FP32 rate).
__device__ __forceinline__ int2 pixel_of(const ViewDesc* V, const PixelMap& M, float4 q) {
  constexpr float ulps = 8.0f * 5.97e-8f;
  const float jx = (fmaf(q.x, M.ax, fmaf(q.y, M.ay, q.z * M.az)) - M.minx) * M.kx + 0.5f;
  const float iy = (fmaf(q.x, M.bx, q.y * M.by) - M.miny) * M.ky + 0.5f;
  const float mag = fabsf(q.x) + fabsf(q.y) + fabsf(q.z);
  const float Ex = ((mag + fabsf(M.minx)) * M.kx + fabsf(jx) + 1.0f) * ulps;
  const float Ey = ((mag + fabsf(M.miny)) * M.ky + fabsf(iy) + 1.0f) * ulps;
  const bool ok = fabsf(jx - rintf(jx)) > Ex && fabsf(iy - rintf(iy)) > Ey && fabsf(jx) < 1e9f && fabsf(iy) < 1e9f;
  if (!ok) return pixel_f64(V, q);
  return make_int2((int)floorf(jx), (int)floorf(iy));
}

__global__ void __launch_bounds__(kProjThreads) projection_kernel(SnapDev snap, const ViewDesc* __restrict__ views,
                                                                  const LineDesc* __restrict__ lines, int nlines,
                                                                  int imaging) {
  const ViewDesc* V = views + blockIdx.y;
  const LineDesc* LD = lines + (int64_t)blockIdx.y * nlines;
  const int nx = V->nx, ny = V->ny, L = V->L;
  const PixelMap map(V);
  const float ux = V->ux, uy = V->uy, uz = V->uz;
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (kProjThreads / 32);
  for (int64_t base = ((int64_t)blockIdx.x * (kProjThreads / 32) + (threadIdx.x >> 5)) * 32; base < snap.n;
       base += warps * 32) {
    const int64_t p = base + lane;
    int pix = -1;
    float vlos = 0.0f;
    if (p < snap.n) {
      const float4 q = __ldg(snap.pts + p);
      const int2 at = pixel_of(V, map, q);
      // a degenerate extent's points may fall outside: they are dropped
      if (at.x >= 0 && at.x < nx && at.y >= 0 && at.y < ny) pix = at.y * nx + at.x;
      if (!imaging) {
        const float4 vv = __ldg(snap.vel + p);
        vlos = fmaf(uz, vv.z, fmaf(uy, vv.y, ux * vv.x));
      }
    }
    if (imaging) {
      for (int l = 0; l < nlines; ++l) {
        const LineDesc& D = LD[l];
        if (!D.ew || pix < 0) continue;
        const float e = __ldg(D.ew + p).x;
        if (e != 0.0f)
          atomicAdd(D.out + FOMO_IDX(pix, (int64_t)nx * ny, kSiteProjection), (float)(D.is_dn ? V->scale_dn : V->scale) * e);
      }
      continue;
    }
    for (int s = 0; s < 32; ++s) {
      const int ps = __shfl_sync(kFull, pix, s);
      const float vs = __shfl_sync(kFull, vlos, s);
      if (ps < 0) continue;  // the same for every lane
      for (int l = 0; l < nlines; ++l) {
        const LineDesc& D = LD[l];
        if (!D.ew) continue;  // views may have fewer lines than the launch
        const float2 pw = __ldg(D.ew + base + s);
        if (pw.x == 0.0f) continue;
        const float sc = __fdividef(2.0f, pw.y);
        const float ns = -(vs * D.shift_k) * sc;
        const float scale = (float)(D.is_dn ? V->scale_dn : V->scale);
        float* out = D.out + FOMO_IDX((int64_t)ps * L, (int64_t)nx * ny * L, kSiteProjection);
        for (int m = 0; m < D.nw; ++m) {
          const int il = D.wstart + 32 * m + lane;
          if (il < L) {
            const float qq = fmaf(__ldg(D.lam + FOMO_IDX(il, L, kSiteLam)), sc, ns);
            const float v = pw.x * ex2_approx(-qq * qq);
            if (v != 0.0f) atomicAdd(out + il, v * scale);
          }
        }
      }
    }
  }
}

// ---- by pixel
constexpr int kBinThreads = 128;
constexpr int kBinWarps = kBinThreads / 32;
constexpr int kPixelWhole = 512;   // points of a pixel one warp sums; a pixel with more is summed in pieces of these

// Points per pixel below which the spectra are scaled by FP32 pairs: with more, FP64 hides behind the profiles (0.5M points, 4
// lines x 128 bins: 12 points a pixel 267 pairs / 308 us FP64, 24 231 / 232, 48 220 / 209).
constexpr int64_t kPairsBelow = 24;

// Each point's pixel and its place among the pixel's points.
__global__ void __launch_bounds__(kProjThreads)
    proj_count_kernel(SnapDev snap, const ViewDesc* __restrict__ V, int* __restrict__ count, int2* __restrict__ at) {
  const PixelMap map(V);
  const int nx = V->nx, ny = V->ny;
  const int lane = threadIdx.x & 31;
  for (int64_t p0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; p0 < snap.n;
       p0 += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = p0 + lane;
    int pix = -1;
    if (p < snap.n) {
      const int2 a = pixel_of(V, map, __ldg(snap.pts + p));
      if (a.x >= 0 && a.x < nx && a.y >= 0 && a.y < ny) pix = a.y * nx + a.x;
    }
    // one atomic for the warp's points of a pixel (neighbours in the cell order often share
    // one, and a dense cloud seen along its axis puts most of its points in a few pixels)
    const unsigned same = __match_any_sync(kFull, pix);
    const int head = __ffs(same) - 1;
    int base = 0;
    if (lane == head && pix >= 0)
      base = atomicAdd(count + FOMO_IDX(pix, (int64_t)nx * ny, kSiteProjection), __popc(same));
    base = __shfl_sync(kFull, base, head);
    if (p < snap.n) at[p] = make_int2(pix, base + __popc(same & ((1u << lane) - 1u)));
  }
}

__global__ void __launch_bounds__(kProjThreads)
    proj_list_kernel(int64_t n, const int2* __restrict__ at, const int* __restrict__ first, int* __restrict__ list) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n; p += (int64_t)gridDim.x * blockDim.x) {
    const int2 a = at[p];
    if (a.x >= 0) list[FOMO_IDX(first[a.x] + a.y, n, kSiteProjection)] = (int)p;
  }
}

// One warp per pixel, taken from a queue; a pixel of more than kPixelWhole points is
// cleared, and its pieces are queued for the second launch (PIECES), which adds them
// with atomics.
template <int NL, int NB, bool PIECES, bool PAIRS>
__global__ void __launch_bounds__(kBinThreads, 8)
    proj_bin_kernel(SnapDev snap, const ViewDesc* __restrict__ V, const LineDesc* __restrict__ LD, int nlines,
                    const int* __restrict__ first, const int* __restrict__ list, int2* __restrict__ pieces,
                    int pieces_cap, unsigned long long* __restrict__ ctr) {
  __shared__ BinShared<NL, NB> staged[kBinWarps];
  BinShared<NL, NB>& sh = staged[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int npix = V->nx * V->ny;
  const int nqueue = PIECES ? min((int)ctr[kCtrHard], pieces_cap) : npix;
  // pixels per atomic: up to four where each warp of the grid gets several
  const int grab = PIECES ? 1 : max(1, min(4, npix / ((int)gridDim.x * kBinWarps * 4)));
  SpectralBins<NL, NB, PAIRS> bins;
  bins.view(V, LD, nlines, sh);
  for (;;) {
    int q0 = 0;
    if (lane == 0) q0 = (int)atomicAdd(ctr + (PIECES ? kCtrHardHead : kCtrRays), (unsigned long long)grab);
    q0 = __shfl_sync(kFull, q0, 0);
    if (q0 >= nqueue) return;
    for (int q = q0; q < min(q0 + grab, nqueue); ++q) {
      const int2 piece = PIECES ? pieces[FOMO_IDX(q, pieces_cap, kSiteHard)] : make_int2(q, 0);
      const int pix = piece.x;
      int b = first[pix], e = first[pix + 1];
      if (PIECES) {
        b += piece.y * kPixelWhole;
        e = min(e, b + kPixelWhole);
      } else if (e - b > kPixelWhole) {
        const int np = (e - b + kPixelWhole - 1) / kPixelWhole;
        int at = 0;
        if (lane == 0) at = (int)atomicAdd(ctr + kCtrHard, (unsigned long long)np);
        at = __shfl_sync(kFull, at, 0);
        for (int i = lane; i < np; i += 32) pieces[FOMO_IDX(at + i, pieces_cap, kSiteHard)] = make_int2(pix, i);
        e = b;  // only cleared here
      }
      bins.clear();
      for (int i = b; i < e; i += 32) {
        const int m = min(32, e - i);
        bins.add(snap, V, sh, m, lane < m ? __ldg(list + FOMO_IDX(i + lane, snap.n, kSiteProjection)) : -1, 1, nullptr);
      }
      bins.template write<PIECES>(V, LD, sh, pix);
    }
  }
}

template <int NL, int NB>
cudaError_t launch_bins(const ProjScratch& P, SnapDev snap, const ViewDesc* V, const LineDesc* LD, int nlines,
                        int64_t npix, int sm_count, cudaStream_t s) {
  const int cap = sm_count * 8;
  const int blocks = (int)std::min<int64_t>(cap, (npix + kBinWarps - 1) / kBinWarps);
  const auto kernel = snap.n < kPairsBelow * npix ? proj_bin_kernel<NL, NB, false, true> : proj_bin_kernel<NL, NB, false, false>;
  kernel<<<blocks, kBinThreads, 0, s>>>(snap, V, LD, nlines, P.first, P.list, P.pieces, P.pieces_cap, P.ctr);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && snap.n > kPixelWhole) {
    const int64_t most = snap.n / kPixelWhole * 2;
    proj_bin_kernel<NL, NB, true, false><<<(int)std::min<int64_t>(cap, (most + kBinWarps - 1) / kBinWarps), kBinThreads, 0, s>>>(
        snap, V, LD, nlines, P.first, P.list, P.pieces, P.pieces_cap, P.ctr);
    e = cudaGetLastError();
  }
  return e;
}

}  // namespace

FOMO_DEFINE_CHECK_READER(check_word_projection)

bool projection_by_pixel(int64_t n, int64_t npix, int nlines, int max_windows, bool imaging) {
  if (imaging || n * nlines * max_windows < kProjListed || n < (nlines == 1 ? 4 : 3) * npix) return false;
  return max_windows <= (nlines <= 1 ? 8 : 4) && nlines <= 4;
}

int projection_pieces(int64_t n) { return (int)(2 * (n / kPixelWhole) + 1); }

cudaError_t launch_projection_view(const ProjScratch& P, SnapDev snap, const ViewDesc* V, const LineDesc* LD, int nlines,
                                   int max_windows, int64_t npix, int sm_count, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(P.ctr, 0, sizeof(unsigned long long) * kCtrCount, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(P.count, 0, sizeof(int) * (size_t)(npix + 1), s);
  if (e != cudaSuccess) return e;
  const int blocks = (int)std::min<int64_t>((snap.n + kProjThreads - 1) / kProjThreads, (int64_t)sm_count * 8);
  proj_count_kernel<<<blocks, kProjThreads, 0, s>>>(snap, V, P.count, P.at);
  e = cudaGetLastError();
  if (e == cudaSuccess)
    e = launch_exclusive_scan(P.count, P.first, npix + 1, P.scan, exclusive_scan_scratch_ints(npix + 1), s);
  if (e != cudaSuccess) return e;
  proj_list_kernel<<<blocks, kProjThreads, 0, s>>>(snap.n, P.at, P.first, P.list);
  e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const int nb = max_windows;
#define FOMO_BINS(NL_, NB_) \
  if (nlines <= NL_ && nb <= NB_) return launch_bins<NL_, NB_>(P, snap, V, LD, nlines, npix, sm_count, s)
  FOMO_BINS(1, 1);
  FOMO_BINS(1, 2);
  FOMO_BINS(1, 8);
  FOMO_BINS(2, 1);
  FOMO_BINS(2, 4);
  FOMO_BINS(4, 1);
  FOMO_BINS(4, 2);
  FOMO_BINS(4, 4);
#undef FOMO_BINS
  return cudaErrorInvalidValue;
}

cudaError_t launch_projection(SnapDev snap, const ViewDesc* views, const LineDesc* lines, int nviews, int nlines,
                              bool imaging, int sm_count, cudaStream_t s) {
  if (nviews <= 0 || snap.n <= 0) return cudaSuccess;
  if (nviews > 65535) return cudaErrorInvalidValue;
  const int64_t warps_needed = (snap.n + 31) / 32;
  int64_t blocks = ((warps_needed + kProjThreads / 32 - 1) / (kProjThreads / 32));
  const int64_t cap = (int64_t)sm_count * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  projection_kernel<<<dim3((unsigned)blocks, (unsigned)nviews), kProjThreads, 0, s>>>(snap, views, lines, nlines,
                                                                                     imaging ? 1 : 0);
  return cudaGetLastError();
}

}  // namespace fomo
