// K3: per-view set-up, entirely on the device (no host round trip).
//
//  * the extents: Stage A of the reference (fomo-c/src/fomo-nearestneighbour.cpp:
//    76-108): the points rotated in FP64 with the reference's operand order,
//    min/max reduced through order-preserving 64-bit atomics (exact, order
//    independent).  An FP32 rotation with a proven error bound screens the points
//    first, block by block, so that only those near an extreme are rotated in
//    FP64 (view_bounds_kernel, view_extents_blocks_kernel).  For Thomson every
//    point takes the pole-blended rotation with clamped cos/sin and sin^2(chi)
//    (fomo-thomson.cpp:139-199; view_extents_kernel).
//  * view_finalize_kernel: maxdistance (nn:138 / thomson:249-260), delta z,
//    path length and DN pixel area (nn:235-267), and the per-LOS-sample FP64
//    table z_k*sin(b)*cos(l), z_k*sin(b)*sin(l), z_k*cos(b) that the march
//    adds to the per-ray terms -- the same roundings as the reference's
//    derotation expression (nn:162-165).
// Transcendentals (cos, sin, exp of the blends) are evaluated on the host with
// the host libm and passed in; everything here is +, -, *, /, sqrt in IEEE
// FP64 with explicit round-to-nearest intrinsics (no FMA contraction).
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include "fomo_device.cuh"
#include "fomo_internal.h"

namespace fomo {

namespace {

__device__ __forceinline__ unsigned long long d2ord(double d) {
  unsigned long long u = (unsigned long long)__double_as_longlong(d);
  return (u & 0x8000000000000000ull) ? ~u : (u | 0x8000000000000000ull);
}
__device__ __forceinline__ double ord2d(unsigned long long u) {
  u = (u & 0x8000000000000000ull) ? (u & 0x7fffffffffffffffull) : ~u;
  return __longlong_as_double((long long)u);
}

// float <-> int with the same order (atomicMax / atomicMin on floats)
__device__ __forceinline__ int ford(float f) {
  const int i = __float_as_int(f);
  return i >= 0 ? i : i ^ 0x7fffffff;
}
__device__ __forceinline__ float fdeord(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7fffffff); }

// The interval of view V's rotated coordinates (x', y', z' of nn:83-85) over
// block b's bounding box, widened by M: lo[a] <= the FP64 rotated coordinate
// a of every point of the block <= hi[a].  False for an empty block.  The
// rotation is evaluated in FP32 (centre . row +- |row| . half-size); M covers
// its rounding (M = 2E, E the FP32 screen's error bound below).
__device__ __forceinline__ bool block_interval(const SnapDev& snap, int64_t b, float cbf, float sbf, float clf,
                                               float slf, float M, float (&lo)[3], float (&hi)[3]) {
  const float* bb = snap.blk + FOMO_IDX(6 * b, 6 * (int64_t)snap.bdx * snap.bdy * snap.bdz, kSitePts);
  const float ax = bb[0], ay = bb[1], az = bb[2], bx = bb[3], by = bb[4], bz = bb[5];
  if (!(ax <= bx)) return false;  // empty
  const float cx = 0.5f * (ax + bx), cy = 0.5f * (ay + by), cz = 0.5f * (az + bz);
  const float hx = 0.5f * (bx - ax), hy = 0.5f * (by - ay), hz = 0.5f * (bz - az);
  // rows of the rotation: x' = (cb cl, -cb sl, -sb), y' = (sl, cl, 0), z' = (sb cl, -sb sl, cb)
  const float r[3][3] = {{cbf * clf, -cbf * slf, -sbf}, {slf, clf, 0.0f}, {sbf * clf, -sbf * slf, cbf}};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float m = r[a][0] * cx + r[a][1] * cy + r[a][2] * cz;
    const float e = fabsf(r[a][0]) * hx + fabsf(r[a][1]) * hy + fabsf(r[a][2]) * hz;
    lo[a] = m - e - M;
    hi[a] = m + e + M;
  }
  return true;
}

__device__ __forceinline__ float screen_bound(const GridParams& g) {
  return ldexpf(fmaxf(fabsf(g.minx), fabsf(g.maxx)) + fmaxf(fabsf(g.miny), fabsf(g.maxy)) +
                    fmaxf(fabsf(g.minz), fabsf(g.maxz)),
                -20);
}

// Phase 1 of the block-bounded extents (views other than Thomson), one thread
// per block: every point's rotated coordinate a lies in its block's interval,
// so the maximum over all points is at least the largest lower bound over the
// blocks, and the minimum at most the smallest upper bound.  grid: (blocks, views)
__global__ void view_bounds_kernel(SnapDev snap, ViewDesc* views) {
  ViewDesc* V = views + blockIdx.y;
  const int64_t nblk = (int64_t)snap.bdx * snap.bdy * snap.bdz;
  const float cbf = (float)V->rcb, sbf = (float)V->rsb, clf = (float)V->cl, slf = (float)V->sl;
  const float M = 2.0f * screen_bound(snap.g);
  float lbm[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX}, ubm[3] = {FLT_MAX, FLT_MAX, FLT_MAX};
  for (int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; b < nblk; b += (int64_t)gridDim.x * blockDim.x) {
    float lo[3], hi[3];
    if (!block_interval(snap, b, cbf, sbf, clf, slf, M, lo, hi)) continue;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lbm[a] = fmaxf(lbm[a], lo[a]);
      ubm[a] = fminf(ubm[a], hi[a]);
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lbm[a] = fmaxf(lbm[a], __shfl_xor_sync(0xffffffffu, lbm[a], o));
      ubm[a] = fminf(ubm[a], __shfl_xor_sync(0xffffffffu, ubm[a], o));
    }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      atomicMax(&V->bnd[2 * a], ford(lbm[a]));
      atomicMin(&V->bnd[2 * a + 1], ford(ubm[a]));
    }
  }
}

__device__ __forceinline__ void warp_minmax(unsigned long long& mn, unsigned long long& mx) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long a = __shfl_xor_sync(0xffffffffu, mn, o);
    unsigned long long b = __shfl_xor_sync(0xffffffffu, mx, o);
    mn = a < mn ? a : mn;
    mx = b > mx ? b : mx;
  }
}

// Thomson: every point takes the blended rotation in FP64, and its sin^2 chi.
// grid: (blocks over points, views)
__global__ void view_extents_kernel(SnapDev snap, ViewDesc* views, float* s2) {
  ViewDesc* V = views + blockIdx.y;
  const double cb = V->rcb, sb = V->rsb, cl = V->cl, sl = V->sl;
  const double blend = V->blend;
  const double omb = __dsub_rn(1.0, blend);
  unsigned long long mn[3] = {~0ull, ~0ull, ~0ull}, mx[3] = {0ull, 0ull, 0ull};
  float* s2v = s2 + (int64_t)blockIdx.y * snap.n;
  // LOS unit for sin^2 chi (thomson:194): clamped sin_b/cos_b with cos(l), sin(l)
  const double u0 = __dmul_rn(sb, cl), u1 = __dmul_rn(-sb, sl), u2 = cb;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < snap.n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const float4 p = snap.pts[i];
    const double gx = p.x, gy = p.y, gz = p.z;
    // full rotation (nn:83-85, thomson:179-181)
    double xa = __dsub_rn(__dsub_rn(__dmul_rn(__dmul_rn(gx, cb), cl), __dmul_rn(__dmul_rn(gy, cb), sl)),
                          __dmul_rn(gz, sb));
    double ya = __dadd_rn(__dmul_rn(gx, sl), __dmul_rn(gy, cl));
    double za = __dadd_rn(__dsub_rn(__dmul_rn(__dmul_rn(gx, sb), cl), __dmul_rn(__dmul_rn(gy, sb), sl)),
                          __dmul_rn(gz, cb));
    // pole rotation and blend (thomson:184-191)
    const double pxr = __dsub_rn(__dmul_rn(gx, cl), __dmul_rn(gy, sl));
    const double pyr = __dadd_rn(__dmul_rn(gx, sl), __dmul_rn(gy, cl));
    const double pzr = gz;
    xa = __dadd_rn(__dmul_rn(xa, omb), __dmul_rn(pxr, blend));
    ya = __dadd_rn(__dmul_rn(ya, omb), __dmul_rn(pyr, blend));
    za = __dadd_rn(__dmul_rn(za, omb), __dmul_rn(pzr, blend));
    // sin^2 chi = 1 - (u.r)^2 / (r.r)  (thomson:194-199)
    double ip = __dmul_rn(u0, xa);
    ip = __dadd_rn(ip, __dmul_rn(u1, ya));
    ip = __dadd_rn(ip, __dmul_rn(u2, za));
    double pp = __dmul_rn(xa, xa);
    pp = __dadd_rn(pp, __dmul_rn(ya, ya));
    pp = __dadd_rn(pp, __dmul_rn(za, za));
    s2v[FOMO_IDX(i, snap.n, kSiteS2)] = __double2float_rn(__dsub_rn(1.0, __ddiv_rn(__dmul_rn(ip, ip), pp)));
    const unsigned long long ex = d2ord(xa), ey = d2ord(ya), ez = d2ord(za);
    mn[0] = ex < mn[0] ? ex : mn[0];
    mx[0] = ex > mx[0] ? ex : mx[0];
    mn[1] = ey < mn[1] ? ey : mn[1];
    mx[1] = ey > mx[1] ? ey : mx[1];
    mn[2] = ez < mn[2] ? ez : mn[2];
    mx[2] = ez > mx[2] ? ez : mx[2];
  }
#pragma unroll
  for (int d = 0; d < 3; ++d) warp_minmax(mn[d], mx[d]);
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      atomicMin(&V->ext_bits[2 * d], mn[d]);
      atomicMax(&V->ext_bits[2 * d + 1], mx[d]);
    }
  }
}

// Phase 2, one warp per block: a block whose interval on some axis reaches the
// bound of phase 1 (above the largest lower bound, or below the smallest upper
// bound) may hold the point of that extreme, and only those blocks' points are
// rotated.  In FP32 first: |x32 - x64| <= E for every point (E: screen_bound), so the
// point of an FP64 extreme lies within 2E of the block's FP32 extreme and
// within E beyond phase 1's bound; a second pass over the block (from L1) rotates
// those points in FP64, a few per view.  (One pass with a running FP32 extreme
// rotated every new one in FP64, at 1/64 of the FP32 rate, and each lane met
// several: 35 to 48 us per launch, of the 100 us that a small render takes.)
// grid: (blocks / 4, views)
__global__ void view_extents_blocks_kernel(SnapDev snap, ViewDesc* views) {
  ViewDesc* V = views + blockIdx.y;
  const int lane = threadIdx.x & 31;
  const int64_t b = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t nblk = (int64_t)snap.bdx * snap.bdy * snap.bdz;
  if (b >= nblk) return;  // the whole warp
  const float cbf = (float)V->rcb, sbf = (float)V->rsb, clf = (float)V->cl, slf = (float)V->sl;
  const GridParams& g = snap.g;
  const float E = screen_bound(g);
  float lo[3], hi[3];
  if (!block_interval(snap, b, cbf, sbf, clf, slf, 2.0f * E, lo, hi)) return;
  float top[3], bot[3];  // phase 1's bounds of the maximum and the minimum
  bool reach = false;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    top[a] = fdeord(V->bnd[2 * a]);
    bot[a] = fdeord(V->bnd[2 * a + 1]);
    reach = reach || hi[a] >= top[a] || lo[a] <= bot[a];
  }
  if (!reach) return;
  const int bx = (int)(b % snap.bdx), by = (int)((b / snap.bdx) % snap.bdy), bz = (int)(b / ((int64_t)snap.bdx * snap.bdy));
  const int x0 = bx * kBlockCells, x1 = min(x0 + kBlockCells, g.dx) - 1;
  const int64_t entries = (int64_t)g.dx * g.dy * g.dz + 1;
  // this lane's two rows of the block's 8 x 8
  int p0[2], p1[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const int row = lane + 32 * r;
    const int cy = by * kBlockCells + row % kBlockCells, cz = bz * kBlockCells + row / kBlockCells;
    p0[r] = p1[r] = 0;
    if (cy < g.dy && cz < g.dz) {
      const int64_t rowbase = ((int64_t)cz * g.dy + cy) * g.dx;
      p0[r] = snap.cell_start[FOMO_IDX(rowbase + x0, entries, kSiteCellStart)];
      p1[r] = snap.cell_start[FOMO_IDX(rowbase + x1 + 1, entries, kSiteCellStart)];
    }
  }
  auto rotate32 = [&](const float4 p, float (&v)[3]) {
    v[0] = (p.x * cbf) * clf - (p.y * cbf) * slf - p.z * sbf;
    v[1] = p.x * slf + p.y * clf;
    v[2] = (p.x * sbf) * clf - (p.y * sbf) * slf + p.z * cbf;
  };
  float rmn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, rmx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
#pragma unroll
  for (int r = 0; r < 2; ++r)
    for (int i = p0[r]; i < p1[r]; ++i) {
      float v[3];
      rotate32(__ldg(snap.pts + FOMO_IDX(i, snap.n, kSitePts)), v);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        rmn[a] = fminf(rmn[a], v[a]);
        rmx[a] = fmaxf(rmx[a], v[a]);
      }
    }
  bool any = false;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    // what a point must reach: 2E from the block's extreme, E from the bound
    top[a] = fmaxf(top[a] - 2.0f * E, fdeord(__reduce_max_sync(0xffffffffu, ford(rmx[a]))) - 2.0f * E);
    bot[a] = fminf(bot[a] + 2.0f * E, fdeord(__reduce_min_sync(0xffffffffu, ford(rmn[a]))) + 2.0f * E);
    any = any || rmx[a] >= top[a] || rmn[a] <= bot[a];
  }
  unsigned long long mn[3] = {~0ull, ~0ull, ~0ull}, mx[3] = {0ull, 0ull, 0ull};
  if (any) {  // this lane has such points
    const double cb = V->rcb, sb = V->rsb, cl = V->cl, sl = V->sl;
#pragma unroll 1
    for (int r = 0; r < 2; ++r)
      for (int i = p0[r]; i < p1[r]; ++i) {
        const float4 p = __ldg(snap.pts + FOMO_IDX(i, snap.n, kSitePts));
        float v[3];
        rotate32(p, v);
        if (v[0] >= top[0] || v[0] <= bot[0] || v[1] >= top[1] || v[1] <= bot[1] || v[2] >= top[2] || v[2] <= bot[2]) {
          const double gx = p.x, gy = p.y, gz = p.z;
          // full rotation (nn:83-85)
          const double xa =
              __dsub_rn(__dsub_rn(__dmul_rn(__dmul_rn(gx, cb), cl), __dmul_rn(__dmul_rn(gy, cb), sl)),
                        __dmul_rn(gz, sb));
          const double ya = __dadd_rn(__dmul_rn(gx, sl), __dmul_rn(gy, cl));
          const double za =
              __dadd_rn(__dsub_rn(__dmul_rn(__dmul_rn(gx, sb), cl), __dmul_rn(__dmul_rn(gy, sb), sl)),
                        __dmul_rn(gz, cb));
          const unsigned long long ex = d2ord(xa), ey = d2ord(ya), ez = d2ord(za);
          mn[0] = ex < mn[0] ? ex : mn[0];
          mx[0] = ex > mx[0] ? ex : mx[0];
          mn[1] = ey < mn[1] ? ey : mn[1];
          mx[1] = ey > mx[1] ? ey : mx[1];
          mn[2] = ez < mn[2] ? ez : mn[2];
          mx[2] = ez > mx[2] ? ez : mx[2];
        }
      }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      if (mx[d]) {
        atomicMin(&V->ext_bits[2 * d], mn[d]);
        atomicMax(&V->ext_bits[2 * d + 1], mx[d]);
      }
    }
  }
}

__device__ __forceinline__ double dmax_ref(double a, double b) { return (a < b) ? b : a; }  // std::max

__device__ __forceinline__ float2 fp32_pair(double v) {
  const float hi = __double2float_rn(v);
  return make_float2(hi, __double2float_rn(__dsub_rn(v, (double)hi)));
}

// grid: (1 + chunks of kTabChunk table entries, views): an image side may have more chunks than
// the 65,535 of the grid's y axis.  Block (0, v) fills the view's scalars,
// independent chains of FP64 divisions on lanes of their own (on one thread, with
// the tables after them in the same block: 10 us per launch, an FP64 division
// taking about 0.7); the others fill the tables of ray x, ray y and LOS
// positions, one entry per thread, from the extents.
constexpr int kTabChunk = 128;
__global__ void __launch_bounds__(kTabChunk) view_finalize_kernel(ViewDesc* views, double3* ktab, float2* ktf, int ktab_stride) {
  ViewDesc* V = views + blockIdx.y;
  const double minx = ord2d(V->ext_bits[0]), maxx = ord2d(V->ext_bits[1]);
  const double miny = ord2d(V->ext_bits[2]), maxy = ord2d(V->ext_bits[3]);
  const double minz = ord2d(V->ext_bits[4]), maxz = ord2d(V->ext_bits[5]);
  const double dxr = __dsub_rn(maxx, minx), dyr = __dsub_rn(maxy, miny);
  const int nx = V->nx, ny = V->ny, nz = V->nz;
  if (blockIdx.x == 0) {
    __shared__ double s_px, s_py;
    if (threadIdx.x == 0) {
      V->minx = minx;
      V->maxx = maxx;
      V->dxr = dxr;
      s_px = __ddiv_rn(dxr, (double)(nx - 1));
    } else if (threadIdx.x == 32) {
      V->miny = miny;
      V->maxy = maxy;
      V->dyr = dyr;
      s_py = __ddiv_rn(dyr, (double)(ny - 1));
    } else if (threadIdx.x == 64) {
      V->minz = minz;
      V->maxz = maxz;
      double deltaz = __dsub_rn(maxz, minz), pathlength = __ddiv_rn(deltaz, (double)(nz - 1));
      if (nz != 1) deltaz = pathlength;
      V->deltaz = deltaz;
      if (maxz == minz || nz == 1) pathlength = 1.0;
      V->pathlength = pathlength;
      V->scale = __dmul_rn(__dmul_rn(pathlength, 1e8), 1.0);
    } else if (threadIdx.x == 96) {
      V->lwa = __ddiv_rn(__dmul_rn(V->lambda_width, V->lambda0), FOMO_SPEED_OF_LIGHT);
      V->ux = __double2float_rn(__dmul_rn(V->sb, V->cl));
      V->uy = __double2float_rn(__dmul_rn(-V->sb, V->sl));
      V->uz = __double2float_rn(V->cb);
    }
    __syncthreads();
    const double px = s_px, py = s_py;
    if (threadIdx.x == 0) {
      double md;
      if (V->method == kMethodThomson) {
        const double eq = dmax_ref(__dmul_rn(0.5, __dsqrt_rn(__dadd_rn(__dmul_rn(px, px), __dmul_rn(py, py)))),
                                   __ddiv_rn(__dmul_rn(0.1, dxr), (double)(nx - 1)));
        const double away = __ddiv_rn(dmax_ref(px, py), 0.005);
        md = __dadd_rn(__dmul_rn(eq, __dsub_rn(1.0, V->mdblend)), __dmul_rn(away, V->mdblend));
      } else {
        md = __ddiv_rn(dmax_ref(px, py), .3);
      }
      V->md = md;
    } else if (threadIdx.x == 64) {
      const float dxf = __double2float_rn(px), dyf = __double2float_rn(py);
      const double as = FOMO_PI / 180. / 3600.;
      const double apix = __dmul_rn(__dmul_rn(__ddiv_rn((double)dxf, FOMO_MM_PER_ARCSEC), __ddiv_rn((double)dyf, FOMO_MM_PER_ARCSEC)),
                                    __dmul_rn(as, as));
      V->apix = apix;
      V->scale_dn = __dmul_rn(__dmul_rn(V->pathlength, 1e8), apix);
    }
    return;
  }
  int i = (blockIdx.x - 1) * kTabChunk + threadIdx.x;
  if (i < nz) {
    double dz = __dsub_rn(maxz, minz);
    if (nz != 1) dz = __ddiv_rn(dz, (double)(nz - 1));
    const double z = __dadd_rn(__dmul_rn((double)i, dz), minz);  // nn:162
    const double zsb = __dmul_rn(z, V->sb);
    const double3 t = make_double3(__dmul_rn(zsb, V->cl), __dmul_rn(zsb, V->sl), __dmul_rn(z, V->cb));
    const int64_t k = (int64_t)blockIdx.y * ktab_stride + FOMO_IDX(i, ktab_stride, kSiteKtab);
    ktab[k] = t;
    if (ktf) {
      float2* f = ktf + 3 * k;
      f[0] = fp32_pair(t.x);
      f[1] = fp32_pair(-t.y);
      f[2] = fp32_pair(t.z);
    }
    return;
  }
  i -= nz;
  // ray positions in the image plane (nn:152-153)
  if (i < nx)
    V->xt[FOMO_IDX(i, nx, kSiteRayXY)] = __dadd_rn(__dmul_rn(__ddiv_rn((double)i, (double)(nx - 1)), dxr), minx);
  else if (i - nx < ny)
    V->yt[FOMO_IDX(i - nx, ny, kSiteRayXY)] = __dadd_rn(__dmul_rn(__ddiv_rn((double)(i - nx), (double)(ny - 1)), dyr), miny);
}

}  // namespace

FOMO_DEFINE_CHECK_READER(check_word_view)

cudaError_t launch_view_extents(SnapDev snap, ViewDesc* views, int nviews, float* s2, cudaStream_t s) {
  if (!s2) {
    // bounded by the per-block boxes: the blocks' intervals, then the points
    // of the blocks that reach the bounds
    const int64_t nblk = (int64_t)snap.bdx * snap.bdy * snap.bdz;
    int64_t b1 = (nblk + 255) / 256;
    if (b1 > 64) b1 = 64;
    view_bounds_kernel<<<dim3((unsigned)b1, (unsigned)nviews), 256, 0, s>>>(snap, views);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    view_extents_blocks_kernel<<<dim3((unsigned)((nblk + 3) / 4), (unsigned)nviews), 128, 0, s>>>(snap, views);
    return cudaGetLastError();
  }
  int64_t blocks = (snap.n + 255) / 256;
  int64_t cap = (152 * 8 + nviews - 1) / nviews;
  if (cap < 8) cap = 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  dim3 grid((unsigned)blocks, (unsigned)nviews);
  view_extents_kernel<<<grid, 256, 0, s>>>(snap, views, s2);
  return cudaGetLastError();
}

cudaError_t launch_view_finalize(ViewDesc* views, int nviews, double3* ktab, float2* ktf, int ktab_stride,
                                 int max_entries, cudaStream_t s) {
  const unsigned chunks = (unsigned)((max_entries + kTabChunk - 1) / kTabChunk);
  view_finalize_kernel<<<dim3(1 + chunks, (unsigned)nviews), kTabChunk, 0, s>>>(views, ktab, ktf, ktab_stride);
  return cudaGetLastError();
}

}  // namespace fomo
