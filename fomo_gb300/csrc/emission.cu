// K1: per-point emissivity, computed once per (snapshot, table, observation
// type) and kept resident next to the sorted points.
//
//  * emission_kernel restates emissionfromdatacube (fomo-c/src/fomo-CHIANTI.cpp:
//    228-322): log10 of n and T (fomo-operations.cpp:63-84, <= 0 -> 0), the
//    G(T, n) lookup of goft (fomo-CHIANTI.cpp:64-121: linear in logT, nearest
//    in logn, index arithmetic in FP32, interpolation in FP64), the thermal
//    FWHM of linefwhm (:220-226) and eps = k * 10^(2 log n) * G / w (:292-293),
//    rounding to FP32 at the same points as the reference's vector operators.
//    log10 is that of FP64 rounded once (correctly rounded except for
//    double-rounding cases); glibc's log10f is within 1 ulp of that.
//  * thomson_emission_kernel restates thomsonfromdatacube / getThomsonGeomFactor
//    (fomo-thomson.cpp:39-92).
// The G table is staged in shared memory when it fits.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>

#include "fomo_device.cuh"
#include "fomo_internal.h"

namespace fomo {

namespace {

constexpr int kMaxSmemTableFloats = 40 * 1024;  // 160 KB: covers the 200x200 instrument tables

// FP64 runs at 1/64 of the FP32 rate on this GPU, and a point's two log10, pow,
// interpolation and two scalings in FP64 were all of the kernel's time (2M points:
// 682 us; the bytes take 5).  Each of these FP64 results is rounded to FP32 as
// soon as it is there, so it is computed as an unevaluated sum of two FP32 numbers
// first, with a bound E on its error: where hi + (lo + E) and hi + (lo - E) round to
// the same float, the FP64 result (whose own error is far below E) rounds to it too.
// Where they differ (at most one value in 8,000 over 14 <= a < 22, n and T from 1e4 to
// 1e12) the FP64 expression is evaluated as before.  The results are the same bits.
// The logarithm and the exponential are table-driven reductions with short
// series, after P. T. P. Tang, ACM TOMS 16 (1990) 378 and 15 (1989) 144.
__device__ __noinline__ float log10_f64(float v) { return __double2float_rn(log10((double)v)); }
__device__ __noinline__ float exp10_f64(float a) { return __double2float_rn(pow(10.0, (double)a)); }
__device__ __noinline__ float lerp_f64(float lT, float fx1, float fy1, float fx2, float fy2) {
  // goft (fomo-CHIANTI.cpp:95-116)
  const double x1 = fx1, y1 = fy1, x2 = fx2, y2 = fy2;
  return __double2float_rn(__dadd_rn(
      __ddiv_rn(__dmul_rn(__dsub_rn((double)lT, x1), __dsub_rn(y2, y1)), __dsub_rn(x2, x1)), y1));
}
__device__ __noinline__ float scale_f64(double c, float v) { return __double2float_rn(__dmul_rn(c, (double)v)); }

// Lookup tables of the FP32 pairs, made on the host in FP64.
constexpr int kLogTab = 128, kExpTab = 128;
struct PairTables {
  float4 lg[kLogTab];  // for a mantissa in [1 + i/128, 1 + (i+1)/128): c = fl(1 / middle), -log10(c) high and low
  float2 ex[kExpTab];  // 2^(i/128)
  float2 el[256];      // log10(2) times (biased exponent - 127)
};

// fl(log10 v), v > 0.  v = 2^e m, log10 v = e log10 2 - log10 c + log10(1 + r) with r = m c
// - 1, |r| < 2^-7.9: the series' first term as a pair, the rest (below 2^-17)
// in FP32.  The lower parts stay below 2^-16 and are added with errors of 2^-41 each.
__device__ __forceinline__ float log10_rn(float v, const PairTables& tab) {
  const unsigned u = __float_as_uint(v);
  const unsigned be = u >> 23;
  if (be == 0u || be >= 255u) return log10_f64(v);  // subnormal, infinite, NaN
  const float m = __uint_as_float((u & 0x007fffffu) | 0x3f800000u);
  const float4 c = tab.lg[(u >> 16) & 127u];
  const float2 el = tab.el[be];
  const float p = __fmul_rn(m, c.x), rl = fmaf(m, c.x, -p), r = __fsub_rn(p, 1.0f);
  constexpr float Kh = 0.434294492f, Kl = -1.0103050118e-8f;  // 1 / ln 10
  const float t = __fmul_rn(r, Kh);
  const float rk = rl * Kh;
  float low = fmaf(r, Kh, -t) + fmaf(r, Kl, fmaf(-rk, r, rk));
  low += r * r * (-0.5f * Kh + r * (Kh / 3.0f + r * (-0.25f * Kh + r * (0.2f * Kh))));
  const Pair s1 = two_sum(el.x, c.y), s2 = two_sum(s1.h, t);
  low += (s1.l + s2.l) + (el.y + c.z);
  float out;
  if (!pair_round(s2.h, low, 3.6e-12f, out)) out = log10_f64(v);  // 2^-38
  return out;
}

// fl(10^a).  10^a = 2^n 2^(j/128) 2^g, |g| <= 1/256: the argument and 2^g - 1 as pairs.
__device__ __forceinline__ float exp10_rn(float a, const PairTables& tab) {
  if (!(a > -36.0f && a < 38.0f)) return exp10_f64(a);
  constexpr float Lh = 3.32192802f, Ll = 7.0595369e-8f;    // log2 10
  constexpr float Eh = 0.693147182f, El = -1.9046542e-9f;  // ln 2
  const float y = __fmul_rn(a, Lh), yl = fmaf(a, Lh, -y) + a * Ll;
  const float nf = rintf(y * 128.0f);
  const int n = (int)nf;
  const Pair g = two_sum(fmaf(nf, -0.0078125f, y), yl);
  const float uh = __fmul_rn(g.h, Eh);
  const float ul = fmaf(g.h, Eh, -uh) + fmaf(g.h, El, g.l * Eh);
  const float vl = fmaf(uh, ul, ul) + uh * uh * (0.5f + uh * (0.16666667f + uh * (0.041666668f + uh * 0.0083333333f)));
  const float2 T = tab.ex[n & 127];
  const float q = __fmul_rn(T.x, uh), ql = fmaf(T.x, uh, -q);
  const float s = __fadd_rn(T.x, q), e = __fsub_rn(q, __fsub_rn(s, T.x));
  const float low = (e + ql) + fmaf(T.x, vl, fmaf(T.y, uh, T.y));
  float out;
  if (!pair_round(s, low, 3.6e-12f, out)) return exp10_f64(a);  // 2^-38 of a value in [1, 2)
  // the exponent in two steps: the first stays in range, the second is exact (a normal result)
  const int k = n >> 7;
  return out * __uint_as_float((unsigned)(127 + k / 2) << 23) * __uint_as_float((unsigned)(127 + k - k / 2) << 23);
}

// fl(((lT - x1) (y2 - y1)) / (x2 - x1) + y1) of the FP64 expression.  The table values
// are scaled by 2^64, so that the low parts of the smallest ones stay normal.
__device__ __forceinline__ float lerp_rn(float lT, float x1, float y1, float x2, float y2) {
  constexpr float up = 18446744073709551616.0f, down = 5.421010862427522e-20f;
  const float big = fmaxf(fabsf(y1), fabsf(y2));
  if (big == 0.0f) return lerp_f64(lT, x1, y1, x2, y2);
  const float a1 = y1 * up, a2 = y2 * up;
  const Pair dx = two_sum(lT, -x1), dn = two_sum(x2, -x1), dy = two_sum(a2, -a1);
  // (dx.h + dx.l) (dy.h + dy.l)
  const float p = __fmul_rn(dx.h, dy.h);
  const float pl = fmaf(dx.h, dy.h, -p) + fmaf(dx.h, dy.l, dx.l * dy.h);
  const float q = __fdiv_rn(p, dn.h);
  const float ql = __fdividef(fmaf(-q, dn.h, p) + pl - q * dn.l, dn.h);
  const Pair s = two_sum(a1, q);
  float out;
  const float E = (fabsf(q) + big * up) * 2.3e-13f;  // 2^-42 of the terms
  const bool ok = pair_round(s.h, s.l + ql, E, out) && big < 1e18f;
  out *= down;
  // the scaled value rounds as the value itself only where that is a normal number
  if (!ok || !(fabsf(out) > 2.4e-38f)) out = lerp_f64(lT, x1, y1, x2, y2);
  return out;
}

// fl(c v), c = ch + cl (FP64 constant as a pair).
__device__ __forceinline__ float scale_rn(double c, float ch, float cl, float v) {
  const float p = __fmul_rn(ch, v), pl = fmaf(ch, v, -p) + cl * v;
  float out;
  if (v == 0.0f && fabsf(ch) < 1e37f) return p;
  if (!(pair_round(p, pl, fabsf(p) * 2.9e-14f, out) && fabsf(p) > 1e-30f && fabsf(p) < 1e37f && fabsf(ch) > 1e-30f))
    out = scale_f64(c, v);  // 2^-45
  return out;
}

template <bool kSmem>
__global__ void __launch_bounds__(256) emission_kernel(const float* __restrict__ ne_s, const float* __restrict__ T_s,
                                                       int64_t n, TableDev t, const __grid_constant__ PairTables pt,
                                                       float2* __restrict__ ew, unsigned int* __restrict__ wmax_bits) {
  extern __shared__ float sm[];
  __shared__ PairTables tab;
  __shared__ unsigned int smax;
  for (int i = threadIdx.x; i < kLogTab; i += blockDim.x) tab.lg[i] = pt.lg[i];
  for (int i = threadIdx.x; i < kExpTab; i += blockDim.x) tab.ex[i] = pt.ex[i];
  for (int i = threadIdx.x; i < 256; i += blockDim.x) tab.el[i] = pt.el[i];
  if (threadIdx.x == 0) smax = 0u;
  const float* G = t.G;
  const float* logT = t.logT;
  if (kSmem) {
    float* sG = sm;
    float* sT = sm + (size_t)t.nt * t.nrho;
    for (int i = threadIdx.x; i < t.nt * t.nrho; i += blockDim.x) sG[i] = t.G[i];
    for (int i = threadIdx.x; i < t.nt; i += blockDim.x) sT[i] = t.logT[i];
    G = sG;
    logT = sT;
  }
  __syncthreads();
  const float T0 = t.logT[0], T1 = t.logT[1];
  const float r0 = t.logn[0], r1 = t.logn[1];
  const float dT = __fsub_rn(T1, T0), dR = __fsub_rn(r1, r0);
  const float cwh = __double2float_rn(t.cw), cwl = __double2float_rn(__dsub_rn(t.cw, (double)cwh));
  const float kh = __double2float_rn(t.k), kl = __double2float_rn(__dsub_rn(t.k, (double)kh));
  unsigned int m = 0u;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float nv = ne_s[i];
    const float Tv = T_s[i];
    const float logrho = nv <= 0.0f ? 0.0f : log10_rn(nv, tab);
    const float lT = Tv <= 0.0f ? 0.0f : log10_rn(Tv, tab);
    // goft (fomo-CHIANTI.cpp:95-116)
    float g = 0.0f;
    const float qT = floorf(__fdiv_rn(__fsub_rn(lT, T0), dT));
    const float qR = roundf(__fdiv_rn(__fsub_rn(logrho, r0), dR));
    if (qT >= 0.0f && qT + 1.0f <= (float)(t.nt - 1) && qR >= 0.0f && qR <= (float)(t.nrho - 1)) {
      const int ft = (int)qT, ct = ft + 1, ri = (int)qR;
      const int gi = ri * t.nt + ct;
      const int ng = t.nt * t.nrho;
      g = lerp_rn(lT, logT[FOMO_IDX(ct, t.nt, kSiteTable)], G[FOMO_IDX(gi, ng, kSiteTable)],
                  logT[FOMO_IDX(ft, t.nt, kSiteTable)], G[FOMO_IDX(gi - 1, ng, kSiteTable)]);
    }
    const float w = t.imaging ? 1.0f : scale_rn(t.cw, cwh, cwl, __fsqrt_rn(Tv));
    const float a = __fmul_rn(2.0f, logrho);  // exact, as the FP64 product is
    const float b = exp10_rn(a, tab);
    const float c = __fmul_rn(b, g);
    const float d = scale_rn(t.k, kh, kl, c);
    const float e = __fdiv_rn(d, w);
    ew[i] = make_float2(e, w);
    // the largest width among points that emit (eps != 0) bounds the lambda window the march
    // evaluates; NaN and inf map to +inf (the host then evaluates every bin).  Non-negative floats
    // order like their bits.
    if (e != 0.0f) {
      float wa = fabsf(w);
      if (!(wa <= 3.0e38f)) wa = __int_as_float(0x7f800000);
      m = max(m, __float_as_uint(wa));
    }
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(&smax, m);
  __syncthreads();
  if (threadIdx.x == 0 && smax) atomicMax(wmax_bits, smax);
}

// getThomsonGeomFactor (fomo-thomson.cpp:39-58), FP32 storage points as there.
__device__ void thomson_geom(float r, float* totterm, float* polterm) {
  const double U = FOMO_LIMB_U;
  const float sinomega = __double2float_rn(__ddiv_rn(FOMO_RSUN, (double)r));
  const float coeff = __double2float_rn(
      __dmul_rn(__dmul_rn(0.5 * FOMO_PI, __dmul_rn(FOMO_ELECTRON_RADIUS, FOMO_ELECTRON_RADIUS)), FOMO_IRRADIANCE));
  const float ss = __fmul_rn(sinomega, sinomega);
  const float cs = __fsub_rn(1.0f, ss);
  const float co = __fsqrt_rn(cs);
  const float lt = __double2float_rn(log(__ddiv_rn(__dadd_rn(1.0, (double)sinomega), (double)co)));
  const float a = __fmul_rn(co, ss);
  const double dss = ss, dcs = cs, dso = sinomega, dlt = lt;
  const float b = __double2float_rn(__dmul_rn(
      -1.0 / 8.0, __dsub_rn(__dsub_rn(1.0, __dmul_rn(3.0, dss)),
                            __dmul_rn(__dmul_rn(dcs, __ddiv_rn(__dadd_rn(1.0, __dmul_rn(3.0, dss)), dso)), dlt))));
  const float c = __double2float_rn(__dsub_rn(__dsub_rn(4.0 / 3.0, (double)co), __ddiv_rn((double)__fmul_rn(co, cs), 3.0)));
  const float d = __double2float_rn(__dmul_rn(
      1.0 / 8.0, __dsub_rn(__dadd_rn(5.0, dss), __dmul_rn(__dmul_rn(dcs, __ddiv_rn(__dsub_rn(5.0, dss), dso)), dlt))));
  const double kk = __dmul_rn((double)coeff, 1. / (1. - U / 3.));
  *polterm = __double2float_rn(__dmul_rn(kk, __dadd_rn((double)a, __dmul_rn(U, (double)__fsub_rn(b, a)))));
  *totterm = __double2float_rn(
      __dmul_rn(kk, __dmul_rn(2.0, __dadd_rn((double)c, __dmul_rn(U, (double)__fsub_rn(d, c))))));
}

__global__ void thomson_emission_kernel(const float4* __restrict__ pts, const float* __restrict__ ne_s, int64_t n,
                                        float2* __restrict__ totpol) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float4 p = pts[i];
    const double px = p.x, py = p.y, pz = p.z;
    const float r = __double2float_rn(
        __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(px, px), __dmul_rn(py, py)), __dmul_rn(pz, pz))));
    float tt, pt;
    thomson_geom(r, &tt, &pt);
    const float nv = ne_s[i];
    totpol[i] = make_float2(__fmul_rn(nv, tt), __fmul_rn(nv, pt));
  }
}

// Largest speed |v| of a snapshot: bounds the Doppler shift of every LOS.
// One atomic per block (per warp, 19,456 of them on one address took most of the kernel's 17 us).
__global__ void speed_max_kernel(const float4* __restrict__ vel, int64_t n, unsigned int* vmax_bits) {
  __shared__ unsigned int smax;
  if (threadIdx.x == 0) smax = 0u;
  __syncthreads();
  unsigned int m = 0u;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const float4 v = vel[i];
    float s = sqrtf(fmaf(v.z, v.z, fmaf(v.y, v.y, v.x * v.x))) * 1.0001f;
    if (!(s <= 3.0e38f)) s = __int_as_float(0x7f800000);
    m = max(m, __float_as_uint(s));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) atomicMax(&smax, m);
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(vmax_bits, smax);
}

// Sorted payload back to the caller's point order: out[orig(i)] = ew[i].
__global__ void unsort_kernel(const float4* __restrict__ pts, const float2* __restrict__ ew, int64_t n,
                              float* __restrict__ a, float* __restrict__ b) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t o = FOMO_IDX(__float_as_int(pts[i].w), n, kSitePts);
    const float2 v = ew[i];
    a[o] = v.x;
    b[o] = v.y;
  }
}

int blocks_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  if (b > 152 * 16) b = 152 * 16;
  if (b < 1) b = 1;
  return (int)b;
}

}  // namespace

FOMO_DEFINE_CHECK_READER(check_word_emission)

cudaError_t launch_emission(const float* ne_s, const float* T_s, int64_t n, TableDev t, float2* ew,
                            unsigned int* wmax_bits, cudaStream_t s) {
  static const PairTables pt = [] {
    PairTables p;
    auto split = [](double v, float& h, float& l) {
      h = (float)v;
      l = (float)(v - (double)h);
    };
    for (int i = 0; i < kLogTab; ++i) {
      p.lg[i].x = (float)(1.0 / (1.0 + (i + 0.5) / kLogTab));
      split(-std::log10((double)p.lg[i].x), p.lg[i].y, p.lg[i].z);
      p.lg[i].w = 0.0f;
    }
    for (int i = 0; i < kExpTab; ++i) split(std::exp2((double)i / kExpTab), p.ex[i].x, p.ex[i].y);
    for (int i = 0; i < 256; ++i) split((i - 127) * std::log10(2.0), p.el[i].x, p.el[i].y);
    return p;
  }();
  cudaError_t e = cudaMemsetAsync(wmax_bits, 0, sizeof(unsigned int), s);
  if (e != cudaSuccess) return e;
  // a few blocks per SM: each first copies the tables to shared memory
  const int blocks = std::min(blocks_for(n, 256), 152 * 4);
  const int64_t tab = (int64_t)t.nt * t.nrho + t.nt;
  if (tab <= kMaxSmemTableFloats) {
    const size_t bytes = (size_t)tab * sizeof(float);
    if (bytes > 40 * 1024) {
      e = cudaFuncSetAttribute(emission_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
      if (e != cudaSuccess) return e;
    }
    emission_kernel<true><<<blocks, 256, bytes, s>>>(ne_s, T_s, n, t, pt, ew, wmax_bits);
  } else {
    emission_kernel<false><<<blocks, 256, 0, s>>>(ne_s, T_s, n, t, pt, ew, wmax_bits);
  }
  return cudaGetLastError();
}

cudaError_t launch_speed_max(const float4* vel, int64_t n, unsigned int* vmax_bits, cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(vmax_bits, 0, sizeof(unsigned int), s);
  if (e != cudaSuccess) return e;
  speed_max_kernel<<<std::min(blocks_for(n, 256), 152 * 4), 256, 0, s>>>(vel, n, vmax_bits);
  return cudaGetLastError();
}

cudaError_t launch_unsort_payload(const float4* pts, const float2* ew, int64_t n, float* a, float* b,
                                  cudaStream_t s) {
  unsort_kernel<<<blocks_for(n, 256), 256, 0, s>>>(pts, ew, n, a, b);
  return cudaGetLastError();
}

cudaError_t launch_thomson_emission(const float4* pts, const float* ne_s, int64_t n, float2* totpol,
                                    cudaStream_t s) {
  thomson_emission_kernel<<<blocks_for(n, 256), 256, 0, s>>>(pts, ne_s, n, totpol);
  return cudaGetLastError();
}

}  // namespace fomo
