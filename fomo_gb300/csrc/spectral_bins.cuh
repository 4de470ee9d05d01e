// One warp's spectra of one pixel: the line profiles of a list of points summed
// in the lambda bins of up to NL lines.  The emission pass of the march and the
// projection bin through it.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "fomo_device.cuh"
#include "fomo_internal.h"

namespace fomo {

// A warp's staging: a batch's points and the bins' wavelengths, per line.
template <int NL, int NB>
struct __align__(16) BinShared {
  float4 runs[NL][32];
  float2 scale[NL];         // of the written sums, as an FP32 pair
  float lams[NL][NB * 32];  // lambdaval (nn:200), evaluated in FP64 on the host, stored FP32
};

// NL lines x up to NB 32-bin windows per line.  A batch's points (a point and
// the number of samples it stands for) are staged as (peak x length, 2/w, Doppler
// term) per line, compacted to those with a neighbour, and binned line by line and
// window by window: the warp is four groups of eight lanes, group g adds points g,
// g + 4, ... and each lane evaluates four of the window's bins.  With one point
// for the whole warp, every (point, line) cost a 16-byte broadcast to 32 lanes, 512
// bytes through the shared-memory port, which was the bound (64 views x 4 lines
// of 256 x 256 x 512 samples: 22.7 ms, L1 at 85 %); a load now serves four points
// (18.0 ms).  The groups' sums are joined by an exchange that leaves bin `lane`
// in each lane, and folded into the pixel's Kahan sum.  PAIRS: the sums are scaled
// by FP32 pairs where that decides their rounding (scaled), else in FP64.
template <int NL, int NB, bool PAIRS>
struct SpectralBins {
  float acc[NL][NB], comp[NL][NB], shk[NL];
  const float2* ew[NL];
  int nw[NL];  // windows of the line; 0: the view has fewer lines than the launch

  // Warp-collective, as all members: the lines of view V.
  __device__ __forceinline__ void view(const ViewDesc* V, const LineDesc* LD, int nlines, BinShared<NL, NB>& sh) {
    const int lane = threadIdx.x & 31, L = V->L;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      const bool on = l < nlines && LD[l].ew != nullptr;
      ew[l] = on ? LD[l].ew : nullptr;
      shk[l] = on ? LD[l].shift_k : 0.0f;
      nw[l] = on ? min(LD[l].nw, NB) : 0;
      const double scale = on && LD[l].is_dn ? V->scale_dn : V->scale;
      const float high = __double2float_rn(scale);
      const bool usable = fabsf(high) > 1e-30f && fabsf(high) < 1e37f;  // else NaN: every value takes FP64
      if (PAIRS && lane == 0)
        sh.scale[l] = make_float2(usable ? high : __int_as_float(0x7fffffff), __double2float_rn(__dsub_rn(scale, (double)high)));
#pragma unroll
      for (int m = 0; m < NB; ++m) {
        if (m < nw[l]) {
          const int il = LD[l].wstart + m * 32 + lane;
          sh.lams[l][m * 32 + lane] = il < L ? __ldg(LD[l].lam + FOMO_IDX(il, L, kSiteLam)) : 3.0e30f;
        }
      }
    }
    __syncwarp();
  }

  // The next pixel's sums start.
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int l = 0; l < NL; ++l)
#pragma unroll
      for (int m = 0; m < NB; ++m) acc[l][m] = comp[l][m] = 0.0f;
  }

  // Lane i < m adds point pos (sorted position; -1: none) len times.
  __device__ __forceinline__ void add(const SnapDev& snap, const ViewDesc* V, BinShared<NL, NB>& sh, int m, int pos,
                                      int len, unsigned long long* stats) {
    constexpr unsigned kAll = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int group = lane >> 3;
    const unsigned fills = __ballot_sync(kAll, lane < m && pos >= 0);
    const int nruns = __popc(fills);
    if (!nruns) return;
    const int npad = (nruns + 3) & ~3;
    if (lane < m && pos >= 0) {
      const float cnt = (float)len;
      const float4 vv = __ldg(snap.vel + FOMO_IDX(pos, snap.n, kSitePts));
      float2 pw[NL];
#pragma unroll
      for (int l = 0; l < NL; ++l)
        pw[l] = nw[l] ? __ldg(ew[l] + FOMO_IDX(pos, snap.n, kSitePts)) : make_float2(0.0f, 1.0f);
      const float vlos = fmaf(V->uz, vv.z, fmaf(V->uy, vv.y, V->ux * vv.x));
      const int d = __popc(fills & ((1u << lane) - 1u));
#pragma unroll
      for (int l = 0; l < NL; ++l) {
        // a peak of 0 (intpolpeak ? ... : 0, nn:204) is staged as all zeros and adds nothing
        // exp(-4 ln2 (d/w)^2) = 2^(-(2d/w)^2); one Newton step takes the quotient's 2 ulp, which the exponent
        // doubles, to half an ulp (not where w is 0 or out of range)
        float sc = __fdividef(2.0f, pw[l].y);
        const float rest = fmaf(-pw[l].y, sc, 2.0f);
        if (fabsf(rest) < 1e-3f) sc = fmaf(0.5f * sc, rest, sc);
        sh.runs[l][d] = pw[l].x != 0.0f ? make_float4(pw[l].x * cnt, sc, -(vlos * shk[l]) * sc, 0.0f)
                                        : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    }
    if (lane >= nruns && lane < npad) {
#pragma unroll
      for (int l = 0; l < NL; ++l) sh.runs[l][lane] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    __syncwarp();
    if (stats && lane == 0) {
      int nwin = 0;
#pragma unroll
      for (int l = 0; l < NL; ++l) nwin += nw[l];
      atomicAdd(stats + kStatRuns, (unsigned long long)nruns);
      atomicAdd(stats + kStatEx2, 32ull * (unsigned long long)(nruns * nwin));
    }
#pragma unroll
    for (int l = 0; l < NL; ++l) {
#pragma unroll
      for (int m2 = 0; m2 < NB; ++m2) {
        if (m2 >= nw[l]) break;
        float lam[4], part[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          lam[j] = sh.lams[l][m2 * 32 + 8 * j + (lane & 7)];
          part[j] = 0.0f;
        }
#pragma unroll 2
        for (int q0 = group; q0 < npad; q0 += 4) {
          const float4 t = sh.runs[l][q0];  // the same address in the group's lanes
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float q = fmaf(lam[j], t.y, t.z);
            part[j] = fmaf(t.x, ex2_approx(-q * q), part[j]);
          }
        }
        // lane 8 g + i ends with the four groups' sum of bin 8 g + i
        const bool hi = lane & 16, mid = lane & 8;
        const float k0 = (hi ? part[2] : part[0]) + __shfl_xor_sync(kAll, hi ? part[0] : part[2], 16);
        const float k1 = (hi ? part[3] : part[1]) + __shfl_xor_sync(kAll, hi ? part[1] : part[3], 16);
        kahan_add(acc[l][m2], comp[l][m2], (mid ? k1 : k0) + __shfl_xor_sync(kAll, mid ? k0 : k1, 8));
      }
    }
    __syncwarp();  // the staged points are rewritten by the next batch
  }

  // fl(scale (acc - comp)) in FP64, and from FP32 pairs where their bound (2^-43; they err by less than 2^-44, the FP64
  // expression by 2^-52) decides the rounding: the same bits.  A Kahan sum's rest is below 2^-22 of it, so three
  // operations split the difference; 2^-146 in the bound covers what a tiny product's low part loses below the normal
  // range; an overflow makes the low part NaN, which decides nothing.  FP64 runs at 1/64 of the FP32 rate, and where rays
  // have few runs the writes were the emission pass's time: 300 x 300 rays, 4 lines x 100 bins, 2.4 / 27 / 86 runs a ray 469 /
  // 637 / 1491 us in FP64, 250 / 516 / 1450 from pairs.
  static __device__ __forceinline__ float scaled_f64(double scale, float acc, float comp) {
    return __double2float_rn(__dmul_rn(scale, __dsub_rn((double)acc, (double)comp)));
  }
  static __device__ __forceinline__ float scaled(const double* scale, float2 s, float acc, float comp) {
    const float v = __fsub_rn(acc, comp), rest = __fsub_rn(__fsub_rn(acc, v), comp);
    const float p = __fmul_rn(v, s.x);
    const float low = fmaf(v, s.x, -p) + fmaf(v, s.y, rest * s.x);
    float out;
    if (!pair_round(p, low, fmaf(fabsf(p), 1.14e-13f, 1.2e-44f), out))
      out = acc == 0.0f && s.x == s.x ? p : scaled_f64(*scale, acc, comp);
    return out;
  }

  // The pixel's spectra, scaled, into the cubes; ATOMIC: added to what is there.
  template <bool ATOMIC = false>
  __device__ __forceinline__ void write(const ViewDesc* V, const LineDesc* LD, const BinShared<NL, NB>& sh, int64_t ray) {
    const int lane = threadIdx.x & 31, L = V->L;
    const int64_t ncube = (int64_t)V->nx * V->ny * L;
#pragma unroll
    for (int l = 0; l < NL; ++l) {
      if (nw[l]) {
        const double* at = LD[l].is_dn ? &V->scale_dn : &V->scale;
        const double scale = PAIRS ? 0.0 : *at;
        float* out = LD[l].out;
        const int wlo = LD[l].wstart, whi = wlo + 32 * nw[l];
        for (int il = lane; !ATOMIC && il < L; il += 32)
          if (il < wlo || il >= whi) out[FOMO_IDX(ray * L + il, ncube, kSiteCube)] = 0.0f;  // below 2^-64 of every peak
#pragma unroll
        for (int m = 0; m < NB; ++m) {
          const int il = wlo + m * 32 + lane;
          if (m < nw[l] && il < L) {
            // the sum with what its last additions dropped
            const float v = PAIRS ? scaled(at, sh.scale[l], acc[l][m], comp[l][m]) : scaled_f64(scale, acc[l][m], comp[l][m]);
            if (ATOMIC)
              atomicAdd(out + FOMO_IDX(ray * L + il, ncube, kSiteCube), v);
            else
              out[FOMO_IDX(ray * L + il, ncube, kSiteCube)] = v;
          }
        }
      }
    }
  }
};

}  // namespace fomo
