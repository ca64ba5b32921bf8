// lines.cuh -- sums of many photon energies at one observer: the mixed-precision terms formed once per pair
// of samples and added up for a tile of energies (the spectra's kernels and the batched ones).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>

#include "device_common.cuh"
#include "fd_common.cuh"

namespace osc {
namespace dev {

constexpr int kLnThreads = 128;
constexpr int kLnWarps = kLnThreads / 32;
constexpr int kLnPer = 2;               // energies per lane
constexpr int kLnTile = 32 * kLnPer;    // energies per tile

// The terms of pair_sample that do not depend on the energy, one pair per thread.
constexpr int kLnFold = 16;             // pairs per FP32 partial sum before it is folded into FP64
constexpr int kLnPairs = kLnThreads;    // pairs per chunk

struct LinePairs {
  float4 v01[kLnPairs];   // v_x, v_y of both samples
  float4 v2k[kLnPairs];   // v_z and -1/(D om)
  float4 ct[kLnPairs];    // D - R_z and tau_s of both samples
  double2 d[kLnPairs];    // the first sample's FP64 D - R_z and tau_s
  float2 s[kLnPairs];     // second sample minus first: D - R_z and tau_s
};

// The pair's terms into slot i, with the operations of pair_sample and fp64_turns.
__device__ __forceinline__ void line_pair(const float4* __restrict__ q, const PairObs& o, LinePairs& t, int i) {
  const float4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4], q5 = q[5], q6 = q[6];
  const double2* dq = reinterpret_cast<const double2*>(q + 7);
  const double2 DXY = dq[0], DZT = dq[1];
  const float2 X = make_float2(q0.x, q0.y), Y = make_float2(q0.z, q0.w);
  const float2 Z = make_float2(q1.x, q1.y), T = make_float2(q1.z, q1.w);
  const float2 NBX = make_float2(q2.x, q2.y), NBY = make_float2(q2.z, q2.w);
  const float2 EB = make_float2(q3.x, q3.y), BZ = make_float2(q3.z, q3.w);
  const float2 G = make_float2(q4.x, q4.y), AZ = make_float2(q4.z, q4.w);
  const float2 AX = make_float2(q5.x, q5.y), AY = make_float2(q5.z, q5.w);
  const float2 M1 = f2(-1.f);
  const float2 rx = fma2(X, M1, o.ox), ry = fma2(Y, M1, o.oy), rz = fma2(Z, M1, o.oz);
  const float2 rho2 = fma2(rx, rx, mul2(ry, ry));
  const float2 d2 = fma2(rz, rz, rho2);
  const float2 iD = make_float2(rsqrt_ftz(d2.x), rsqrt_ftz(d2.y));
  const float2 ri = mul2(rho2, iD);
  const float2 qq = mul2(ri, iD);
  const float2 corr = mul2(ri, fma2(f2(0.125f), qq, f2(0.5f)));
  const float2 DD = mul2(d2, iD);
  const float inv = rcp_ftz(DD.x + DD.y);
  const float num = fmaf(q6.x, rx.x + rx.y, fmaf(q6.y, ry.x + ry.y, -q6.z * (corr.x + corr.y)));
  const float2 nx = mul2(rx, iD), ny = mul2(ry, iD), en = mul2(corr, iD);
  const float2 ux = add2(nx, NBX), uy = add2(ny, NBY), uz = fma2(en, M1, EB);
  const float2 om = fma2(ny, NBY, fma2(nx, NBX, fma2(en, BZ, EB)));
  const float2 nio = make_float2(rcp_ftz(-om.x), rcp_ftz(-om.y));
  const float2 na = fma2(nx, AX, fma2(ny, AY, mul2(fma2(en, M1, f2(1.f)), AZ)));
  const float2 nh = mul2(nio, fma2(G, iD, na));
  const float2 vx = fma2(nh, ux, AX), vy = fma2(nh, uy, AY), vz = fma2(nh, uz, AZ);
  const float2 nk2 = mul2(nio, iD);
  t.v01[i] = make_float4(vx.x, vx.y, vy.x, vy.y);
  t.v2k[i] = make_float4(vz.x, vz.y, nk2.x, nk2.y);
  t.ct[i] = make_float4(corr.x, corr.y, T.x, T.y);
  t.d[i] = make_double2(fp64_corr(DXY.x, DXY.y, DZT.x, corr.x, 0.5f * iD.x, o), DZT.y);
  t.s[i] = make_float2(num * inv, q6.w);
}

// Shared memory of a CTA's pair terms: two chunks, and D - R_z and tau_s of the sample before chunk c at c & 3
// (NaN: none).
struct LineStage {
  LinePairs t[2];
  float2 before[4];
};

// A lane's energies: frequency factors, sums, and whether a phase step reached pi (all that the stop rule asks).
struct LineSums {
  float2 w[kLnPer], wc[kLnPer];
  float wt[kLnPer], wct[kLnPer];
  bool wide[kLnPer];
  double dwt[kLnPer], dwct[kLnPer], S[kLnPer][6];
};
__device__ __forceinline__ void line_energy(LineSums& e, int k, double om) {
  const PairObs o = make_pair_obs(0.0, 0.0, 0.0, om);
  e.w[k] = o.w; e.wc[k] = o.wc; e.wt[k] = o.wt; e.wct[k] = o.wct; e.dwt[k] = o.dwt; e.dwct[k] = o.dwct;
  e.wide[k] = false;
#pragma unroll
  for (int c = 0; c < 6; ++c) e.S[k][c] = 0;
}

// Whether a phase step of the warp's pairs [j0, j1) reaches pi, for each of a lane's energies.  A step is
// |P_j - P_{j-1}| of P = RN(wc corr + RN(w T)), so it stays below wc |dcorr| + w |dT| plus the roundings of both P
// (2^-24 (wc |corr| + 2 w |T|) each) and of the bound itself.  The quarter's largest |dcorr|, |dT|, |corr| and |T| serve
// all energies, and a step is formed as such only where that bound does not clear pi (the coarse levels) and no earlier
// step settled it: 6 of the 39 instructions an (energy, pair) took when every step was formed.
__device__ __forceinline__ void line_steps(const LinePairs& t, float2 before, int j0, int j1, int per, LineSums& e) {
  float dc = 0.f, dt = 0.f, c = 0.f, tt = 0.f;
  for (int j = j0 + (threadIdx.x & 31); j < j1; j += 32) {
    const float4 ct = t.ct[j];
    const float2 b = j > 0 ? make_float2(t.ct[j - 1].y, t.ct[j - 1].w) : before;  // (NaN: no step into the pair)
    dc = fmaxf(dc, fmaxf(fabsf(ct.x - b.x), fabsf(ct.y - ct.x)));
    dt = fmaxf(dt, fmaxf(fabsf(ct.z - b.y), fabsf(ct.w - ct.z)));
    c = fmaxf(c, fmaxf(fmaxf(fabsf(ct.x), fabsf(ct.y)), fabsf(b.x)));
    tt = fmaxf(tt, fmaxf(fmaxf(fabsf(ct.z), fabsf(ct.w)), fabsf(b.y)));
  }
  auto over_warp = [](float v) { return __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(v))); };
  dc = over_warp(dc); dt = over_warp(dt); c = over_warp(c); tt = over_warp(tt);
#pragma unroll
  for (int k = 0; k < kLnPer; ++k) {
    if (k >= per || e.wide[k]) continue;
    const float wc = fabsf(e.wc[k].x), w = fabsf(e.w[k].x);
    if (fmaf(wc, dc, w * dt) * 1.00001f + fmaf(wc, c, 2.f * w * tt) * 2.5e-7f < 3.1415f) continue;
    const float2 b = j0 > 0 ? make_float2(t.ct[j0 - 1].y, t.ct[j0 - 1].w) : before;
    float last = fmaf(e.wc[k].x, b.x, __fmul_rn(e.w[k].x, b.y));
    for (int j = j0; j < j1; ++j) {
      const float4 ct = t.ct[j];
      const float2 ph = fma2(e.wc[k], make_float2(ct.x, ct.y), mul2(e.w[k], make_float2(ct.z, ct.w)));
      e.wide[k] |= (double)fmaxf(fabsf(ph.x - last), fabsf(ph.y - ph.x)) >= kPiD;
      last = ph.y;
    }
  }
}

// Pairs [p0, p1) of `rec` for the tile: `joins` when pair p0 - 1 precedes them; `per` (1 or kLnPer, uniform over
// the CTA) energies a lane are in use; `steps` (uniform) when the stop rule will read their phase steps.  Every
// thread of the CTA takes part.  The folds of 16 pairs start at the quarter chunks' starts, as in
// k_fd_wave_mixed_pair.
__device__ __forceinline__ void line_sum(LineStage& st, unsigned& chunk, const float4* __restrict__ rec, int64_t p0,
                                         int64_t p1, bool joins, const PairObs& o, int per, bool steps, LineSums& e) {
  const int tid = threadIdx.x, warp = tid >> 5;
  for (int64_t lo = p0; lo < p1; lo += kLnPairs, ++chunk) {
    const int n = (int)min((int64_t)kLnPairs, p1 - lo);
    LinePairs& t = st.t[chunk & 1u];
    if (tid < n) {
      line_pair(rec + kPairF4 * (lo + tid), o, t, tid);
      if (tid == n - 1) st.before[(chunk + 1) & 3u] = make_float2(t.ct[tid].y, t.ct[tid].w);
    }
    if (lo == p0 && tid == (n < kLnThreads ? kLnThreads - 1 : 0)) {  // the predecessor
      float2 b = f2(__int_as_float(0x7fc00000));
      if (joins) {
        const float* r = reinterpret_cast<const float*>(rec + kPairF4 * (lo - 1));
        b = make_float2(pair_corr(r[1], r[3], r[5], o), r[7]);
      }
      st.before[chunk & 3u] = b;
    }
    __syncthreads();
    const int j0 = (warp * n) / kLnWarps, j1 = ((warp + 1) * n) / kLnWarps;
    if (steps) line_steps(t, st.before[chunk & 3u], j0, j1, per, e);
    auto folds = [&](auto used) {
      constexpr int PER = decltype(used)::value;
      for (int jb = j0; jb < j1; jb += kLnFold) {
        const int je = min(j1, jb + kLnFold);
        float2 acc[PER][6];
#pragma unroll
        for (int k = 0; k < PER; ++k)
#pragma unroll
          for (int c = 0; c < 6; ++c) acc[k][c] = f2(0.f);
#pragma unroll 4
        for (int j = jb; j < je; ++j) {
          const float4 v01 = t.v01[j], v2k = t.v2k[j];
          const double2 d = t.d[j];
          const float2 s = t.s[j];
          const float2 vx = make_float2(v01.x, v01.y), vy = make_float2(v01.z, v01.w), vz = make_float2(v2k.x, v2k.y);
          const float2 nk2 = make_float2(v2k.z, v2k.w);
#pragma unroll
          for (int k = 0; k < PER; ++k) {
            const float t0 = turn_fraction(fma(e.dwct[k], d.x, fma(e.dwt[k], d.y, kTurnBase)));
            const float t1 = t0 + fmaf(e.wct[k], s.x, e.wt[k] * s.y);
            const float2 ph = mul2(make_float2(t0, t1), f2(kTwoPiF));
            float2 sn, cs;
            sincos_ftz(ph.x, &sn.x, &cs.x);
            sincos_ftz(ph.y, &sn.y, &cs.y);
            const float2 kc = mul2(nk2, cs), ks = mul2(nk2, sn);
            acc[k][0] = fma2(vx, kc, acc[k][0]);
            acc[k][1] = fma2(vx, ks, acc[k][1]);
            acc[k][2] = fma2(vy, kc, acc[k][2]);
            acc[k][3] = fma2(vy, ks, acc[k][3]);
            acc[k][4] = fma2(vz, kc, acc[k][4]);
            acc[k][5] = fma2(vz, ks, acc[k][5]);
          }
        }
#pragma unroll
        for (int k = 0; k < PER; ++k)
#pragma unroll
          for (int c = 0; c < 6; c += 2) {
            e.S[k][c] += (double)acc[k][c].x + (double)acc[k][c].y;
            e.S[k][c + 1] -= (double)acc[k][c + 1].x + (double)acc[k][c + 1].y;
          }
      }
    };
    if (per == kLnPer) folds(std::integral_constant<int, kLnPer>{});
    else folds(std::integral_constant<int, 1>{});
  }
}

// Combine the warps' sums of a unit in warp order: warp 0 gets them.  red: (kLnWarps - 1) x 7 x kLnTile doubles.
__device__ __forceinline__ void line_combine(double (*S)[6], double* dm, double* red) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp > 0) {
#pragma unroll
    for (int k = 0; k < kLnPer; ++k) {
      double* r = red + (warp - 1) * 7 * kLnTile + lane + 32 * k;
#pragma unroll
      for (int c = 0; c < 6; ++c) r[c * kLnTile] = S[k][c];
      r[6 * kLnTile] = dm[k];
    }
  }
  __syncthreads();
  if (warp != 0) return;
#pragma unroll
  for (int k = 0; k < kLnPer; ++k)
    for (int w = 0; w < kLnWarps - 1; ++w) {
      const double* r = red + w * 7 * kLnTile + lane + 32 * k;
#pragma unroll
      for (int c = 0; c < 6; ++c) S[k][c] += r[c * kLnTile];
      dm[k] = fmax(dm[k], r[6 * kLnTile]);
    }
}

}  // namespace dev
}  // namespace osc
