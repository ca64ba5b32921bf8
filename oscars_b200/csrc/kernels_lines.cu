// kernels_lines.cu -- frequency-domain sums of many photon energies at one observer (spectra).
//
// The retarded time and the amplitude of a sample depend on the observer, not on the energy; only the
// phase, its sine and cosine and the sums do.  Here each CTA forms the samples' terms once, one sample
// (pair) per thread, in shared memory, and its 4 warps, each on a quarter of the staged samples, add
// them up for 64 energies, two per lane.  A term costs the FP64 kernel 59 + 3 instructions and an
// energy 26 more (95 for the pair when every energy forms its own term); the mixed kernel ~85 and ~33.
// Results: the operations of k_fd_wave_fp64 and of pair_sample (same phases, amplitudes, sine and
// cosine; the mixed kernel also keeps the FP32 sums of 16 pairs), so only the order of the FP64 sums
// differs.
#include <cstdint>
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "fd_common.cuh"
#include "kernels.h"

namespace osc {
namespace dev {

constexpr int kLnThreads = 128;
constexpr int kLnWarps = kLnThreads / 32;
constexpr int kLnPer = 2;               // energies per lane
constexpr int kLnTile = 32 * kLnPer;    // energies per tile

// What both kernels share: the wave's units (tile, segment, span), spans fastest; a CTA starts with its
// own and takes the others from the counter.
struct LineUnits {
  WavePlan P;
  int64_t next;
};
__device__ __forceinline__ void line_unit_range(const WavePlan& P, int64_t u, int64_t& b0, int64_t& b1) {
  const int64_t r = u >> P.log2_spans;
  const int g = P.nseg == 2 ? (int)(r & 1) : 0;
  b0 = seg_begin(P, g) + (u & (P.spans - 1)) * seg_span(P, g);
  b1 = min(seg_end(P, g), b0 + seg_span(P, g));
}

// Entry of slot q of a tile: the active list's (one observer), or, without a list, energy block
// tile % A.e_tiles of observer tile / A.e_tiles.
struct LineEntry {
  int64_t slot;
  unsigned item, ie;
  bool live;
};
__device__ __forceinline__ LineEntry line_entry(const FdWaveArgs& A, int64_t tile, int64_t n_act, int q) {
  LineEntry e;
  if (A.act) {
    e.slot = tile * kLnTile + q;
    e.live = e.slot < n_act;
    e.item = e.live ? (unsigned)A.act[e.slot] : 0u;
    e.ie = e.item;
  } else {
    const int64_t io = tile / A.e_tiles;
    e.ie = (unsigned)(tile - io * A.e_tiles) * kLnTile + (unsigned)q;
    e.live = e.ie < (unsigned)A.n_e;
    if (!e.live) e.ie = 0;
    e.slot = io * A.n_e + e.ie;
    e.item = (unsigned)e.slot;
  }
  return e;
}

// Combine the warps' sums of a unit in warp order and store one partial per entry: S holds this warp's
// sums of entries lane + 32 k.  red: (kLnWarps - 1) x 7 x kLnTile doubles.
__device__ __forceinline__ void line_store(const FdWaveArgs& A, const WavePlan& P, int64_t tile, int g, int span,
                                           const LineEntry* e, double (*S)[6], const double* dm, double* red) {
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
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < kLnPer; ++k) {
      double m = dm[k];
      for (int w = 0; w < kLnWarps - 1; ++w) {
        const double* r = red + w * 7 * kLnTile + lane + 32 * k;
#pragma unroll
        for (int c = 0; c < 6; ++c) S[k][c] += r[c * kLnTile];
        m = fmax(m, r[6 * kLnTile]);
      }
      if (!e[k].live) continue;
      double* p = A.fused ? A.part + fused_part_index(P, tile, g, span, 0, lane + 32 * k, kLnTile)
                          : A.part + (e[k].slot * P.nseg * P.spans + g * P.spans + span) * kFdPartials;
      const int64_t cs = A.fused ? kLnTile : 1;
#pragma unroll
      for (int c = 0; c < 6; ++c) p[c * cs] = S[k][c];
      p[8 * cs] = m;
    }
  }
}

// ---- FP64 ---------------------------------------------------------------------------------------
// Phase steps: |RN(w tau_j) - RN(w tau_{j-1})| >= pi is decided for a warp's quarter of a chunk from the
// largest |tau_j - tau_{j-1}| (rounded up to a float) unless w times it lies within the roundings'
// reach of pi, in which case the quarter's steps are formed one by one.
constexpr int kLnChunk = kLnThreads;  // samples per chunk, one per thread

struct LineTerms {
  double2 te[kLnChunk];  // tau, e_x
  double2 ee[kLnChunk];  // e_y, e_z
};

__global__ void __launch_bounds__(kLnThreads, 4) k_fd_lines_fp64(FdWaveArgs A) {
  if (A.tile_entries != kLnTile) {  // the host sized the partials for another tile
    if (threadIdx.x == 0) atomicOr(A.err, kErrPlan);
    return;
  }
  __shared__ __align__(16) LineTerms st[2];
  __shared__ double before[4];  // tau of the sample before chunk c, at c & 3 (NaN: none)
  __shared__ double red[(kLnWarps - 1) * 7 * kLnTile];
  __shared__ LineUnits U;
  __shared__ int s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  launch_dependents();
  wait_predecessor();
  if (A.fused && blockIdx.x == 0 && tid == 0) {  // counters of the following wave
    if (A.zero_u32) *A.zero_u32 = 0;
    if (A.zero_u64) *A.zero_u64 = 0;
  }
  const int64_t n_act = A.act ? (int64_t)*A.n_act : A.n_items;
  if (tid == 0) {
    U.P = wave_plan(A.first, A.level, n_act, kLnTile, A.target_units, A.min_span);
    if (!A.act) U.P.tiles = A.n_items / A.n_e * A.e_tiles;
  }
  __syncthreads();
  const WavePlan& P = U.P;
  const int64_t units = (P.tiles * P.nseg) << P.log2_spans;
  const double* L = A.lev;
  const int64_t cap = A.cap;
  int64_t u = blockIdx.x;
  unsigned chunk = 0;  // chunks taken so far
  while (u < units) {
    int64_t b0, b1;
    line_unit_range(P, u, b0, b1);
    const int span = (int)u & (P.spans - 1);
    const int g = P.nseg == 2 ? (int)(u >> P.log2_spans) & 1 : 0;
    const int64_t tile = u >> (P.log2_spans + P.nseg - 1);
    int64_t after = 0;
    if (tid == 0) after = (int64_t)gridDim.x + (int64_t)atomicAdd(A.work, 1ull);
    if (b0 == 0) b0 = 1;  // sample 0 is the unused slot
    double smp[10];       // this thread's sample of the chunk ahead
    auto fetch = [&](int64_t lo) {
      const double* q = L + min(lo + tid, b1 - 1);
#pragma unroll
      for (int c = 0; c < 10; ++c) smp[c] = q[c * cap];
    };
    fetch(b0);
    const double* ob = A.obs + 3 * (A.act ? 0 : tile / A.e_tiles);
    const double Ox = ob[0], Oy = ob[1], Oz = ob[2];
    LineEntry e[kLnPer];
    double mw[kLnPer], S[kLnPer][6];
    bool wide[kLnPer];
#pragma unroll
    for (int k = 0; k < kLnPer; ++k) {
      e[k] = line_entry(A, tile, n_act, lane + 32 * k);
      mw[k] = -A.omega[e[k].ie];
      wide[k] = false;
#pragma unroll
      for (int c = 0; c < 6; ++c) S[k][c] = 0;
    }
    bool near = true;
#pragma unroll
    for (int k = 0; k < kLnPer; ++k) near = near && phase_reach(A, Ox, Oy, Oz, mw[k]) < kPhaseFast;
    near = __all_sync(0xffffffffu, near);
    for (int64_t lo = b0; lo < b1; lo += kLnChunk, ++chunk) {
      const int n = (int)min((int64_t)kLnChunk, b1 - lo);
      LineTerms& t = st[chunk & 1u];
      if (tid < n) {
        const FdTerm f = fd_term(smp[0], smp[1], smp[2], smp[3], smp[4], smp[5], smp[6], smp[7], smp[8], smp[9],
                                 one_minus_b2(smp[4], smp[5], smp[6]), Ox, Oy, Oz);
        t.te[tid] = make_double2(f.tau, f.ex);
        t.ee[tid] = make_double2(f.ey, f.ez);
        if (tid == n - 1) before[(chunk + 1) & 3u] = f.tau;
      }
      if (lo == b0 && tid == (n < kLnThreads ? kLnThreads - 1 : 0)) {  // the unit's first chunk: the span's predecessor
        double tau = __longlong_as_double(0x7ff8000000000000ll);
        if (span > 0) {
          const double* q = L + lo - 1;
          tau = fd_tau(q[0], q[cap], q[2 * cap], q[3 * cap], Ox, Oy, Oz);
        }
        before[chunk & 3u] = tau;
      }
      __syncthreads();
      if (lo + kLnChunk < b1) fetch(lo + kLnChunk);
      const int j0 = (warp * n) / kLnWarps, j1 = ((warp + 1) * n) / kLnWarps;
      // the quarter's largest step and |tau|, rounded up
      float dt = 0.f, ta = 0.f;
      if (j0 + lane < j1) {
        const int j = j0 + lane;
        const double tj = t.te[j].x, tp = j > 0 ? t.te[j - 1].x : before[chunk & 3u];
        const double d = fabs(tj - tp);
        dt = d == d ? __double2float_ru(d) : 0.f;
        ta = __double2float_ru(fabs(tj) + (d == d ? d : 0.0));
      }
      dt = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(dt)));
      ta = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(ta)));
#pragma unroll
      for (int k = 0; k < kLnPer; ++k) {
        // both phases are rounded, and their difference: 2^-52 |w tau| each, and 2^-23 for the float
        const double step = fabs(mw[k]) * (double)dt, reach = fabs(mw[k]) * (double)ta * 1e-15 + step * 3e-7;
        if (step + reach < kPiD) continue;
        if (step - reach >= kPiD) {
          wide[k] = true;
          continue;
        }
        for (int j = j0; j < j1; ++j) {
          const double tp = j > 0 ? t.te[j - 1].x : before[chunk & 3u];
          wide[k] |= fabs(__dsub_rn(__dmul_rn(mw[k], t.te[j].x), __dmul_rn(mw[k], tp))) >= kPiD;
        }
      }
      auto sum = [&](auto trig) {
#pragma unroll 2
        for (int j = j0; j < j1; ++j) {
          const double2 a = t.te[j], b = t.ee[j];
#pragma unroll
          for (int k = 0; k < kLnPer; ++k) {
            double sn, cs;
            trig(__dmul_rn(mw[k], a.x), &sn, &cs);
            S[k][0] = fma(a.y, cs, S[k][0]); S[k][1] = fma(a.y, sn, S[k][1]);
            S[k][2] = fma(b.x, cs, S[k][2]); S[k][3] = fma(b.x, sn, S[k][3]);
            S[k][4] = fma(b.y, cs, S[k][4]); S[k][5] = fma(b.y, sn, S[k][5]);
          }
        }
      };
      if (near) sum([](double ph, double* sn, double* cs) { sincos_fast(ph, sn, cs); });
      else sum([](double ph, double* sn, double* cs) { sincos_far(ph, sn, cs); });
    }
    if (tid == 0) U.next = after;
    double dm[kLnPer];
#pragma unroll
    for (int k = 0; k < kLnPer; ++k) dm[k] = wide[k] ? kPiD : 0.0;
    line_store(A, P, tile, g, span, e, S, dm, red);
    if (A.fused) fused_unit_done_grouped<kLnThreads>(A, P, tile, n_act, &s_last, kLnTile, red, P.nseg * P.spans);
    else __syncthreads();
    u = U.next;
  }
}

// ---- mixed --------------------------------------------------------------------------------------
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

__global__ void __launch_bounds__(kLnThreads, 4) k_fd_lines_mixed(FdWaveArgs A, MixedFrame F) {
  if (A.tile_entries != kLnTile) {
    if (threadIdx.x == 0) atomicOr(A.err, kErrPlan);
    return;
  }
  __shared__ __align__(16) LinePairs st[2];
  __shared__ float2 before[4];  // D - R_z and tau_s of the sample before chunk c, at c & 3 (NaN: none)
  __shared__ double red[(kLnWarps - 1) * 7 * kLnTile];
  __shared__ LineUnits U;
  __shared__ int s_last;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  launch_dependents();
  wait_predecessor();
  if (A.fused && blockIdx.x == 0 && tid == 0) {
    if (A.zero_u32) *A.zero_u32 = 0;
    if (A.zero_u64) *A.zero_u64 = 0;
  }
  const int64_t n_act = A.act ? (int64_t)*A.n_act : A.n_items;
  if (tid == 0) {
    U.P = wave_plan(A.first, A.level, n_act, kLnTile, A.target_units, A.min_span);
    if (!A.act) U.P.tiles = A.n_items / A.n_e * A.e_tiles;
  }
  __syncthreads();
  const WavePlan& P = U.P;
  const int64_t units = (P.tiles * P.nseg) << P.log2_spans;
  const float4* rec = reinterpret_cast<const float4*>(A.lev);
  int64_t u = blockIdx.x;
  unsigned chunk = 0;
  while (u < units) {
    int64_t b0, b1;
    line_unit_range(P, u, b0, b1);
    const int64_t p0 = b0 >> 1, p1 = b1 > b0 ? b1 >> 1 : p0;  // spans are whole pairs
    const int span = (int)u & (P.spans - 1);
    const int g = P.nseg == 2 ? (int)(u >> P.log2_spans) & 1 : 0;
    const int64_t tile = u >> (P.log2_spans + P.nseg - 1);
    int64_t after = 0;
    if (tid == 0) after = (int64_t)gridDim.x + (int64_t)atomicAdd(A.work, 1ull);
    const double* ob = A.obs + 3 * (A.act ? 0 : tile / A.e_tiles);
    const double* R = F.rot;
    const double ox = ob[0] - F.x0[0], oy = ob[1] - F.x0[1], oz = ob[2] - F.x0[2];
    const double fx = R[0] * ox + R[1] * oy + R[2] * oz;
    const double fy = R[3] * ox + R[4] * oy + R[5] * oz;
    const double fz = R[6] * ox + R[7] * oy + R[8] * oz;
    LineEntry e[kLnPer];
    float2 w[kLnPer], wc[kLnPer];
    float wt[kLnPer], wct[kLnPer], dmax[kLnPer];
    double dwt[kLnPer], dwct[kLnPer], S[kLnPer][6];
#pragma unroll
    for (int k = 0; k < kLnPer; ++k) {
      e[k] = line_entry(A, tile, n_act, lane + 32 * k);
      const double om = A.omega[e[k].ie];
      const PairObs o = make_pair_obs(fx, fy, fz, om);
      w[k] = o.w; wc[k] = o.wc; wt[k] = o.wt; wct[k] = o.wct; dwt[k] = o.dwt; dwct[k] = o.dwct;
      if (e[k].live && warp == 0 && span == 0 && !mixed_geometry_ok(fx, fy, fz, om, F)) atomicOr(A.err, kErrBadArgs);
      dmax[k] = 0.f;
#pragma unroll
      for (int c = 0; c < 6; ++c) S[k][c] = 0;
    }
    const PairObs o = make_pair_obs(fx, fy, fz, 0.0);
    for (int64_t lo = p0; lo < p1; lo += kLnPairs, ++chunk) {
      const int n = (int)min((int64_t)kLnPairs, p1 - lo);
      LinePairs& t = st[chunk & 1u];
      if (tid < n) {
        line_pair(rec + kPairF4 * (lo + tid), o, t, tid);
        if (tid == n - 1) before[(chunk + 1) & 3u] = make_float2(t.ct[tid].y, t.ct[tid].w);
      }
      if (lo == p0 && tid == (n < kLnThreads ? kLnThreads - 1 : 0)) {  // the span's predecessor
        float2 b = f2(__int_as_float(0x7fc00000));
        if (span > 0) {
          const float* r = reinterpret_cast<const float*>(rec + kPairF4 * (lo - 1));
          b = make_float2(pair_corr(r[1], r[3], r[5], o), r[7]);
        }
        before[chunk & 3u] = b;
      }
      __syncthreads();
      const int j0 = (warp * n) / kLnWarps, j1 = ((warp + 1) * n) / kLnWarps;
      float last[kLnPer];
      {
        const float2 b = j0 > 0 ? make_float2(t.ct[max(j0, 1) - 1].y, t.ct[max(j0, 1) - 1].w) : before[chunk & 3u];
#pragma unroll
        for (int k = 0; k < kLnPer; ++k) last[k] = fmaf(wc[k].x, b.x, __fmul_rn(w[k].x, b.y));
      }
      for (int jb = j0; jb < j1; jb += kLnFold) {
        const int je = min(j1, jb + kLnFold);
        float2 acc[kLnPer][6];
#pragma unroll
        for (int k = 0; k < kLnPer; ++k)
#pragma unroll
          for (int c = 0; c < 6; ++c) acc[k][c] = f2(0.f);
#pragma unroll 2
        for (int j = jb; j < je; ++j) {
          const float4 v01 = t.v01[j], v2k = t.v2k[j], ct = t.ct[j];
          const double2 d = t.d[j];
          const float2 s = t.s[j];
          const float2 vx = make_float2(v01.x, v01.y), vy = make_float2(v01.z, v01.w), vz = make_float2(v2k.x, v2k.y);
          const float2 nk2 = make_float2(v2k.z, v2k.w), corr = make_float2(ct.x, ct.y), T = make_float2(ct.z, ct.w);
#pragma unroll
          for (int k = 0; k < kLnPer; ++k) {
            const float2 ph32 = fma2(wc[k], corr, mul2(w[k], T));
            dmax[k] = fmaxf(dmax[k], fmaxf(fabsf(ph32.x - last[k]), fabsf(ph32.y - ph32.x)));
            last[k] = ph32.y;
            const float t0 = turn_fraction(fma(dwct[k], d.x, fma(dwt[k], d.y, kTurnBase)));
            const float t1 = t0 + fmaf(wct[k], s.x, wt[k] * s.y);
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
        for (int k = 0; k < kLnPer; ++k)
#pragma unroll
          for (int c = 0; c < 6; c += 2) {
            S[k][c] += (double)acc[k][c].x + (double)acc[k][c].y;
            S[k][c + 1] -= (double)acc[k][c + 1].x + (double)acc[k][c + 1].y;
          }
      }
    }
    if (tid == 0) U.next = after;
    double dm[kLnPer];
#pragma unroll
    for (int k = 0; k < kLnPer; ++k) dm[k] = (double)dmax[k];
    line_store(A, P, tile, g, span, e, S, dm, red);
    if (A.fused) fused_unit_done_grouped<kLnThreads>(A, P, tile, n_act, &s_last, kLnTile, red, P.nseg * P.spans);
    else __syncthreads();
    u = U.next;
  }
}

}  // namespace dev

int lines_entries_per_cta() { return dev::kLnTile; }

int lines_blocks_per_sm(bool mixed) {
  int n = 0;
  if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dev::k_fd_lines_mixed, dev::kLnThreads, 0);
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dev::k_fd_lines_fp64, dev::kLnThreads, 0);
  return n > 0 ? n : 1;
}

cudaError_t launch_fd_lines(const FdWaveArgs& a, const MixedFrame* F, int grid, cudaStream_t st) {
  return F ? launch_overlapped(dev::k_fd_lines_mixed, grid, dev::kLnThreads, st, a, *F)
           : launch_overlapped(dev::k_fd_lines_fp64, grid, dev::kLnThreads, st, a);
}

}  // namespace osc
