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
#include "lines.cuh"

namespace osc {
namespace dev {

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

// Combine the warps' sums of a unit and store one partial per entry: S holds this warp's sums of entries
// lane + 32 k.
__device__ __forceinline__ void line_store(const FdWaveArgs& A, const WavePlan& P, int64_t tile, int g, int span,
                                           const LineEntry* e, double (*S)[6], double* dm, double* red) {
  const int lane = threadIdx.x & 31;
  line_combine(S, dm, red);
  if (threadIdx.x >= 32) return;
#pragma unroll
  for (int k = 0; k < kLnPer; ++k) {
    if (!e[k].live) continue;
    double* p = A.fused ? A.part + fused_part_index(P, tile, g, span, 0, lane + 32 * k, kLnTile)
                        : A.part + (e[k].slot * P.nseg * P.spans + g * P.spans + span) * kFdPartials;
    const int64_t cs = A.fused ? kLnTile : 1;
#pragma unroll
    for (int c = 0; c < 6; ++c) p[c * cs] = S[k][c];
    p[8 * cs] = dm[k];
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
    int per = 1;  // energies a lane in use
#pragma unroll
    for (int k = 0; k < kLnPer; ++k) {
      e[k] = line_entry(A, tile, n_act, lane + 32 * k);
      mw[k] = -A.omega[e[k].ie];
      if (__any_sync(0xffffffffu, e[k].live)) per = k + 1;
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
      auto sum = [&](auto used, auto trig) {
#pragma unroll 2
        for (int j = j0; j < j1; ++j) {
          const double2 a = t.te[j], b = t.ee[j];
#pragma unroll
          for (int k = 0; k < decltype(used)::value; ++k) {
            double sn, cs;
            trig(__dmul_rn(mw[k], a.x), &sn, &cs);
            S[k][0] = fma(a.y, cs, S[k][0]); S[k][1] = fma(a.y, sn, S[k][1]);
            S[k][2] = fma(b.x, cs, S[k][2]); S[k][3] = fma(b.x, sn, S[k][3]);
            S[k][4] = fma(b.y, cs, S[k][4]); S[k][5] = fma(b.y, sn, S[k][5]);
          }
        }
      };
      const auto fast = [](double ph, double* sn, double* cs) { sincos_fast(ph, sn, cs); };
      using Per = std::integral_constant<int, kLnPer>;
      if (near && per == kLnPer) sum(Per{}, fast);
      else if (near) sum(std::integral_constant<int, 1>{}, fast);
      else sum(Per{}, [](double ph, double* sn, double* cs) { sincos_far(ph, sn, cs); });
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
// MINB 4 and 5 CTAs an SM, 128 and 96 registers a thread (launch_fd_lines): long sums are bound by latency and gain from
// the fifth CTA (441 observers x 256 energies at level 12: 802 us at 4, 748 at 5, MUFU 71 % and issue slots 57 %
// busy), waves that are over after a unit or two a CTA lose by the fewer registers.
template <int MINB>
__global__ void __launch_bounds__(kLnThreads, MINB) k_fd_lines_mixed(FdWaveArgs A, MixedFrame F) {
  if (A.tile_entries != kLnTile) {
    if (threadIdx.x == 0) atomicOr(A.err, kErrPlan);
    return;
  }
  __shared__ __align__(16) LineStage st;
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
    LineSums sum;
    int per = 1;
#pragma unroll
    for (int k = 0; k < kLnPer; ++k) {
      e[k] = line_entry(A, tile, n_act, lane + 32 * k);
      const double om = A.omega[e[k].ie];
      line_energy(sum, k, om);
      if (__any_sync(0xffffffffu, e[k].live)) per = k + 1;
      if (e[k].live && warp == 0 && span == 0 && !mixed_geometry_ok(fx, fy, fz, om, F)) atomicOr(A.err, kErrBadArgs);
    }
    line_sum(st, chunk, rec, p0, p1, span > 0, make_pair_obs(fx, fy, fz, 0.0), per, A.fused && g == P.nseg - 1, sum);
    if (tid == 0) U.next = after;
    double dm[kLnPer];
#pragma unroll
    for (int k = 0; k < kLnPer; ++k) dm[k] = sum.wide[k] ? kPiD : 0.0;
    line_store(A, P, tile, g, span, e, sum.S, dm, red);
    if (A.fused) fused_unit_done_grouped<kLnThreads>(A, P, tile, n_act, &s_last, kLnTile, red, P.nseg * P.spans);
    else __syncthreads();
    u = U.next;
  }
}

}  // namespace dev

int lines_entries_per_cta() { return dev::kLnTile; }

int lines_blocks_per_sm(bool mixed) {
  int n = 0;
  if (mixed) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dev::k_fd_lines_mixed<5>, dev::kLnThreads, 0);
  else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dev::k_fd_lines_fp64, dev::kLnThreads, 0);
  return n > 0 ? n : 1;
}

cudaError_t launch_fd_lines(const FdWaveArgs& a, const MixedFrame* F, int grid, cudaStream_t st) {
  if (!F) return launch_overlapped(dev::k_fd_lines_fp64, grid, dev::kLnThreads, st, a);
  // The host does not know how many entries a later wave still has; what the level tells is that entries stop from
  // level 9 on, so that the waves up to 10, and fixed-level sums, hold most of a request's tiles, and later ones
  // fewer.  Kernels of a spectrum of 41 periods over four harmonics, by 4, by 5 and by this rule: 5001 energies 122, 127
  // and 117 us, 20000 205, 205 and 202; of 200 periods up to the ninth harmonic, whose entries stop at level 13 to 15,
  // 218, 228 and 213 us and 449, 443 and 444.  Below about 5000 energies every wave is short and 4 alone
  // would be 1 to 3 us faster (61 energies: 61, 67 and 62).  Either takes any grid (the fewer CTAs that fit
  // take more units each).
  return a.level <= 10 || !a.fused ? launch_overlapped(dev::k_fd_lines_mixed<5>, grid, dev::kLnThreads, st, a, *F)
                                   : launch_overlapped(dev::k_fd_lines_mixed<4>, grid, dev::kLnThreads, st, a, *F);
}

}  // namespace osc
