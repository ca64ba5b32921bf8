// kernels_fp64.cu -- the reference's FP64 method on sm_100a.
//
// Level samples (trajectory spline evaluated at the level-ladder times), the frequency-domain
// (flux / spectrum) and time-domain (power density) sums over those samples, and the per-level
// convergence tests.  Every operation whose rounding can move the retarded phase or the
// 1 - n.beta denominators is written with explicit round-to-nearest intrinsics in the reference's
// association order, so those quantities are bit-identical to the reference CPU build; only the
// order of the final summation and the last-ulp behaviour of sin/cos/pow differ.
//
// Work decomposition ("waves"): every (observer, energy) entry that is still unconverged at level
// L needs the 2^L samples of that level.  A wave's CTAs take units (tile of entries x segment x span of
// the level); each thread owns one entry and walks its part of the span's samples, which a single
// elected thread stages into shared memory with 1-D TMA bulk copies (double buffered, mbarrier
// completion).  All threads read the same sample at the same time (shared-memory broadcast).  Per-span
// partial sums go to global memory; the CTA that finishes a tile's last unit reduces them in span order,
// applies the reference's stop rule and compacts the still-active entries for the next wave (the
// allocation-free entry keeps a finalize kernel).
#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>

#include "device_common.cuh"
#include "fd_common.cuh"
#include "kernels.h"

namespace osc {
namespace dev {

// ---------------------------------------------------------------------------------------------
// Level samples: TParticleTrajectoryInterpolated::FillTParticleTrajectoryPointsLevel
// (src/TParticleTrajectoryInterpolated.cc:124-158) + TSpline1D3::GetValue (include/TOMATH.h:92-121).
// Sample i of level L lives at index 2^L + i of each of the 10 SoA arrays (index 0 unused), so the
// union of levels 0..L is the contiguous range [1, 2^(L+1)) and every level starts 16-byte aligned.
// Levels above ext_from hold the reference's extended levels (same count 2^L, their own spacing:
// level_time), which it evaluates on the fly instead of storing.
// ---------------------------------------------------------------------------------------------
__global__ void k_level_fill(const double* __restrict__ knots, int64_t n, double tstart, double tstop,
                             int64_t s_begin, int64_t s_end, double* __restrict__ lev, int64_t cap, int ext_from) {
  const int64_t s = s_begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= s_end) return;
  const double T = level_time(tstart, tstop, s, ext_from);
  double v[9];
  spline_eval9(knots, n, T, v);
  lev[s] = T;
#pragma unroll
  for (int c = 0; c < 9; ++c) lev[(1 + c) * cap + s] = v[c];
}

// Per-level max |beta_i - beta_{i-1}| over i >= 1 (the power-density stop rule, src/OSCARSSR.cc:
// 2887-2891).  Positive doubles order like their bit patterns, so atomicMax on the bits is exact.
__global__ void k_level_betadiff(const double* __restrict__ lev, int64_t cap, int64_t s_begin, int64_t s_end,
                                 unsigned long long* __restrict__ bdmax_bits) {
  __shared__ unsigned long long blk[32];  // per-level maxima of this block, merged into global at the end
  if (threadIdx.x < 32) blk[threadIdx.x] = 0;
  __syncthreads();
  const int64_t s = s_begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s < s_end) {
    const int L = 63 - __clzll((unsigned long long)s);
    const int64_t i = s - ((int64_t)1 << L);
    if (i > 0) {
      const double* bx = lev + 4 * cap;
      const double* by = lev + 5 * cap;
      const double* bz = lev + 6 * cap;
      const double dx = __dsub_rn(bx[s], bx[s - 1]), dy = __dsub_rn(by[s], by[s - 1]), dz = __dsub_rn(bz[s], bz[s - 1]);
      const double d = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz)));
      atomicMax(&blk[L & 31], (unsigned long long)__double_as_longlong(d));
    }
  }
  __syncthreads();
  if (threadIdx.x < 32 && blk[threadIdx.x]) atomicMax(&bdmax_bits[threadIdx.x], blk[threadIdx.x]);
}

// ---------------------------------------------------------------------------------------------
// Shared-memory staging of sample ranges.
// ---------------------------------------------------------------------------------------------
template <int NARR, int CH>
struct Stage {
  // CH + 2 slots so that a range whose start is rounded down to an even index still fits.
  double v[2][NARR][CH + 2];
  uint64_t bar[2];
};

// Issue the bulk copies of samples [lo_al, hi_al) of the NARR arrays into buffer `b`.
template <int NARR, int CH>
__device__ __forceinline__ void stage_issue(Stage<NARR, CH>& st, int b, const double* lev, int64_t cap,
                                            int64_t lo_al, int64_t hi_al) {
  const uint32_t bytes = (uint32_t)((hi_al - lo_al) * sizeof(double));
  mbar_arrive_expect_tx(&st.bar[b], bytes * NARR);
#pragma unroll
  for (int k = 0; k < NARR; ++k) tma_load_1d(&st.v[b][k][0], lev + k * cap + lo_al, bytes, &st.bar[b]);
}

// ---------------------------------------------------------------------------------------------
// Frequency-domain wave (flux / spectrum).  Integrand: src/OSCARSSR.cc:4202-4220 (flux) and
// :1976-1989 (spectrum), both
//   [ (1-b^2)(n-b) / (D^2 (1-n.b)^2) + n x ((n-b) x a/c) / (D (1-n.b)^2) ] exp(-i w (t + D/c)).
// ---------------------------------------------------------------------------------------------
constexpr int kFdThreads = 128;
constexpr int kFdChunk = 128;

// Sample-split FP64 sum: the CTA's 128 threads form SUB groups of TE = 128 / SUB threads, one entry
// per thread; group g takes the g-th of SUB equal parts of every staged chunk of the 10 level arrays.
// Each part starts from the phase of the sample before it (the chunk's previous sample, the previous
// chunk's last one, or the span's predecessor read from the level cache), so the phase steps of a
// span cover exactly the consecutive pairs of the serial order and spans need no joining; the stop
// rule only asks whether a step reaches pi, so a span stores pi or 0 in the place of its largest
// step.  The groups' sums are combined in shared memory in group order.  Fused waves finalize their tiles with all threads (fused_unit_done_grouped); unfused waves store
// entry-major partials for k_fd_finalize.
//
// Bound by the FP64 pipe: 95 instructions per (entry, sample) at one per two cycles and
// sub-partition, 71 % of its cycles busy in the first wave of a 201 x 201 map (with the library's
// divisions, square root and sincos: ~165 instructions at 64 %).  1 - b^2 depends on the sample
// alone and is formed once per staged chunk.  What a unit waits for before its first sample is
// requested early: the next unit's number at the start of this one, its first chunk during this one's
// last, the span's predecessor before the observer.
template <int SUB, int MINB>
__global__ void __launch_bounds__(kFdThreads, MINB) k_fd_wave_fp64(FdWaveArgs A) {
  constexpr int TE = kFdThreads / SUB;
  if (A.tile_entries != TE) {  // the host sized the partials for another tile
    if (threadIdx.x == 0) atomicOr(A.err, kErrPlan);
    return;
  }
  __shared__ __align__(16) Stage<10, kFdChunk> st;
  __shared__ double ob2[kFdChunk + 2];
  __shared__ double red[SUB > 1 ? SUB - 1 : 1][7][TE];
  __shared__ int s_last;
  __shared__ int64_t next_unit;
  // the plan is uniform over the CTA; keeping it in shared memory frees the registers its
  // fields would otherwise hold across the sample loop
  __shared__ WavePlan P;
  const int tid = threadIdx.x;
  const int grp = tid / TE, q = tid % TE;
  launch_dependents();
  if (tid == 0) {
    mbar_init(&st.bar[0], 1);
    mbar_init(&st.bar[1], 1);
    fence_barrier_init();
  }
  wait_predecessor();
  if (A.fused && blockIdx.x == 0 && tid == 0) {  // counters of the following wave
    if (A.zero_u32) *A.zero_u32 = 0;
    if (A.zero_u64) *A.zero_u64 = 0;
  }
  const int64_t n_act = A.act ? (int64_t)*A.n_act : A.n_items;
  if (tid == 0) P = wave_plan(A.first, A.level, n_act, TE, A.target_units, A.min_span);
  __syncthreads();
  // units (tile, segment, span), spans fastest: the first is the CTA's own, the others come from a
  // shared counter until the wave's units run out
  const int64_t units = (P.tiles * P.nseg) << P.log2_spans;
  auto unit_range = [&](int64_t u, int64_t& b0, int64_t& b1) {
    const int64_t r = u >> P.log2_spans;
    const int g = P.nseg == 2 ? (int)(r & 1) : 0;
    b0 = seg_begin(P, g) + (u & (P.spans - 1)) * seg_span(P, g);
    b1 = min(seg_end(P, g), b0 + seg_span(P, g));
  };
  auto issue = [&](int64_t lo, int64_t end, int b) {  // chunk [lo, lo + kFdChunk) of a range ending at end
    const int64_t hi = min(end, lo + kFdChunk);
    stage_issue<10, kFdChunk>(st, b, A.lev, A.cap, lo & ~(int64_t)1, (hi + 1) & ~(int64_t)1);
  };
  uint32_t staged = 0;  // chunks taken so far: buffer staged & 1, its completion parity (staged >> 1) & 1
  int64_t u = blockIdx.x;
  if (tid == 0 && u < units) {
    int64_t b0, b1;
    unit_range(u, b0, b1);
    if (b0 < b1) issue(b0, b1, 0);
  }
  while (u < units) {
    int64_t after = 0;
    if (tid == 0) after = (int64_t)gridDim.x + (int64_t)atomicAdd(A.work, 1ull);
    int64_t b0, b1;
    unit_range(u, b0, b1);
    const int64_t nchunks = b1 > b0 ? (b1 - b0 + kFdChunk - 1) / kFdChunk : 0;
    const int span = (int)u & (P.spans - 1);
    const int g = P.nseg == 2 ? (int)(u >> P.log2_spans) & 1 : 0;
    const int64_t tile = u >> (P.log2_spans + P.nseg - 1);
    // the sample before the span (sample 0, the unused slot, never is one)
    const bool joins = span > 0 && nchunks > 0 && b0 - 1 >= 1;
    double cT = 0, cX = 0, cY = 0, cZ = 0;
    if (joins) {
      const double* c = A.lev + (b0 - 1);
      cT = c[0]; cX = c[A.cap]; cY = c[2 * A.cap]; cZ = c[3 * A.cap];
    }
    const int64_t slot = tile * TE + q;
    const bool live = slot < n_act;
    const unsigned item = live ? (A.act ? (unsigned)A.act[slot] : (unsigned)slot) : 0u;
    const unsigned io = item / (unsigned)A.n_e, ie = item - io * (unsigned)A.n_e;
    const double* ob = A.obs + 3 * (int64_t)io;
    const double Ox = ob[0], Oy = ob[1], Oz = ob[2];
    const double mw = -A.omega[ie];
    const bool near = phase_reach(A, Ox, Oy, Oz, mw) < kPhaseFast;  // (false for NaN)
    // phase of the sample before a part that starts a chunk: the span's predecessor, then the previous
    // chunk's last sample (NaN: no step into the segment's first sample)
    double carry = __longlong_as_double(0x7ff8000000000000ll);
    if (joins) carry = fd_phase(cT, cX, cY, cZ, Ox, Oy, Oz, mw);
    double sxr = 0, sxi = 0, syr = 0, syi = 0, szr = 0, szi = 0;
    bool wide = false;  // a phase step of pi or more
    bool any = false;
    for (int64_t c = 0; c < nchunks; ++c, ++staged) {
      const int buf = (int)(staged & 1u);
      const int64_t lo = b0 + c * kFdChunk, hi = min(b1, lo + kFdChunk);
      if (tid == 0) {  // the chunk after this one, of this unit or the next, into the other buffer
        if (c + 1 < nchunks) {
          issue(lo + kFdChunk, b1, buf ^ 1);
        } else if (after < units) {
          int64_t n0, n1;
          unit_range(after, n0, n1);
          if (n0 < n1) issue(n0, n1, buf ^ 1);
        }
      }
      if (!mbar_wait(&st.bar[buf], (staged >> 1) & 1u)) {
        if (tid == 0) atomicOr(A.err, kErrTmaTimeout);
        return;
      }
      const int64_t lo_al = lo & ~(int64_t)1;
      const double* sT = st.v[buf][0];
      const double* sX = st.v[buf][1];
      const double* sY = st.v[buf][2];
      const double* sZ = st.v[buf][3];
      const double* sBx = st.v[buf][4];
      const double* sBy = st.v[buf][5];
      const double* sBz = st.v[buf][6];
      const double* sAx = st.v[buf][7];
      const double* sAy = st.v[buf][8];
      const double* sAz = st.v[buf][9];
      const int ja = (int)(max(lo, (int64_t)1) - lo_al);  // sample 0 is the unused slot
      const int jb = (int)(hi - lo_al);
      const int j0 = ja + ((jb - ja) * grp) / SUB, j1 = ja + ((jb - ja) * (grp + 1)) / SUB;  // this group's part
      for (int j = tid; j < jb; j += kFdThreads) ob2[j] = one_minus_b2(sBx[j], sBy[j], sBz[j]);
      __syncthreads();
      if (live && j0 < j1) {
        double last = carry;
        if (j0 > ja) last = fd_phase(sT[j0 - 1], sX[j0 - 1], sY[j0 - 1], sZ[j0 - 1], Ox, Oy, Oz, mw);
        auto sum = [&](auto trig) {
#pragma unroll 2
          for (int j = j0; j < j1; ++j) {
            const FdTerm f = fd_term(sT[j], sX[j], sY[j], sZ[j], sBx[j], sBy[j], sBz[j], sAx[j], sAy[j], sAz[j], ob2[j],
                                     Ox, Oy, Oz);
            const double ph = __dmul_rn(mw, f.tau);
            wide |= fabs(__dsub_rn(ph, last)) >= kPiD;
            last = ph;
            double sn, cs;
            trig(ph, &sn, &cs);
            sxr = fma(f.ex, cs, sxr); sxi = fma(f.ex, sn, sxi);
            syr = fma(f.ey, cs, syr); syi = fma(f.ey, sn, syi);
            szr = fma(f.ez, cs, szr); szi = fma(f.ez, sn, szi);
          }
        };
        if (near) sum([](double ph, double* sn, double* cs) { sincos_fast(ph, sn, cs); });
        else sum([](double ph, double* sn, double* cs) { sincos_far(ph, sn, cs); });
        any = true;
      }
      if (live && c + 1 < nchunks) {  // a full chunk: its last sample precedes the next chunk
        const int jl = jb - 1;
        carry = fd_phase(sT[jl], sX[jl], sY[jl], sZ[jl], Ox, Oy, Oz, mw);
      }
      __syncthreads();  // everyone is done with `buf` before it is refilled
    }
    if (nchunks == 0) {  // (no unit of a planned wave is empty)
      if (tid == 0 && after < units) {
        int64_t n0, n1;
        unit_range(after, n0, n1);
        if (n0 < n1) issue(n0, n1, (int)(staged & 1u));
      }
      __syncthreads();
    }
    // combine the groups' sums in group order; group 0 stores the span's partial
    double S[6] = {sxr, sxi, syr, syi, szr, szi};
    double dm = any ? (wide ? kPiD : 0.0) : -1.0;
    if (SUB > 1) {
      if (grp > 0) {
#pragma unroll
        for (int k = 0; k < 6; ++k) red[grp - 1][k][q] = S[k];
        red[grp - 1][6][q] = dm;
      }
      __syncthreads();
      if (grp == 0)
        for (int o = 0; o < SUB - 1; ++o) {
#pragma unroll
          for (int k = 0; k < 6; ++k) S[k] += red[o][k][q];
          dm = fmax(dm, red[o][6][q]);
        }
    }
    if (live && grp == 0) {
      // entry-major for the finalize kernel (an entry's spans contiguous); tile-major when fused
      double* p = A.fused ? A.part + fused_part_index(P, tile, g, span, 0, q, TE)
                          : A.part + (slot * P.nseg * P.spans + g * P.spans + span) * kFdPartials;
      const int64_t cs = A.fused ? TE : 1;  // stride between components
#pragma unroll
      for (int k = 0; k < 6; ++k) p[k * cs] = S[k];
      if (!A.fused) p[6] = p[7] = 0.0;  // no step left to join between spans
      p[8 * cs] = dm;  // -1 marks an empty span
    }
    if (tid == 0) next_unit = after;
    if (A.fused) fused_unit_done_grouped<kFdThreads>(A, P, tile, n_act, &s_last, TE, &red[0][0][0], P.nseg * P.spans);
    else __syncthreads();
    u = next_unit;
  }
}

// Reduce the span partials of the wave, apply the stop rule of src/OSCARSSR.cc:4222-4238, finish
// converged / last-level entries (:4246-4267) and append the others to the next active list
// (span partials reduced by kFinLanes-lane groups, fd_common.cuh).

__global__ void k_fd_finalize(FdFinalArgs A) {
  if (blockIdx.x == 0 && threadIdx.x == 0 && A.work_reset) *A.work_reset = 0;
  const int64_t n_act = A.act ? (int64_t)*A.n_act : A.n_items;
  const int lane = threadIdx.x % kFinLanes;
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kFinLanes;
  if ((int64_t)blockIdx.x * blockDim.x / kFinLanes >= n_act) return;  // whole block idle
  const bool live = slot < n_act;
  const WavePlan P = wave_plan(A.first, A.level, n_act, A.tile_entries, A.target_units, A.min_span);
  const int64_t item = live ? (A.act ? (int64_t)A.act[slot] : slot) : 0;
  // sums and max phase step of segment g over this lane's spans, then over the group
  auto seg_sum = [&](int g, C3& s, double& dmax) {
    C3 t = {0, 0, 0, 0, 0, 0};
    double dm = 0;
    if (live) {
      const double* base = A.part + (slot * P.nseg * P.spans + g * P.spans) * kFdPartials;
      for (int sp = lane; sp < P.spans; sp += kFinLanes) {
        const double* p = base + sp * kFdPartials;
        t.xr += p[0]; t.xi += p[1]; t.yr += p[2]; t.yi += p[3]; t.zr += p[4]; t.zi += p[5];
        if (p[8] >= 0) {  // non-empty span (empty spans only trail the segment)
          dm = fmax(dm, p[8]);
          if (sp > 0) dm = fmax(dm, fabs(__dsub_rn(p[6], p[-kFdPartials + 7])));
        }
      }
    }
    s.xr += group_sum(t.xr); s.xi += group_sum(t.xi); s.yr += group_sum(t.yr);
    s.yi += group_sum(t.yi); s.zr += group_sum(t.zr); s.zi += group_sum(t.zi);
    dmax = fmax(dmax, group_max(dm));
  };
  const int64_t N = A.n_items;
  C3 S = {0, 0, 0, 0, 0, 0};
  double last_mag = -1;
  double dmax = 0;
  if (A.first) {
    double unused = 0;
    if (P.nseg == 2) {
      seg_sum(0, S, unused);
      C3 t = c3_scale(S, A.dt_prev);
      if (A.project) t = c3_project(t, A.pol);
      last_mag = c3_mag2(t);
    }
    seg_sum(P.nseg - 1, S, dmax);
  } else {
    if (live) {
      S = {A.state[item], A.state[N + item], A.state[2 * N + item], A.state[3 * N + item], A.state[4 * N + item],
           A.state[5 * N + item]};
      last_mag = A.state[6 * N + item];
    }
    seg_sum(0, S, dmax);
  }
  bool finished = false, unconverged = false, survive = false;
  if (live && lane == 0) fd_entry_decide(A, item, S, last_mag, dmax, finished, unconverged, survive);
  finalize_bookkeeping(finished, unconverged, survive, item, A.level, A.act_next, A.n_next, A.not_converged, A.samples,
                       A.level_max);
}

// ---------------------------------------------------------------------------------------------
// Power density (src/OSCARSSR.cc:2869-2922):
//   sum += [(N1 x ((N1 - b) x a/c)) . Nk]^2 / (1 - b.N1)^5 / |O - X|^2 * (N1 . normal),  k = 2, 3
// The term is pd_term (fd_common.cuh); N1 . normal, whose sign is the directional cut, rounds as the
// reference's operations do.
// Sample-split and fused like the flux waves; 67 FP64 instructions per (entry, sample) (with the
// library's square root and four divisions: ~130, a separate finalize launch and 128 entries per CTA).
// ---------------------------------------------------------------------------------------------
constexpr int kPdThreads = 128;
constexpr int kPdChunk = 128;
constexpr int kPdSub = 4;                       // groups of a CTA
constexpr int kPdTile = kPdThreads / kPdSub;    // entries per CTA

template <bool NORMAL, bool DIRECTIONAL>
__device__ __forceinline__ double pd_sample(double X, double Y, double Z, double bx, double by, double bz, double ax,
                                            double ay, double az, double Ox, double Oy, double Oz, double Nx, double Ny,
                                            double Nz) {
  const double Rx = __dsub_rn(Ox, X), Ry = __dsub_rn(Oy, Y), Rz = __dsub_rn(Oz, Z);
  const double s = __dadd_rn(__dadd_rn(__dmul_rn(Rx, Rx), __dmul_rn(Ry, Ry)), __dmul_rn(Rz, Rz));
  const double y = rsqrt_near(s), D = sqrt_by(s, y);
  const double nx = quot_by(Rx, D, y), ny = quot_by(Ry, D, y), nz = quot_by(Rz, D, y);
  const double t = pd_term(nx, ny, nz, y, bx, by, bz, ax, ay, az);
  if (!NORMAL) return t;
  const double n1dn = __dadd_rn(__dadd_rn(__dmul_rn(nx, Nx), __dmul_rn(ny, Ny)), __dmul_rn(nz, Nz));
  return DIRECTIONAL && n1dn <= 0 ? 0.0 : t * n1dn;
}

__global__ void __launch_bounds__(kPdThreads, 5) k_pd_wave_fp64(PdWaveArgs A) {
  constexpr int TE = kPdTile, SUB = kPdSub;
  if (A.tile_entries != TE) {  // the host sized the partials for another tile
    if (threadIdx.x == 0) atomicOr(A.err, kErrPlan);
    return;
  }
  __shared__ __align__(16) Stage<9, kPdChunk> st;  // x y z beta a/c: the times are not needed
  __shared__ double red[SUB - 1][TE];
  __shared__ WavePlan P;
  __shared__ int64_t next_unit;
  __shared__ int s_last;
  const int tid = threadIdx.x;
  const int grp = tid / TE, q = tid % TE;
  launch_dependents();
  if (tid == 0) {
    mbar_init(&st.bar[0], 1);
    mbar_init(&st.bar[1], 1);
    fence_barrier_init();
  }
  wait_predecessor();
  if (blockIdx.x == 0 && tid == 0) {  // counters of the following wave
    if (A.zero_u32) *A.zero_u32 = 0;
    if (A.zero_u64) *A.zero_u64 = 0;
  }
  const int64_t n_act = A.act ? (int64_t)*A.n_act : A.n_items;
  if (tid == 0) P = wave_plan(A.first, A.level, n_act, TE, A.target_units, A.min_span);
  __syncthreads();
  // units (tile, segment, span) and their early requests as in k_fd_wave_fp64
  const int64_t units = (P.tiles * P.nseg) << P.log2_spans;
  auto unit_range = [&](int64_t u, int64_t& b0, int64_t& b1) {
    const int64_t r = u >> P.log2_spans;
    const int g = P.nseg == 2 ? (int)(r & 1) : 0;
    b0 = seg_begin(P, g) + (u & (P.spans - 1)) * seg_span(P, g);
    b1 = min(seg_end(P, g), b0 + seg_span(P, g));
  };
  auto issue = [&](int64_t lo, int64_t end, int b) {
    const int64_t hi = min(end, lo + kPdChunk);
    stage_issue<9, kPdChunk>(st, b, A.lev + A.cap, A.cap, lo & ~(int64_t)1, (hi + 1) & ~(int64_t)1);
  };
  uint32_t staged = 0;
  int64_t u = blockIdx.x;
  if (tid == 0 && u < units) {
    int64_t b0, b1;
    unit_range(u, b0, b1);
    if (b0 < b1) issue(b0, b1, 0);
  }
  while (u < units) {
    int64_t after = 0;
    if (tid == 0) after = (int64_t)gridDim.x + (int64_t)atomicAdd(A.work, 1ull);
    int64_t b0, b1;
    unit_range(u, b0, b1);
    const int64_t nchunks = b1 > b0 ? (b1 - b0 + kPdChunk - 1) / kPdChunk : 0;
    const int span = (int)u & (P.spans - 1);
    const int g = P.nseg == 2 ? (int)(u >> P.log2_spans) & 1 : 0;
    const int64_t tile = u >> (P.log2_spans + P.nseg - 1);
    const int64_t slot = tile * TE + q;
    const bool live = slot < n_act;
    const int64_t item = live ? (A.act ? (int64_t)A.act[slot] : slot) : 0;
    const double Ox = A.obs[3 * item], Oy = A.obs[3 * item + 1], Oz = A.obs[3 * item + 2];
    double Nx = 0, Ny = 0, Nz = 0;
    if (A.has_normal) { Nx = A.normals[3 * item]; Ny = A.normals[3 * item + 1]; Nz = A.normals[3 * item + 2]; }
    double sum = 0;
    for (int64_t c = 0; c < nchunks; ++c, ++staged) {
      const int buf = (int)(staged & 1u);
      const int64_t lo = b0 + c * kPdChunk, hi = min(b1, lo + kPdChunk);
      if (tid == 0) {
        if (c + 1 < nchunks) {
          issue(lo + kPdChunk, b1, buf ^ 1);
        } else if (after < units) {
          int64_t n0, n1;
          unit_range(after, n0, n1);
          if (n0 < n1) issue(n0, n1, buf ^ 1);
        }
      }
      if (!mbar_wait(&st.bar[buf], (staged >> 1) & 1u)) {
        if (tid == 0) atomicOr(A.err, kErrTmaTimeout);
        return;
      }
      const int64_t lo_al = lo & ~(int64_t)1;
      const int ja = (int)(max(lo, (int64_t)1) - lo_al), jb = (int)(hi - lo_al);  // sample 0 is the unused slot
      const int j0 = ja + ((jb - ja) * grp) / SUB, j1 = ja + ((jb - ja) * (grp + 1)) / SUB;  // this group's part
      auto add = [&](auto normal, auto directional) {
#pragma unroll 2
        for (int j = j0; j < j1; ++j)
          sum += pd_sample<normal.value, directional.value>(
              st.v[buf][0][j], st.v[buf][1][j], st.v[buf][2][j], st.v[buf][3][j], st.v[buf][4][j], st.v[buf][5][j],
              st.v[buf][6][j], st.v[buf][7][j], st.v[buf][8][j], Ox, Oy, Oz, Nx, Ny, Nz);
      };
      if (live) {
        if (A.has_normal && A.directional) add(std::true_type{}, std::true_type{});
        else if (A.has_normal) add(std::true_type{}, std::false_type{});
        else add(std::false_type{}, std::false_type{});
      }
      __syncthreads();  // everyone is done with `buf` before it is refilled
    }
    if (nchunks == 0) {  // (no unit of a planned wave is empty)
      if (tid == 0 && after < units) {
        int64_t n0, n1;
        unit_range(after, n0, n1);
        if (n0 < n1) issue(n0, n1, (int)(staged & 1u));
      }
      __syncthreads();
    }
    // the groups' sums in group order; group 0 stores the span's partial
    if (grp > 0) red[grp - 1][q] = sum;
    __syncthreads();
    if (grp == 0 && live) {
      for (int o = 0; o < SUB - 1; ++o) sum += red[o][q];
      A.part[((tile * P.nseg + g) * P.spans + span) * TE + q] = sum;
    }
    if (tid == 0) next_unit = after;
    pd_unit_done(A, P, tile, n_act, &s_last, TE, P.nseg * P.spans);
    u = next_unit;
  }
}

}  // namespace dev

// ---- launch wrappers ------------------------------------------------------------------------
cudaError_t launch_level_fill(const double* knots, int64_t n, double tstart, double tstop, int64_t s_begin,
                              int64_t s_end, double* lev, int64_t cap, int ext_from,
                              unsigned long long* bdmax_bits, cudaStream_t st) {
  if (s_end <= s_begin) return cudaSuccess;
  const int T = 256;
  const int64_t nblk = (s_end - s_begin + T - 1) / T;
  dev::k_level_fill<<<(unsigned)nblk, T, 0, st>>>(knots, n, tstart, tstop, s_begin, s_end, lev, cap, ext_from);
  dev::k_level_betadiff<<<(unsigned)nblk, T, 0, st>>>(lev, cap, s_begin, s_end, bdmax_bits);
  return cudaGetLastError();
}

// Compiled variants of the FP64 wave kernel: groups SUB of 128 / SUB entries, minimum CTAs per SM.
// Variant 0 keeps 128 entries per CTA (the allocation-free entry point sizes its partials for it); the
// others trade registers for resident warps (132, 122 and 80 a thread): 3 to 6 CTAs measured within 3 %
// of each other on a 201 x 201 map, fewer the better on small grids, so the autotuner chooses.
#define OSC_FP64_VARIANTS(X) \
  X(0, 1, 7)                 \
  X(1, 4, 3)                 \
  X(2, 4, 4)                 \
  X(3, 4, 6)

#define OSC_SUB(i, sub, minb) sub,
static const int kFp64Sub[kFp64Variants] = {OSC_FP64_VARIANTS(OSC_SUB)};

int fp64_entries_per_cta(int variant) { return dev::kFdThreads / kFp64Sub[variant]; }
const char* fp64_variant_name(int variant) {
#define OSC_NAME(i, sub, minb) "k_fd_wave_fp64<" #sub "," #minb ">",
  static const char* const kNames[kFp64Variants] = {OSC_FP64_VARIANTS(OSC_NAME)};
  return variant >= 0 && variant < kFp64Variants ? kNames[variant] : "";
}

cudaError_t launch_fd_wave_fp64(const FdWaveArgs& a, int grid, int variant, cudaStream_t st) {
  switch (variant) {
#define OSC_LAUNCH(i, sub, minb) \
    case i: return launch_overlapped(dev::k_fd_wave_fp64<sub, minb>, grid, dev::kFdThreads, st, a);
    OSC_FP64_VARIANTS(OSC_LAUNCH)
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_fd_finalize(const FdFinalArgs& a, int64_t n_act_bound, cudaStream_t st) {
  if (n_act_bound == 0) return cudaSuccess;
  const int T = 256;
  const int64_t threads = n_act_bound * dev::kFinLanes;
  dev::k_fd_finalize<<<(unsigned)((threads + T - 1) / T), T, 0, st>>>(a);
  return cudaGetLastError();
}

int pd_fp64_entries_per_cta() { return dev::kPdTile; }
cudaError_t launch_pd_wave_fp64(const PdWaveArgs& a, int grid, cudaStream_t st) {
  return launch_overlapped(dev::k_pd_wave_fp64, grid, dev::kPdThreads, st, a);
}

int fp64_blocks_per_sm(bool power_density, int variant) {
  int n = 0;
  if (power_density) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dev::k_pd_wave_fp64, dev::kPdThreads, 0);
  } else {
    switch (variant) {
#define OSC_OCC(i, sub, minb) \
      case i: cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dev::k_fd_wave_fp64<sub, minb>, dev::kFdThreads, 0); break;
      OSC_FP64_VARIANTS(OSC_OCC)
    }
  }
  return n > 0 ? n : 1;
}

}  // namespace osc
