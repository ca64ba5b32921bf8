// kernels_stl.cu -- power density on the facets of STL meshes (src/OSCARSSR.cc:3318-3521, the
// reference's Mode 2): for each facet i, the level samples whose ray to the facet centre crosses any
// other facet j (TTriangle3D::RayIntersectionDistance, src/TTriangle3D.cc, Moller-Trumbore) are
// skipped; the others add the power-density integrand with |N1 . normal|, and the beta-difference
// stop criterion runs over the visible samples only (src/OSCARSSR.cc:3446-3451).
//
// Waves: the first holds levels 0..9 (no facet stops before), one CTA a facet; each later one a level of the
// facets left, split into spans.  A CTA first drops the facets that cannot stand between its centre and any sample
// (stl_clear: the barycentric coordinates of the ray's crossing are ratios of functions linear in the
// sample's position, so their ranges over the samples' bounding box are exact up to rounding); testing
// every pair for every sample was all of the time before (514 facets: 2.7 ms of launches, of which
// 0.07 ms remain).  The threads then take the samples in chunks of kStlThreads (sample order = thread
// order inside a chunk), test each against the facets left, and find each visible sample's predecessor
// among the visible ones (warp ballot, then the previous warps' last visible samples, then the previous
// chunks') for the beta differences.  Sums are reduced in a fixed order; the stop rule
// (src/OSCARSSR.cc:3483-3497) is applied by thread 0 on the facet's running state.  The ray tests and
// the beta differences round as the reference's operations do, so the shadowing decisions are the
// reference's exactly; a term's well-conditioned rest is formed as in the power-density wave (fd_common.cuh).
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "fd_common.cuh"
#include "kernels.h"

namespace osc {
namespace dev {

constexpr int kStlThreads = 256;
constexpr int kStlTile = 64;     // facets staged in shared memory per pass (9 doubles each)
constexpr int kStlCand = 1024;   // facets a CTA keeps after the cull; more: it tests them all

struct D3 {
  double x, y, z;
};
__device__ __forceinline__ D3 d3(double x, double y, double z) { return {x, y, z}; }
__device__ __forceinline__ D3 sub3(D3 a, D3 b) { return {__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y), __dsub_rn(a.z, b.z)}; }
__device__ __forceinline__ double dot3(D3 a, D3 b) {
  return __dadd_rn(__dadd_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)), __dmul_rn(a.z, b.z));
}
__device__ __forceinline__ D3 cross3(D3 a, D3 b) {  // TVector3D::Cross
  return {__dsub_rn(__dmul_rn(a.y, b.z), __dmul_rn(b.y, a.z)), __dsub_rn(__dmul_rn(a.z, b.x), __dmul_rn(b.z, a.x)),
          __dsub_rn(__dmul_rn(a.x, b.y), __dmul_rn(b.x, a.y))};
}
__device__ __forceinline__ double mag3(D3 a) { return __dsqrt_rn(dot3(a, a)); }
// TVector3D::UnitVector, componentwise division by Mag(), which goes to *mag (its reciprocal to *inv)
__device__ __forceinline__ D3 unit3v(D3 a, double* mag, double* inv = nullptr) {
  const double s = dot3(a, a), y = rsqrt_near(s), m = sqrt_by(s, y);
  *mag = m;
  if (inv) *inv = y;
  return {quot_by(a.x, m, y), quot_by(a.y, m, y), quot_by(a.z, m, y)};
}

// TTriangle3D::RayIntersectionDistance for a facet given as its vertex A and edges B - A, C - A
// (f[0..8]); `dir` is the ray direction, normalised again from the direction passed as the reference does.
__device__ __forceinline__ double ray_distance(const double* f, D3 origin, D3 dir) {
  const D3 A = d3(f[0], f[1], f[2]), e1 = d3(f[3], f[4], f[5]), e2 = d3(f[6], f[7], f[8]);
  const D3 pvec = cross3(dir, e2);
  const double det = dot3(e1, pvec);
  if (det > -1e-12 && det < 1e-12) return -1;
  const double inv_det = __drcp_rn(det);
  const D3 tvec = sub3(origin, A);
  const double u = __dmul_rn(dot3(tvec, pvec), inv_det);
  if (u < 0.0 || u > 1.0) return -1;
  const D3 qvec = cross3(tvec, e1);
  const double v = __dmul_rn(dot3(dir, qvec), inv_det);
  if (v < 0.0 || __dadd_rn(u, v) > 1.0) return -1;
  const double t = __dmul_rn(dot3(e2, qvec), inv_det);
  if (t < 0) return -1;
  return t;
}


// Whether facet f (vertex A, edges e1, e2) is clear of every ray from a sample in the box mid +- half to
// centre C.  With P = X - C, the crossing's barycentric coordinates are u = N_u / det, v = N_v / det,
//   det = P.(e1 x e2),  N_u = P.((C - A) x e2),  N_v = P.(e1 x (C - A))     (times 1 / |P|),
// all linear in P, so a box's range of each is its value at the middle +- |normal|.half.  The facet is
// clear when det keeps one sign and, with it, u < 0, v < 0 or u + v > 1 everywhere, by more than the
// roundings of the test itself (its sums of products of |tvec| |e2|, |dir| = 1) and of these ranges.
__device__ __forceinline__ bool stl_clear(const double* f, D3 C, D3 mid, D3 half) {
  const D3 e1 = d3(f[3], f[4], f[5]), e2 = d3(f[6], f[7], f[8]);
  const D3 a = d3(C.x - f[0], C.y - f[1], C.z - f[2]);
  const D3 p = d3(mid.x - C.x, mid.y - C.y, mid.z - C.z);
  auto cross = [](D3 q, D3 r) { return d3(q.y * r.z - q.z * r.y, q.z * r.x - q.x * r.z, q.x * r.y - q.y * r.x); };
  auto range = [&](D3 n, double& lo, double& hi) {
    const double c = n.x * p.x + n.y * p.y + n.z * p.z;
    const double h = fabs(n.x) * half.x + fabs(n.y) * half.y + fabs(n.z) * half.z;
    lo = c - h;
    hi = c + h;
  };
  const D3 nd = cross(e1, e2), nu = cross(a, e2), nv = cross(e1, a);
  const D3 nw = d3(nu.x + nv.x - nd.x, nu.y + nv.y - nd.y, nu.z + nv.z - nd.z);
  double dl, dh, ul, uh, vl, vh, wl, wh;
  range(nd, dl, dh);
  range(nu, ul, uh);
  range(nv, vl, vh);
  range(nw, wl, wh);
  // |P| and |X - A| at most, then the roundings' reach: 1e-12 is 4500 units in the last place
  const double r = fabs(p.x) + half.x + fabs(p.y) + half.y + fabs(p.z) + half.z;
  const double ra = r + fabs(a.x) + fabs(a.y) + fabs(a.z);
  const double l1 = fabs(e1.x) + fabs(e1.y) + fabs(e1.z), l2 = fabs(e2.x) + fabs(e2.y) + fabs(e2.z);
  const double tol = 1e-12 * r * ((ra + l1) * (l1 + l2) + l1 * l2);
  if (dl > tol) return uh < -tol || vh < -tol || wl > tol;
  if (dh < -tol) return ul > tol || vl > tol || wh < -tol;
  return false;
}

// Before a wave: boxes of the samples [s_begin, s_end), one per block (NaN samples, which block nothing
// and are blocked by nothing, are left out), and the list of the facets not yet done.  With `first` the
// start of a request too: facet geometry from the vertices (A, B - A, C - A as RayIntersectionDistance
// forms them) and normals, states and flags.
__global__ void __launch_bounds__(1024) k_stl_prepare(StlWaveArgs a, int64_t s_begin, int64_t s_end,
                                                      const double* __restrict__ tri, double* __restrict__ geo,
                                                      double* __restrict__ nrm, double* __restrict__ box) {
  const int64_t n = a.n, stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (a.first) {
    for (int64_t i = t0; i < n; i += stride) {
      const double* t = tri + 12 * i;
      for (int c = 0; c < 3; ++c) {
        geo[9 * i + c] = t[c];
        geo[9 * i + 3 + c] = __dsub_rn(t[3 + c], t[c]);
        geo[9 * i + 6 + c] = __dsub_rn(t[6 + c], t[c]);
        nrm[3 * i + c] = t[9 + c];
      }
      a.state[4 * i] = 0;       // sum
      a.state[4 * i + 1] = -1;  // last level value
      a.state[4 * i + 2] = -1;  // result precision
      a.state[4 * i + 3] = 0;   // last level
      a.done[i] = 0;
      a.level_out[i] = -1;
      a.spans_done[i] = 0;
    }
    if (t0 < 32) a.n_active[t0] = 0;
  } else if (blockIdx.x == gridDim.x - 1) {
    // in facet order: the list is the same from run to run
    __shared__ int sums[32], base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    for (int64_t i0 = 0; i0 < n; i0 += blockDim.x) {
      const int64_t i = i0 + threadIdx.x;
      const bool on = i < n && !a.done[i];
      const unsigned m = __ballot_sync(0xffffffffu, on);
      if ((threadIdx.x & 31) == 0) sums[threadIdx.x >> 5] = __popc(m);
      __syncthreads();
      int at = base;
      for (int w = 0; w < (int)(threadIdx.x >> 5); ++w) at += sums[w];
      if (on) a.act[at + __popc(m & ((1u << (threadIdx.x & 31)) - 1u))] = (int)i;
      __syncthreads();
      if (threadIdx.x == 0)
        for (int w = 0; w < (int)blockDim.x / 32; ++w) base += sums[w];
      __syncthreads();
    }
    if (threadIdx.x == 0) *a.n_act = base;
  }
  __shared__ double red[6][32];
  double v[6] = {1e300, 1e300, 1e300, -1e300, -1e300, -1e300};
  for (int64_t s = s_begin + t0; s < s_end; s += stride)
    for (int c = 0; c < 3; ++c) {
      const double x = a.lev[(1 + c) * a.cap + s];
      v[c] = fmin(v[c], x);
      v[3 + c] = fmax(v[3 + c], x);
    }
  for (int c = 0; c < 6; ++c) {
    for (int o = 16; o > 0; o >>= 1) {
      const double w = __shfl_xor_sync(0xffffffffu, v[c], o);
      v[c] = c < 3 ? fmin(v[c], w) : fmax(v[c], w);
    }
    if ((threadIdx.x & 31) == 0) red[c][threadIdx.x >> 5] = v[c];
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    double r = red[threadIdx.x][0];
    for (int w = 1; w < (int)blockDim.x / 32; ++w) r = threadIdx.x < 3 ? fmin(r, red[threadIdx.x][w]) : fmax(r, red[threadIdx.x][w]);
    box[6 * blockIdx.x + threadIdx.x] = r;
  }
}

// src/OSCARSSR.cc:3483-3500 on facet i's running state: `before` its sum below level L, `last` that level's
// value, `add` and bdm the level's own sum and largest beta step.
__device__ __forceinline__ void stl_decide(const StlWaveArgs& a, int64_t i, double before, double last, double add,
                                           double bdm) {
  double* S = a.state + 4 * i;  // [0] sum, [1] last level value, [2] result precision, [3] last level
  const int L = a.level;
  const double sum = __dadd_rn(before, add);
  const double ts = __dmul_rn(sum, a.dt_level);
  double prec = fabs(__dsub_rn(ts, last)) / last;
  bool done = false;
  if ((L > 8 && prec < a.precision && bdm < a.two_over_gamma) || (L > 8 && bdm < a.two_over_gamma && ts == last)) {
    done = true;
  } else if (L > 8 && ts == last) {
    done = true;
    prec = 0;
  }
  S[0] = sum;
  S[2] = prec;
  S[3] = (double)L;
  if (done) {
    a.done[i] = 1;
    a.level_out[i] = L;
  } else {
    S[1] = ts;
    atomicAdd(a.n_active + L, 1u);
  }
}

// Spans of a level for n_act facets: the first wave has one, a later one a power of two that gives every
// CTA of the grid about four, each at least 2 x kStlThreads samples long.  (One CTA a facet walked a whole
// level before: a facet on a shadow's edge that stops at level 21 took 30 ms at 4 us per 256 samples.)
__device__ __forceinline__ int stl_spans(const StlWaveArgs& a, int64_t n_act) {
  int k = 0;
  while (!a.first && (n_act << k) < 4 * (int64_t)gridDim.x && (((int64_t)1 << a.level) >> (k + 1)) >= 2 * kStlThreads) ++k;
  return 1 << k;
}

__global__ void __launch_bounds__(kStlThreads) k_stl_wave(StlWaveArgs a) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int kWarps = kStlThreads / 32;
  __shared__ double fac[kStlTile][9];
  __shared__ int cand[kStlCand];
  __shared__ int n_cand;
  __shared__ double wlastB[kWarps][3];
  __shared__ int wlast[kWarps];
  __shared__ double carry[3];   // beta of the span's last visible sample so far (Last_Beta)
  __shared__ int carried;       // whether there is one
  __shared__ double firstB[3];  // beta of a later span's first visible sample
  __shared__ double rsum[kStlThreads], rlow[kStlThreads], rmax[kStlThreads];
  __shared__ double box[6];
  __shared__ int s_last;
  const int L = a.level;
  const int64_t ns = (int64_t)1 << L;
  const double* lev = a.lev;
  const int64_t cap = a.cap;
  const int64_t n_act = a.first ? a.n : (int64_t)*a.n_act;
  const int spans = stl_spans(a, n_act);
  const int64_t span_len = ns / spans;
  if (tid < 6) {
    double r = a.box[tid];
    for (int w = 1; w < a.n_box; ++w) r = tid < 3 ? fmin(r, a.box[6 * w + tid]) : fmax(r, a.box[6 * w + tid]);
    box[tid] = r;
  }
  __syncthreads();
  const D3 mid = d3(0.5 * (box[0] + box[3]), 0.5 * (box[1] + box[4]), 0.5 * (box[2] + box[5]));
  const D3 half = d3(0.5 * (box[3] - box[0]), 0.5 * (box[4] - box[1]), 0.5 * (box[5] - box[2]));
  for (int64_t unit = blockIdx.x; unit < n_act * spans; unit += gridDim.x) {
    const int64_t slot = unit / spans;
    const int span = (int)(unit - slot * spans);
    const int64_t i = a.first ? slot : (int64_t)a.act[slot];
    const D3 obs = d3(a.centers[3 * i], a.centers[3 * i + 1], a.centers[3 * i + 2]);
    const D3 normal = d3(a.normals[3 * i], a.normals[3 * i + 1], a.normals[3 * i + 2]);
    if (tid == 0) {
      carry[0] = carry[1] = carry[2] = 0.0;
      carried = 0;
      n_cand = 0;
    }
    __syncthreads();
    // the facets that may stand in a sample's way
    for (int64_t j = tid; j < a.n; j += kStlThreads) {
      if (j == i || stl_clear(a.geometry + 9 * j, obs, mid, half)) continue;
      const int k = atomicAdd(&n_cand, 1);
      if (k < kStlCand) cand[k] = (int)j;
    }
    __syncthreads();
    const bool all = n_cand > kStlCand;
    const int64_t nc = all ? a.n : n_cand;
    auto stage = [&](int64_t j0, int nt) {
      for (int k = tid; k < nt * 9; k += kStlThreads) {
        const int64_t j = all ? j0 + k / 9 : (int64_t)cand[j0 + k / 9];
        fac[k / 9][k % 9] = a.geometry[9 * j + k % 9];
      }
      __syncthreads();
    };
    if (nc <= kStlTile) stage(0, (int)nc);  // a single tile is staged once
    // is the sample at X blocked on its way to the centre, `dist` along `dir`?
    auto blocked_by = [&](bool active, D3 X, D3 dir, double dist) {
      bool blocked = false;
      double unused;
      const D3 dir2 = nc > 0 ? unit3v(dir, &unused) : dir;
      for (int64_t j0 = 0; j0 < nc; j0 += kStlTile) {
        const int nt = (int)min((int64_t)kStlTile, nc - j0);
        if (nc > kStlTile) {
          __syncthreads();
          stage(j0, nt);
        }
        if (active && !blocked)
          for (int k = 0; k < nt; ++k) {
            if (all && j0 + k == i) continue;
            const double d = ray_distance(fac[k], X, dir2);
            if (d > 0 && d < dist) {
              blocked = true;
              break;
            }
          }
      }
      return blocked;
    };
    // one sample's term, |N1 . normal| times the power-density term
    auto term = [&](D3 N1, double y, D3 B, D3 A) {
      return pd_term(N1.x, N1.y, N1.z, y, B.x, B.y, B.z, A.x, A.y, A.z) * fabs(dot3(N1, normal));
    };
    double plow = 0.0, psum = 0.0, bdmax = -1.0;
    if (a.first) {  // the levels below: their sum alone
      for (int64_t base = 1; base < ns; base += kStlThreads) {
        const int64_t s = min(base + tid, ns - 1);
        const bool active = base + tid < ns;
        const D3 X = d3(lev[cap + s], lev[2 * cap + s], lev[3 * cap + s]);
        const D3 to = sub3(obs, X);
        double dist, y;
        const D3 dir = unit3v(to, &dist, &y);
        if (!blocked_by(active, X, dir, dist) && active)
          plow += term(dir, y, d3(lev[4 * cap + s], lev[5 * cap + s], lev[6 * cap + s]),
                       d3(lev[7 * cap + s], lev[8 * cap + s], lev[9 * cap + s]));
      }
    }
    const int64_t it1 = (span + 1) * span_len;
    for (int64_t base = span * span_len; base < it1; base += kStlThreads) {
      const int64_t it = base + tid;  // index of the sample inside the level
      const bool active = it < it1;
      const int64_t s = ns + (active ? it : it1 - 1);
      const D3 X = d3(lev[cap + s], lev[2 * cap + s], lev[3 * cap + s]);
      const D3 B = d3(lev[4 * cap + s], lev[5 * cap + s], lev[6 * cap + s]);
      const D3 to = sub3(obs, X);
      double dist, y;
      const D3 dir = unit3v(to, &dist, &y);
      const bool visible = !blocked_by(active, X, dir, dist) && active;
      // predecessor of each visible sample among the visible ones (Last_Beta of the reference); a later
      // span's first one has its predecessor in an earlier span and waits for the join
      const unsigned m = __ballot_sync(0xffffffffu, visible);
      const unsigned below = m & ((1u << lane) - 1u);
      const int src = below ? 31 - __clz(below) : lane;
      const double pbx = __shfl_sync(0xffffffffu, B.x, src), pby = __shfl_sync(0xffffffffu, B.y, src),
                   pbz = __shfl_sync(0xffffffffu, B.z, src);
      if (lane == 0) wlast[warp] = m ? 31 - __clz(m) : -1;
      if (m && lane == 31 - __clz(m)) {
        wlastB[warp][0] = B.x;
        wlastB[warp][1] = B.y;
        wlastB[warp][2] = B.z;
      }
      __syncthreads();
      if (visible) {
        D3 prev = d3(carry[0], carry[1], carry[2]);
        bool have = carried != 0 || span == 0;  // (the level's first one: the zero vector)
        if (below) {
          prev = d3(pbx, pby, pbz);
          have = true;
        } else {
          int w = warp - 1;
          while (w >= 0 && wlast[w] < 0) --w;
          if (w >= 0) {
            prev = d3(wlastB[w][0], wlastB[w][1], wlastB[w][2]);
            have = true;
          }
        }
        if (have) {
          const double bd = mag3(sub3(B, prev));
          if (it > 0 && bd > bdmax) bdmax = bd;
        } else {
          firstB[0] = B.x;
          firstB[1] = B.y;
          firstB[2] = B.z;
        }
        psum += term(dir, y, B, d3(lev[7 * cap + s], lev[8 * cap + s], lev[9 * cap + s]));
      }
      __syncthreads();
      if (tid == 0) {  // the chunk's last visible sample becomes the carry
        int w = kWarps - 1;
        while (w >= 0 && wlast[w] < 0) --w;
        if (w >= 0) {
          carry[0] = wlastB[w][0];
          carry[1] = wlastB[w][1];
          carry[2] = wlastB[w][2];
          carried = 1;
        }
      }
      __syncthreads();
    }
    auto reduce = [&]() {  // rsum, rlow, rmax over the threads, in a fixed order
      __syncthreads();
      for (int o = kStlThreads / 2; o > 0; o >>= 1) {
        if (tid < o) {
          rsum[tid] = __dadd_rn(rsum[tid], rsum[tid + o]);
          rlow[tid] = __dadd_rn(rlow[tid], rlow[tid + o]);
          rmax[tid] = fmax(rmax[tid], rmax[tid + o]);
        }
        __syncthreads();
      }
    };
    rsum[tid] = psum;
    rlow[tid] = plow;
    rmax[tid] = bdmax;
    reduce();
    if (spans == 1) {
      if (tid == 0) {
        const double before = a.first ? rlow[0] : a.state[4 * i];
        const double last = a.first ? (L >= 1 ? __dmul_rn(before, a.dt_prev) : -1.0) : a.state[4 * i + 1];
        stl_decide(a, i, before, last, rsum[0], rmax[0]);
      }
      __syncthreads();
      continue;
    }
    // the span's sum, largest step, whether it saw anything, and its first and last visible betas
    double* p = a.part + unit * kStlPartials;
    if (tid == 0) {
      p[0] = rsum[0];
      p[1] = rmax[0];
      p[2] = carried ? 1.0 : 0.0;
      for (int c = 0; c < 3; ++c) {
        p[3 + c] = firstB[c];
        p[6 + c] = carry[c];
      }
      __threadfence();
      s_last = atomicAdd(a.spans_done + i, 1u) == (unsigned)(spans - 1);
      if (s_last) __threadfence();
    }
    __syncthreads();
    if (s_last) {  // the CTA of the facet's last span joins them
      const double* f = a.part + slot * spans * kStlPartials;
      double sum = 0, bd = -1.0;
      for (int k = tid; k < spans; k += kStlThreads) {
        const double* q = f + k * kStlPartials;
        sum += __ldcg(q);
        bd = fmax(bd, __ldcg(q + 1));
        if (k > 0 && __ldcg(q + 2) != 0.0) {  // the step into its first visible sample
          int w = k - 1;
          while (w >= 0 && __ldcg(f + w * kStlPartials + 2) == 0.0) --w;
          const double* e = f + (w >= 0 ? w : 0) * kStlPartials + 6;
          const D3 prev = w >= 0 ? d3(__ldcg(e), __ldcg(e + 1), __ldcg(e + 2)) : d3(0.0, 0.0, 0.0);
          const double b = mag3(sub3(d3(__ldcg(q + 3), __ldcg(q + 4), __ldcg(q + 5)), prev));
          if (b > bd) bd = b;
        }
      }
      rsum[tid] = sum;
      rmax[tid] = bd;
      reduce();
      if (tid == 0) {
        stl_decide(a, i, a.state[4 * i], a.state[4 * i + 1], rsum[0], rmax[0]);
        a.spans_done[i] = 0;
      }
    }
    __syncthreads();
  }
}

}  // namespace dev

int stl_box_blocks(int64_t samples) { return (int)std::min<int64_t>(148, std::max<int64_t>(1, samples / 8192)); }

int stl_blocks_per_sm() {
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, dev::k_stl_wave, dev::kStlThreads, 0);
  return n > 0 ? n : 1;
}

cudaError_t launch_stl_prepare(const StlWaveArgs& a, int64_t s_begin, int64_t s_end, const double* tri, double* geo,
                               double* nrm, double* box, cudaStream_t st) {
  dev::k_stl_prepare<<<(unsigned)a.n_box, 1024, 0, st>>>(a, s_begin, s_end, tri, geo, nrm, box);
  return cudaGetLastError();
}

cudaError_t launch_stl_wave(const StlWaveArgs& a, int grid, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  dev::k_stl_wave<<<(unsigned)grid, dev::kStlThreads, 0, st>>>(a);
  return cudaGetLastError();
}

}  // namespace osc
