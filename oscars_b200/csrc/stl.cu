// stl.cu -- host side of the power density on STL facets (src/OSCARSSR.cc:3154-3521): the particle
// loop, the launches of k_stl_wave (kernels_stl.cu) on the FP64 level cache, and the
// per-facet results with the reference's bookkeeping.
#include <cmath>
#include <cstring>
#include <vector>

#include "engine.h"
#include "kernels.h"

namespace osc {

double dt_inclusive(double tstart, double tstop, int L);

void Engine::power_density_stl(const double* tri, const double* centers, int64_t n, const osc_rad_opts& o,
                               double* out, int32_t* level_out) {
  if (device < 0) throw Error{OSC_ERR_NO_DEVICE, "this context was created without a GPU (device -1)"};
  check(cudaSetDevice(device), "cudaSetDevice");
  use_stream(stream);
  cudaStream_t st = stream;
  pending_.clear();
  last_samples = last_launches = last_not_converged = 0;
  // the levels stop at the deepest one that the reference keeps in memory (26; its samples take 10.7 GB)
  int ext_from = kMaxLevelMemory;
  const int lstop = request_levels(o, kMaxLevelMemory, &ext_from);
  if (n <= 0) return;
  set_level_grid(ext_from);
  for (int64_t i = 0; i < n; ++i) out[i] = 0;
  // facets and centres up in one copy from page-locked memory; states, flags and counters down in one
  const size_t up = sizeof(double) * 15 * n, back = sizeof(double) * 4 * n + sizeof(int) * 2 * n + sizeof(unsigned) * 32;
  stl_geo_.reserve(sizeof(double) * 9 * n);
  stl_cen_.reserve(up);  // facets n x 12, then centres n x 3
  const int grid = wave_grid(7, 0);
  const int64_t n_part = std::max<int64_t>(n, 8 * (int64_t)grid) * kStlPartials;
  // normals, boxes, span partials; list, its count, finished spans
  stl_nrm_.reserve(sizeof(double) * (3 * n + 6 * 148 + n_part) + sizeof(int) * (2 * n + 1));
  stl_state_.reserve(back);
  std::vector<unsigned char> pageable;
  unsigned char* host = bounce_for(std::max(up, back));
  if (!host) {
    pageable.resize(std::max(up, back));
    host = pageable.data();
  }
  std::memcpy(host, tri, sizeof(double) * 12 * n);
  std::memcpy(host + sizeof(double) * 12 * n, centers, sizeof(double) * 3 * n);
  check(cudaMemcpyAsync(stl_cen_.p, host, up, cudaMemcpyHostToDevice, st), "facets");
  double* d_state = stl_state_.as<double>();
  int* d_flags = reinterpret_cast<int*>(d_state + 4 * n);
  unsigned* d_active = reinterpret_cast<unsigned*>(d_flags + 2 * n);
  const int np = o.nparticles;
  const double weight = np > 0 ? 1.0 / (double)np : 1.0;
  const int L1 = std::min(9, lstop);  // facets can stop from level 9 on
  for (int ip = 0; ip < (np > 0 ? np : 1); ++ip) {
    if (np > 0) {  // src/OSCARSSR.cc:3234-3240: a new random particle and its trajectory
      model.random_particle();
      model.compute_trajectory();
    } else {
      model.ensure_trajectory();
    }
    check(cudaStreamSynchronize(st), "particle");  // the previous particle's launches read the caches
    upload_trajectory();
    const Particle& P = model.particle;
    StlWaveArgs a{};
    a.geometry = stl_geo_.as<double>();
    a.centers = stl_cen_.as<double>() + 12 * n;
    a.normals = stl_nrm_.as<double>();
    double* d_box = stl_nrm_.as<double>() + 3 * n;
    a.box = d_box;
    a.part = d_box + 6 * 148;
    a.act = reinterpret_cast<int*>(a.part + n_part);
    a.spans_done = reinterpret_cast<unsigned*>(a.act + n);
    a.n_act = a.act + 2 * n;
    a.n = n;
    a.precision = o.precision;
    a.two_over_gamma = 2. / P.gamma;
    a.state = d_state;
    a.done = d_flags;
    a.level_out = d_flags + n;
    a.n_active = d_active;
    // the first waves go out three at a time, deep ones (which need their level's samples filled) one by one,
    // then the host looks at the counters
    for (int L = L1; L <= lstop;) {
      const int end = std::min(lstop, L + (L <= 12 ? 2 : 0));
      ensure_levels(end);
      a.lev = lev_.as<double>();
      a.cap = lev_cap_;
      for (int l = L; l <= end; ++l) {
        a.first = l == L1;
        a.level = l;
        a.dt_prev = l >= 1 ? dt_inclusive(tstart_, tstop_, l - 1) : 0;
        a.dt_level = dt_inclusive(tstart_, tstop_, l);
        const int64_t s0 = a.first ? 1 : (int64_t)1 << l, s1 = (int64_t)2 << l;
        a.n_box = stl_box_blocks(s1 - s0);
        check(launch_stl_prepare(a, s0, s1, stl_cen_.as<double>(), stl_geo_.as<double>(), stl_nrm_.as<double>(), d_box, st),
              "stl prepare");
        const int64_t units = a.first ? n : n * std::max<int64_t>(1, (s1 - s0) / 512);
        check(launch_stl_wave(a, (int)std::min<int64_t>(units, a.first ? n : (int64_t)grid), st), "stl wave");
        last_launches += 2;
      }
      check(cudaMemcpyAsync(host, d_state, back, cudaMemcpyDeviceToHost, st), "state");
      check(cudaStreamSynchronize(st), "state");
      L = end + 1;
      const unsigned* active = reinterpret_cast<const unsigned*>(host + sizeof(double) * 4 * n + sizeof(int) * 2 * n);
      if (end > 8 && active[end] == 0) break;
    }
    const double* state = reinterpret_cast<const double*>(host);
    const int* flags = reinterpret_cast<const int*>(state + 4 * n);
    const unsigned* active = reinterpret_cast<const unsigned*>(flags + 2 * n);
    for (int l = 0; l <= lstop; ++l) {  // levels some facet still needed
      last_samples += ((int64_t)1 << l) * n;
      if (l > 8 && active[l] == 0) break;
    }
    // src/OSCARSSR.cc:3503-3521.  Result_Level lives outside the loop over facets: a facet that does
    // not stop reports the level of the last facet that did (-1 before any).
    const double scale = std::fabs(P.q * P.current) / (16 * (kPi * kPi) * kEps0 * kC);
    int carried = -1;
    for (int64_t i = 0; i < n; ++i) {
      const int lv = flags[n + i];
      if (lv >= 0) carried = lv;
      else ++last_not_converged;
      double v;
      switch (o.quantity) {
        case 1: v = state[4 * i + 2] * weight; break;
        case 2: v = ((double)carried) * weight; break;
        default: {
          double sum = state[4 * i] * (scale * dt_inclusive(tstart_, tstop_, (int)state[4 * i + 3]));
          sum /= 1e6;
          v = sum * weight;
        }
      }
      out[i] = v + out[i];  // TTriangle3D::AddToValue
      if (level_out) level_out[i] = carried;
    }
  }
}

}  // namespace osc
