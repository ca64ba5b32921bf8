// device_common.cuh -- device helpers shared by the radiation kernels (sm_100a).
//
//  * 1-D TMA bulk copies global -> shared (cp.async.bulk ... mbarrier::complete_tx::bytes), with
//    mbarrier waits that give up after a bounded number of polls and raise an error flag instead
//    of hanging the GPU.
//  * Argument reduction of the retarded phase to [-pi, pi] (Cody & Waite two-constant reduction;
//    the first step is exact with FMA for |phase| < 2^52 ulp(2pi), see reduce_2pi below).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace osc {
namespace dev {

// Error flags written by kernels (bit mask, OR-ed into a device word read back by the host).
// kErrPlan: a kernel was launched with a tile size other than the one it was compiled for (the
// host sized its partial sums for that tile); the kernel returns before touching memory.
enum : unsigned { kErrTmaTimeout = 1u, kErrBadArgs = 2u, kErrSuperluminal = 4u, kErrPlan = 8u };

// Polls of an mbarrier before a wait is declared stuck (each poll is a try_wait that itself may
// suspend the thread for a hardware-defined interval), i.e. far beyond any legitimate latency.
constexpr uint32_t kMaxPolls = 1u << 22;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
               : "memory");
}

// Returns true once the barrier phase with parity `parity` has completed; false if it did not
// complete within kMaxPolls polls.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const uint32_t a = smem_addr(bar);
  for (uint32_t i = 0; i < kMaxPolls; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}

// Programmatic dependent launch: a wave lets the next one's CTAs become resident as soon as its own are
// (launch_dependents), and a wave launched that way waits for its predecessor's end, with its memory
// visible, before it touches anything the predecessor writes (wait).  Without the launch attribute both
// do nothing.
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Bulk copy `bytes` (multiple of 16, both addresses 16-byte aligned) from global to shared memory,
// completing on `bar`.
__device__ __forceinline__ void tma_load_1d(void* smem_dst, const void* gmem_src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_addr(smem_dst)),
      "l"(gmem_src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

// ---------------------------------------------------------------------------------------------
// Phase reduction.  For a double `phi` with |phi| < 2^40, k = rint(phi / 2pi) and
//   r1 = fma(-k, P1, phi)    is exact: phi and k*P1 are both multiples of 2^-50 once |phi| >= 4
//                            and |r1| < 4, so r1 fits in 53 bits;
//   r  = fma(-k, P2, r1)     adds the second term of 2pi = P1 + P2 (+ O(2^-107)).
// The reduced argument carries an absolute error below 1e-15 for |phi| < 2^40 (4 x 10^11 rad at
// 3 keV and 30 m is 2^38.7), so sin/cos of it agree with the correctly rounded sin/cos of phi to a
// few 1e-16.  (Cody & Waite, "Software Manual for the Elementary Functions", 1980.)
// ---------------------------------------------------------------------------------------------
constexpr double kTwoPiHi = 6.283185307179586232;      // RN(2 pi)
constexpr double kTwoPiLo = 2.4492935982947064e-16;    // RN(2 pi - kTwoPiHi)
constexpr double kInvTwoPi = 0.15915494309189535;      // RN(1 / (2 pi))

__device__ __forceinline__ double reduce_2pi(double phi) {
  const double k = rint(phi * kInvTwoPi);
  const double r1 = __fma_rn(-k, kTwoPiHi, phi);
  return __fma_rn(-k, kTwoPiLo, r1);
}

// ---------------------------------------------------------------------------------------------
// FP64 square root, reciprocals and quotients that share one reciprocal square root.
//
// The sums divide three components and the phase by the same distance; correctly rounded library
// divisions would cost ~9 FP64 operations each, and B200's FP64 pipe (one warp instruction per two
// cycles and sub-partition) is what bounds these kernels.  From a ~20-bit hardware seed, one
// third-order step y' = y (1 + e/2 + 3 e^2 / 8), e = 1 - s y^2, gives 1 / sqrt(s) to about an ulp, and
// Markstein's corrections ("Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990) round the square root and each quotient as the exact
// operations do: g + (s - g^2) y / 2 with g = s y, and q + (a - q D) y with q = a y (residuals exact in
// FMA).  200 million random distances and 600 million quotients gave sqrt's and division's bits
// every time (the chance of a difference is ~2^-50 per operation).  The division by the speed of
// light is Brisebarre, Muller and Raina's multiplication by a double-double constant ("Accelerating
// correctly rounded floating-point division when the divisor is known in advance", IEEE Trans.
// Comput. 53, 2004): c has 29 significant bits, so no quotient lies close enough to a midpoint of two
// doubles for the 2^-106 error of the product to matter.
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double rcp_seed(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
// 1 / sqrt(s) to about an ulp.
__device__ __forceinline__ double rsqrt_near(double s) {
  const double y0 = rsqrt_seed(s);
  const double e = __fma_rn(-__dmul_rn(s, y0), y0, 1.0);
  return __fma_rn(y0, __dmul_rn(e, __fma_rn(0.375, e, 0.5)), y0);
}
// 1 / x to about an ulp.
__device__ __forceinline__ double rcp_near(double x) {
  const double y0 = rcp_seed(x);
  const double e = __fma_rn(-x, y0, 1.0);
  return __fma_rn(y0, __fma_rn(e, e, e), y0);
}
// sqrt(s), with y = rsqrt_near(s).
__device__ __forceinline__ double sqrt_by(double s, double y) {
  const double g = __dmul_rn(s, y);
  return __fma_rn(__fma_rn(-g, g, s), 0.5 * y, g);
}
// a / D, with y within about an ulp of 1 / D.
__device__ __forceinline__ double quot_by(double a, double D, double y) {
  const double q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(-q, D, a), y, q);
}
constexpr double kInvC1 = 3.3356409519815204e-09;  // RN(1 / c)
constexpr double kInvC2 = 6.917657862297521e-26;   // RN(1 / c - kInvC1)
__device__ __forceinline__ double over_c(double D) { return __fma_rn(D, kInvC1, __dmul_rn(D, kInvC2)); }

// sin and cos of a phase with |phi| < 2^49 (3 keV at 30 m is 2^38.7): phi - k pi/2 by the two-constant
// reduction above (k from the low word of phi 2/pi + 1.5 2^52), then sin and cos of the remainder in
// [-pi/4, pi/4] by polynomials in its square, Chebyshev fits of (sin r - r) / r^3 and
// (cos r - 1 + r^2/2) / r^4 computed in 60 digits (2.0e-17 and 1.3e-18 off), the quadrant by exchange
// and sign.  19 FP64 operations; within 1.6e-16 of the exact sine and cosine over that range.
constexpr double kTwoOverPi = 0.6366197723675814;       // RN(2 / pi)
constexpr double kHalfPiHi = 1.5707963267948966;        // RN(pi / 2)
constexpr double kHalfPiLo = 6.123233995736766e-17;     // RN(pi / 2 - kHalfPiHi)
constexpr double kRoundBase = 6755399441055744.0;       // 1.5 2^52
constexpr double kPhaseFast = 562949953421312.0;        // 2^49
__device__ __forceinline__ void sincos_fast(double phi, double* sn, double* cs) {
  const double kb = __fma_rn(phi, kTwoOverPi, kRoundBase);
  const int q = __double2loint(kb);
  const double k = __dsub_rn(kb, kRoundBase);
  const double r = __fma_rn(-k, kHalfPiLo, __fma_rn(-k, kHalfPiHi, phi));
  const double z = __dmul_rn(r, r);
  double p = 1.591810123027412e-10, c = -1.1382614868556325e-11;
  p = __fma_rn(p, z, -2.5051131455427946e-08);
  c = __fma_rn(c, z, 2.0876146024689747e-09);
  p = __fma_rn(p, z, 2.755731610068303e-06);
  c = __fma_rn(c, z, -2.7557317270560326e-07);
  p = __fma_rn(p, z, -0.0001984126983675497);
  c = __fma_rn(c, z, 2.4801587298763433e-05);
  p = __fma_rn(p, z, 0.008333333333330946);
  c = __fma_rn(c, z, -0.0013888888888887395);
  p = __fma_rn(p, z, -0.16666666666666666);
  c = __fma_rn(c, z, 0.041666666666666664);
  p = __fma_rn(__dmul_rn(p, z), r, r);
  c = __fma_rn(__fma_rn(c, z, -0.5), z, 1.0);
  const double a = (q & 1) ? c : p, b = (q & 1) ? p : c;
  *sn = __hiloint2double(__double2hiint(a) ^ ((q & 2) << 30), __double2loint(a));
  *cs = __hiloint2double(__double2hiint(b) ^ (((q + 1) & 2) << 30), __double2loint(b));
}
// The same for any phase (beyond kPhaseFast the library's routine on the 2 pi reduction).
static __device__ __noinline__ void sincos_far(double phi, double* sn, double* cs) { sincos(reduce_2pi(phi), sn, cs); }

}  // namespace dev

// Launch that may overlap its predecessor's tail on the stream (the kernel calls wait_predecessor()):
// 2 to 3 us less between the waves of a request.
template <class... P, class... A>
inline cudaError_t launch_overlapped(void (*kernel)(P...), int grid, int threads, cudaStream_t st, A... args) {
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)threads);
  c.stream = st;
  cudaLaunchAttribute a{};
  a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a.val.programmaticStreamSerializationAllowed = 1;
  c.attrs = &a;
  c.numAttrs = 1;
  return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

}  // namespace osc
