// nbr_device.cuh -- sm_100a device helpers shared by the N-body kernels.
//
//  * packed FP32 pair arithmetic (add/sub/mul/fma .f32x2, PTX ISA 8.6,
//    sm_100+): one instruction operates on two particles held in a 64-bit
//    register pair, which halves the issue slots the FP32 pipe needs;
//  * the MUFU reciprocal square root (rsqrt.approx.ftz.f32);
//  * mbarrier + cp.async.bulk (1-D TMA) primitives for the shared-memory
//    j-tile ring.  No multicast form is used anywhere;
//  * bounded waits: every spin has a wall-clock limit after which the kernel
//    records an error code for the host and stops consuming tiles.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace nbr {

// Particles per j-tile; also the group size the FP32 tile origins are taken over.
constexpr int kTile = 128;
// Default wall-clock limit of one bounded wait, in nanoseconds (%globaltimer).
constexpr unsigned long long kWaitLimitNs = 4000000000ull;

// Device error codes (written with atomicCAS(err, 0, code): first one wins).
enum : int {
  kErrNone = 0,
  kErrTileWait = 1,    // a j-tile's bulk copy did not complete in time
  kErrDrainWait = 2,   // draining in-flight copies after an abort timed out
  kErrBounds = 3,      // checked builds: an index outside its array (access skipped)
  kErrGridWait = 4,    // a grid-wide barrier of a persistent launch did not complete in time
};

typedef unsigned long long u64;

// ----------------------------------------------------------------- f32x2 ----
__device__ __forceinline__ u64 pack2(float lo, float hi) {
  u64 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(u64 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ u64 add2(u64 a, u64 b) {
  u64 d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 sub2(u64 a, u64 b) {
  u64 d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b) {
  u64 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c) {
  u64 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
// c - a b (the sign of a flipped off the FMA pipe).
__device__ __forceinline__ u64 fnma2(u64 a, u64 b, u64 c) {
  return fma2(a ^ 0x8000000080000000ull, b, c);
}
// MUFU reciprocal square root of each half.
__device__ __forceinline__ float rsqrt_mufu(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ u64 rsqrt2(u64 v) {
  float lo, hi;
  unpack2(v, lo, hi);
  return pack2(rsqrt_mufu(lo), rsqrt_mufu(hi));
}

// ------------------------------------------------------------------ FP64 ----
// r^-3 / kInvCubeScale for r2 = r^2 >= 0, on the FP64 pipe.  The pair loops
// need 1/r only as its cube (forces) or times a mass (potentials), so one
// series correction of the seed replaces a correctly rounded square root and
// the multiplications that cube it.
//
// The seed y = rsqrt.approx.ftz.f64(r2) has 21 significant bits (its low word
// is zero), so y^2 is exact and h = 1 - r2 y^2 is small: |h| <= 1.9e-6
// (measured over 1.5e9 arguments).  From the binomial series
//     r^-3 = y^3 (1 - h)^(-3/2) = y^3 (1 + 3/2 h + 15/8 h^2 + 35/16 h^3 ...)
// the terms up to h^2 are kept (the next is below 1.5e-17), completed to a
// square so that they cost one addition fused into h's own fma and one fma:
//     1 + 3/2 h + 15/8 h^2 = 15/8 (u^2 + 28/75),   u = h + 2/5 = 7/5 - r2 y^2.
// The factor 15/8 is left to the caller, who scales its sums once.  28/75 is
// rounded to the double that makes 15/8 (u^2 + c) equal 1 at h = 0 to 3e-18
// for the double nearest 7/5.  Five FP64 operations and one MUFU after r2; a
// CUDA rsqrt(double) and its cube take about twelve (rates measured on B200:
// 59 fma, 15.8 seeds and 5.05 rsqrt(double) per clock and SM).  Error against
// extended precision over r2 = 2^-60 .. 2^60 (4 M arguments): largest 4.3e-16,
// rms 1.04e-16; rsqrt(double) cubed 5.5e-16 and 1.56e-16.
//
// r2 = +inf gives 0 and NaN gives NaN, as with rsqrt(): the seed's are 0 and
// NaN, and the clamp of r2's high word (an integer minimum, off the FP64 pipe)
// keeps 0 x inf out of u.  A subnormal r2 gives inf, where the cube of the
// exact result overflows too.  EXCL: r2 = 0 gives 0 (the excluded pair).
constexpr double kInvCubeScale = 1.875;
__device__ __forceinline__ double rsqrt_seed64(double r2) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
  return y;
}
__device__ __forceinline__ double clamp_finite64(double r2) {
  return __hiloint2double(min(__double2hiint(r2), 0x7fefffff), __double2loint(r2));
}
template <bool EXCL>
__device__ __forceinline__ double inv_cube(double r2) {
  double y = rsqrt_seed64(r2);
  if (EXCL) y = __double_as_longlong(r2) != 0 ? y : 0.0;
  const double y2 = y * y;
  const double u = fma(-clamp_finite64(r2), y2, 1.4);
  const double c = fma(u, u, 0.3733333333333334);
  return (y2 * y) * c;
}

// r^-1 / kInvDistScale for r2 = r^2, by the series of inv_cube:
//     r^-1 = y (1 - h)^(-1/2) = y (1 + 1/2 h + 3/8 h^2 + ...)
//          = 3/8 y (u^2 + 20/9),   u = h + 2/3 = 5/3 - r2 y^2,
// the next term below 5/16 (1.9e-6)^3 = 2.1e-18; 20/9 and 3/8 are rounded to
// the doubles whose product is nearest 1 at h = 0 (2e-17).  Four FP64
// operations and one MUFU.  Only for normal r2: a caller whose sums stay
// finite where r2 is subnormal takes inv_dist_tiny there (r2 below kTinyHi).
constexpr double kInvDistScale = 0.37499999999999994;
__device__ __forceinline__ double inv_dist(double r2) {
  const double y = rsqrt_seed64(r2);
  const double u = fma(-clamp_finite64(r2), y * y, 1.6666666666666665);
  return y * fma(u, u, 2.2222222222222228);
}
// High word of r2 >= 0: below kTinyHi if r2 is zero or subnormal.
constexpr int kTinyHi = 0x00100000;
// inv_dist for any r2; EXCL: 0 for r2 = 0.
template <bool EXCL>
__device__ __noinline__ double inv_dist_tiny(double r2) {
  if (EXCL && !(r2 > 0.0)) return 0.0;
  return rsqrt(r2) * (1.0 / kInvDistScale);
}

// Sum of p[0], p[ld], .. p[(K - 1) ld], K a power of two, by halves: the chain
// of roundings (and of latencies) is log2 K long instead of K.
template <int K>
__device__ __forceinline__ double sum_by_halves(const double* p, int ld) {
  if constexpr (K == 1) return *p;
  else return sum_by_halves<K / 2>(p, ld) + sum_by_halves<K / 2>(p + K / 2 * ld, ld);
}

// hi + lo <- hi + lo + x: the rounding error of the sum goes to lo (Knuth TwoSum).
__device__ __forceinline__ void add_error_free(double& hi, double& lo, double x) {
  const double s = hi + x, b = s - hi;
  lo += (hi - (s - b)) + (x - b);
  hi = s;
}
// scale (hi + lo), rounded once; where hi overflowed, its infinity (lo is NaN).
__device__ __forceinline__ double scaled_sum(double scale, double hi, double lo) {
  return isfinite(hi) ? fma(scale, hi, scale * lo) : scale * hi;
}

// Knuth TwoSum of the packed pair (hi + p): hi <- rounded sum, lo += the
// rounding error.  Six packed adds; exact error term for round-to-nearest.
__device__ __forceinline__ void two_sum2(u64& hi, u64& lo, u64 p) {
  u64 s = add2(hi, p);
  u64 bp = sub2(s, hi);
  u64 ap = sub2(s, bp);
  u64 e = add2(sub2(hi, ap), sub2(p, bp));
  lo = add2(lo, e);
  hi = s;
}

// --------------------------------------------------------------- timing -----
__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// ------------------------------------------------------- mbarrier + bulk ----
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for the barrier phase with the given parity; gives up after limit_ns
// and returns false (the caller records the error).
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity,
                                                  unsigned long long limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if (global_ns() - t0 > limit_ns) return false;
  }
}
// 1-D bulk copy global -> this CTA's shared memory, completing on `bar`.
// dst, src 16-byte aligned; bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void record_error(int* err, int code) {
  if (err) atomicCAS(err, 0, code);
}

// Checked builds (-DNBR_CHECKED, libnbr_checked.so) test every array index
// against the array's allocated length, passed with the launch, before the
// access; a failing index is recorded (kErrBounds) and the access skipped.
// In normal builds NBR_IN is the constant true and the length expression is
// never compiled.
__device__ __forceinline__ bool in_bounds(long long idx, long long len, int* err) {
  if (idx >= 0 && idx < len) return true;
  record_error(err, kErrBounds);
  return false;
}
#ifdef NBR_CHECKED
#define NBR_IN(idx, len, err) (::nbr::in_bounds((long long)(idx), (long long)(len), (err)))
#else
#define NBR_IN(idx, len, err) true
#endif

}  // namespace nbr
