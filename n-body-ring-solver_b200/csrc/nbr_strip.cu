// nbr_strip.cu -- Newton-3 force evaluation in strips, one warp each.
//
// Every unordered pair is evaluated once and acts on both particles, as the
// reference's blocked kernels do (compute_forces_avx512_rsqrt_4i_blocked,
// CPU/force_calculation.cpp:1137-1561).  The particles form row blocks of
// 32 NI receivers (NI per lane of a warp) and batches of 32 sources.  A unit is
// one row block against one batch at or after the block's own first batch; the
// units, row block by row block, form one sequence that is cut into strips of
// equal length, one per warp of a grid with one CTA per SM.  So the work is
// spread evenly whatever the size, down to single units, no warp waits for
// another, and nothing but L2 loads and register shuffles feeds the loop.
//
// In a unit the 32 sources sit one per lane and travel through the warp in 32
// steps, carrying their reaction sums, so that each meets the warp's 32 NI
// receivers and is back on its lane with its reaction from them.  In the
// block's own batches the same loop runs and the reactions are dropped (every
// ordered pair is met there).  The reaction of (row block, batch) goes to its
// own slot; a strip's action sums on a row block go to slot (strip + row block),
// which no other segment has, since along the sequence either number grows.
// k_strip_reduce then adds each particle's partial sums in a fixed order and
// runs the epilogue: deterministic, no atomics.
//
// Why strips.  The grid of CTAs over (8 row blocks, chunk of column blocks)
// in nbr_kernels.cu, which shares tiles and sums reactions per CTA, needs about
// 600 CTAs to balance and idles on the diagonal, so it only pays from about
// 16384 particles, and its warps meet at a barrier per tile.  Strips write
// one reaction per (row block, particle) instead of one per (2048 rows,
// particle), 12 B (FP32C) or 24 B (FP64): at N = 262144 0.8 and 2.6 GB, written
// during the loop and read once.  Both forms' times stand where the choice between
// them is made, at choose_config and uses_strips (nbr_capi.cu).
#include "nbr_device.cuh"
#include "nbr_kernels.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <vector>

namespace nbr {

namespace {

// Units of row blocks r0 .. r - 1 (r0 <= r).
__host__ __device__ inline int strip_prefix(const StripPlan& p, int r) {
  return (int)((long long)(r - p.r0) * p.batches -
               (long long)p.tb * (((long long)r * (r - 1) - (long long)p.r0 * (p.r0 - 1)) / 2));
}
// First element of row block r's reactions: [batch after its own][3][32].
__host__ __device__ inline long long strip_rea_off(const StripPlan& p, int r) {
  return 96 * ((long long)(r - p.r0) * p.batches -
               (long long)p.tb * (((long long)r * (r + 1) - (long long)p.r0 * (p.r0 + 1)) / 2));
}
// First unit of strip g: the first p.longer strips hold one unit more.
__host__ __device__ inline int strip_start(const StripPlan& p, int g) {
  return g * p.share + min(g, p.longer);
}
// The strip that holds unit u.
__device__ inline int strip_owner(const StripPlan& p, int u) {
  const int cut = p.longer * (p.share + 1);
  return u < cut ? u / (p.share + 1) : p.longer + (u - cut) / p.share;
}
// The row block that holds unit u: the root of strip_prefix, corrected for
// the rounding of the float estimate.
__device__ inline int strip_row(const StripPlan& p, int u) {
  const float h = (float)p.batches + 0.5f * p.tb - (float)p.tb * p.r0;
  int r = p.r0 + (int)((h - sqrtf(fmaxf(h * h - 2.f * p.tb * (float)u, 0.f))) / p.tb);
  r = max(p.r0, min(r, p.r1 - 1));
  while (r + 1 < p.r1 && strip_prefix(p, r + 1) <= u) ++r;
  while (r > p.r0 && strip_prefix(p, r) > u) --r;
  return r;
}

// The strips and the reduction are launched with programmatic stream
// serialization: a kernel may be set up while the one before it in the stream
// finishes.  It reads nothing that a kernel writes and writes nothing before
// grid_dependency_wait(), which returns when that kernel has completed and its
// writes are visible.  us per evaluation in a graph, without / with: FP64 N = 4224
// 23.9 / 21.3, 6000 34.7 / 33.6; FP32C 4224 18.4 / 15.4, 6000 22.4 / 21.2, 12001 61.9 /
// 59.7.
__device__ __forceinline__ void grid_dependency_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
__device__ __forceinline__ void launch_dependents() {
  asm volatile("griddepcontrol.launch_dependents;");
}

// FP32C.  r^-3 = y^3 (1 - h)^(-3/2) with y the MUFU root and h = 1 - r2 y^2 is
// y^3 (1 + 3/2 h) to first order = 3/2 y^3 (5/3 - r2 y^2): one fma after y^2, and
// the masses of both particles multiply it, so a pair costs 3 differences, 3
// fma, 6 operations for both scalars and 6 fma = 18 (k_force_n3_f32c folds
// the masses into the correction: 19, with one register more per mass).  The
// factor is left to k_strip_reduce, as the double 1 / (c - 1), c the float
// nearest 5/3, so that the constant's rounding cancels at h = 0.
//
// What bounds it: register-file reads.  Packed fma with three distinct 64-bit
// operands issue at 3/4 of the pipe's rate (measured), and the pair needs about
// 42 operand reads for 36 pipe cycles.  What helped, at N = 262144 (GPairs/s):
// more receivers per lane, since a step's 10 shuffles and source registers
// serve them all (NI = 8 2870, 10 3016, 12 3064, 16 3166); keeping the FP64
// action sums, touched once per tile, in shared memory instead of registers
// (NI = 12 2912 -> 3039); doing each operation for all receivers before the
// next one (2805 -> 2912); sources by shuffle rather than from shared memory
// (3133 against 3166 at NI = 16).
//
// Coordinates are relative to the tile's FP64 origin in FP32; per tile of 128
// sources the FP32 action sums are added to FP64 sums.  The origin is the mean of
// the tile's 128 particles, one of the first 32 counted twice: which one goes
// with the row block.  It is taken from the tile's first particle, so that a
// coordinate which all share is its origin exactly: the roundings of the mean of
// 1e60 are past the range of FP32.
//
// Rounding: no more than in the kernels before (lane groups, tiles joined by
// two_sum, reactions in FP64) takes two things.  A reaction is no longer one chain
// of 16 NI additions in each half: at NI = 16 it is added up in two parts of 16
// steps, with a narrower block (FINE) a step's terms are added before they join
// the travelling sum.  And an origin of its own for each row block: a source's
// coordinates are rounded anew for each, where with one origin all its reactions
// carried the same displacement.  Median error of a force (eps 1e-3), before / one
// chain and one origin / now: masses within a factor of three N = 6000
// 3.3e-8 / 4.1e-8 / 3.3e-8, 12001 3.8e-8 / 4.7e-8 / 3.6e-8, 65536 3.5e-8 / 3.7e-8 /
// 3.0e-8, 262144 3.2e-8 / 3.1e-8 / 2.7e-8; masses over many decades (lognormal, one of
// a hundred 1000 times as heavy) 14000 10.7e-8 / 10.1e-8 / 8.4e-8, 131073 6.5e-8 /
// 7.5e-8 / 6.2e-8, 262143 6.0e-8 / 6.6e-8 / 5.2e-8.  FINE took 1.5 % more at NI = 16 than the parts (us per evaluation
// 65536 1388 / 1371, 262144 21.76 / 21.48 ms; one chain 21.38), the parts 1.6 % more
// than FINE at N = 8192 (32.7 / 32.2).
//
// The padding lanes of the last batch take the last particle's coordinates,
// with their own mass, zero: the pair factor multiplies the masses last, and at
// that place it is inf or NaN only if it is for a real pair too.  (Where the
// arrays hold the padding, at the coordinate origin, it may lie 1e20 units from
// a particle, or 1e-14.)
//
// Masses are divided by the mantissa of particle 0's before they are rounded to
// FP32, and the sums multiplied by it.  Equal masses, and whole ratios of them,
// then carry no rounding; otherwise all bodies of a mass act with up to 6e-8 too
// much or too little.  No mass changes by more than a factor of two.  Median error
// of a force, equal masses, without / with: N = 5000 4.5e-8 / 3.5e-8, 7000 3.5e-8 /
// 3.3e-8, 20000 4.3e-8 / 3.1e-8.
constexpr float kC53 = 1.66666663f;
// The mantissa of m, in [1, 2) (1 for zero and subnormal masses).
__device__ __forceinline__ double mass_mantissa(double m) {
  const int hi = __double2hiint(m);
  return hi < 0x00100000 ? 1.0
                         : __hiloint2double((hi & 0x000fffff) | 0x3ff00000, __double2loint(m));
}

template <int NI, bool EXCL>
__global__ void __launch_bounds__(kStripWarps * 32, 1)
    k_strip_f32c(const IParticles ip, const JStream js, const StripPlan sp, const float eps2f,
                 double* act, float* rea, int* err) {
  constexpr int IP = NI / 2, TB = NI;
  constexpr bool FINE = NI < 16;
  constexpr int PART = FINE ? 32 : 16;  // steps of a reaction's chain
  extern __shared__ double strip_acc[];  // [kStripWarps][3][32 NI]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = warp * gridDim.x + blockIdx.x;
  const double unit = 1.0 / mass_mantissa(js.m[0]);  // (no kernel writes masses)
  grid_dependency_wait();
  launch_dependents();
  if (g >= sp.strips) return;
  int u = strip_start(sp, g);
  const int u_end = strip_start(sp, g + 1);
  const int from = (lane + 31) & 31, from_part = (lane + 32 - PART) & 31;
  const u64 EPS2 = pack2(eps2f, eps2f), C53 = pack2(kC53, kC53);
  double* acc = strip_acc + warp * (96 * NI) + lane;
  for (int r = strip_row(sp, u); u < u_end; ++r) {
    const int b0 = r * TB + (u - strip_prefix(sp, r));
    const int b1 = min(sp.batches, b0 + (u_end - u));
    u += b1 - b0;
    const long long ibase = (long long)r * (32 * NI) + lane;
    const int twice = r & 31;        // the particle of a tile that counts twice for its origin
    const int b_rea = (r + 1) * TB;  // first batch whose reactions are kept
    const long long len = 96LL * (sp.batches - b_rea);  // reactions of this row block
    if (!NBR_IN((long long)(r + 1) * (32 * NI) - 1, ip.len, err) ||
        !NBR_IN(32LL * (((b1 - 1) | 3) + 1) - 1, js.len, err) ||
        !NBR_IN((long long)(g + r - sp.r0 + 1) * (96 * NI) - 1, sp.act_doubles, err) ||
        (len > 0 && !NBR_IN(strip_rea_off(sp, r) + len - 1, sp.reactions, err)))
      return;
    float* out = rea + strip_rea_off(sp, r) + lane - 96LL * b_rea;
    u64 MI[IP];
#pragma unroll
    for (int p = 0; p < IP; ++p)
      MI[p] = pack2((float)(unit * ip.m[ibase + 64 * p]), (float)(unit * ip.m[ibase + 64 * p + 32]));
#pragma unroll
    for (int k = 0; k < 3 * NI; ++k) acc[32 * k] = 0.0;
#pragma unroll 1
    for (int b = b0; b < b1;) {
      // one tile of 4 batches and its origin; a ragged tile's particles are each
      // taken several times
      const int b_tile = min(b1, (b & ~3) + 4);
      double ox = 0.0, oy = 0.0, oz = 0.0;
      {
        const long long t0 = (long long)(b & ~3) * 32;
        const int left = (int)min(128LL, ip.n - t0);  // the tile's particles
        const double fx = js.x[t0], fy = js.y[t0], fz = js.z[t0];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int t = (lane + 32 * k) * left >> 7;
          const double w = k == 0 && lane == twice ? 2.0 : 1.0;
          ox = fma(w, js.x[t0 + t] - fx, ox);
          oy = fma(w, js.y[t0 + t] - fy, oy);
          oz = fma(w, js.z[t0 + t] - fz, oz);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          ox += __shfl_xor_sync(0xffffffffu, ox, off);
          oy += __shfl_xor_sync(0xffffffffu, oy, off);
          oz += __shfl_xor_sync(0xffffffffu, oz, off);
        }
        ox = fma(ox, 1.0 / 129.0, fx); oy = fma(oy, 1.0 / 129.0, fy); oz = fma(oz, 1.0 / 129.0, fz);
      }
      u64 XI[IP], YI[IP], ZI[IP], AX[IP], AY[IP], AZ[IP];
#pragma unroll
      for (int p = 0; p < IP; ++p) {
        const long long i = ibase + 64 * p;
        XI[p] = pack2(__double2float_rn(ip.x[i] - ox), __double2float_rn(ip.x[i + 32] - ox));
        YI[p] = pack2(__double2float_rn(ip.y[i] - oy), __double2float_rn(ip.y[i + 32] - oy));
        ZI[p] = pack2(__double2float_rn(ip.z[i] - oz), __double2float_rn(ip.z[i + 32] - oz));
        AX[p] = AY[p] = AZ[p] = 0ull;
      }
#pragma unroll 1
      for (; b < b_tile; ++b) {
        const long long j = 32LL * b + lane, jx = min(j, ip.n - 1);
        float sx = __double2float_rn(js.x[jx] - ox), sy = __double2float_rn(js.y[jx] - oy),
              sz = __double2float_rn(js.z[jx] - oz), sm = (float)(unit * js.m[j]);
        float qx = 0.f, qy = 0.f, qz = 0.f;  // the reaction of the parts before
#pragma unroll 1
        for (int part = 0; part < 32 / PART; ++part) {
          u64 RX = 0ull, RY = 0ull, RZ = 0ull;
#pragma unroll(NI >= 12 ? 2 : 4)
          for (int step = 0; step < PART; ++step) {
            const u64 SX = pack2(sx, sx), SY = pack2(sy, sy), SZ = pack2(sz, sz), SM = pack2(sm, sm);
            u64 dx[IP], dy[IP], dz[IP], r2[IP], y[IP], y2[IP], c[IP];
#pragma unroll
            for (int p = 0; p < IP; ++p) dx[p] = sub2(SX, XI[p]);
#pragma unroll
            for (int p = 0; p < IP; ++p) dy[p] = sub2(SY, YI[p]);
#pragma unroll
            for (int p = 0; p < IP; ++p) dz[p] = sub2(SZ, ZI[p]);
#pragma unroll
            for (int p = 0; p < IP; ++p) r2[p] = fma2(dx[p], dx[p], EPS2);
#pragma unroll
            for (int p = 0; p < IP; ++p) r2[p] = fma2(dy[p], dy[p], r2[p]);
#pragma unroll
            for (int p = 0; p < IP; ++p) r2[p] = fma2(dz[p], dz[p], r2[p]);
#pragma unroll
            for (int p = 0; p < IP; ++p) {
              if (EXCL) {
                float rl, rh;
                unpack2(r2[p], rl, rh);
                y[p] = pack2(rl > 0.f ? rsqrt_mufu(rl) : 0.f, rh > 0.f ? rsqrt_mufu(rh) : 0.f);
              } else {
                y[p] = rsqrt2(r2[p]);
              }
            }
#pragma unroll
            for (int p = 0; p < IP; ++p) y2[p] = mul2(y[p], y[p]);
#pragma unroll
            for (int p = 0; p < IP; ++p) c[p] = fnma2(r2[p], y2[p], C53);
#pragma unroll
            for (int p = 0; p < IP; ++p) y2[p] = mul2(y2[p], y[p]);
#pragma unroll
            for (int p = 0; p < IP; ++p) c[p] = mul2(y2[p], c[p]);
            u64 tx = RX, ty = RY, tz = RZ;  // FINE: the step's reaction alone
#pragma unroll
            for (int p = 0; p < IP; ++p) {
              const u64 sj = mul2(c[p], SM), si = mul2(c[p], MI[p]);
              tx = FINE && p == 0 ? mul2(si, dx[p]) : fma2(si, dx[p], tx);
              ty = FINE && p == 0 ? mul2(si, dy[p]) : fma2(si, dy[p], ty);
              tz = FINE && p == 0 ? mul2(si, dz[p]) : fma2(si, dz[p], tz);
              AZ[p] = fma2(sj, dz[p], AZ[p]);
              AY[p] = fma2(sj, dy[p], AY[p]);
              AX[p] = fma2(sj, dx[p], AX[p]);
            }
            RX = __shfl_sync(0xffffffffu, FINE ? add2(RX, tx) : tx, from);
            RY = __shfl_sync(0xffffffffu, FINE ? add2(RY, ty) : ty, from);
            RZ = __shfl_sync(0xffffffffu, FINE ? add2(RZ, tz) : tz, from);
            sx = __shfl_sync(0xffffffffu, sx, from);
            sy = __shfl_sync(0xffffffffu, sy, from);
            sz = __shfl_sync(0xffffffffu, sz, from);
            sm = __shfl_sync(0xffffffffu, sm, from);
          }
          float l, h;
          unpack2(RX, l, h); qx = __shfl_sync(0xffffffffu, qx, from_part) + (l + h);
          unpack2(RY, l, h); qy = __shfl_sync(0xffffffffu, qy, from_part) + (l + h);
          unpack2(RZ, l, h); qz = __shfl_sync(0xffffffffu, qz, from_part) + (l + h);
        }
        if (b >= b_rea) {
          float* o = out + 96LL * b;
          o[0] = -qx; o[32] = -qy; o[64] = -qz;
        }
      }
#pragma unroll
      for (int p = 0; p < IP; ++p) {
        float l, h;
        unpack2(AX[p], l, h); acc[64 * p] += (double)l; acc[64 * p + 32] += (double)h;
        unpack2(AY[p], l, h); acc[32 * NI + 64 * p] += (double)l; acc[32 * NI + 64 * p + 32] += (double)h;
        unpack2(AZ[p], l, h); acc[64 * NI + 64 * p] += (double)l; acc[64 * NI + 64 * p + 32] += (double)h;
      }
    }
    double* a = act + (long long)(g + r - sp.r0) * (96 * NI) + lane;
#pragma unroll
    for (int k = 0; k < 3 * NI; ++k) a[32 * k] = acc[32 * k];
  }
}

// FP64: 3 differences, 3 fma, 5 operations of inv_cube, 2 for the masses and 6
// fma = 19 per unordered pair.  Bound by the register-file ports as
// k_force_n3_f64 is; the step reads its source from the warp's staging buffer
// in shared memory, one step ahead, and shuffles the three reaction sums.
// N = 262144, GPairs/s: NI = 6 1494, 8 1525, 10 1548 (254 registers).  Two
// receivers at a time, the loop unrolled by 4: 1534 -> 1548.
//
// Rounding: the kernels this one replaces on small systems add in short chains
// (lane groups, tiles, splits).  A strip's sources in one chain and the 32 NI
// terms of a reaction in another made the error of a force 1.3 to 2 times as
// large below 10000 particles.  So every 128 sources the action sums go to a
// second level in shared memory (no cost measured), with FINE a step's
// NI reaction terms are added before they join the travelling sum (three more
// adds per step, 1.3 % of the time; taken below kStripFine64, from where the kernel
// before was the CTA grid and the sums are more exact without it), and the
// reduction adds its warps' sums by halves (in order their last roundings alone
// made half of the error).  Median error of a force (eps 1e-3), the kernel before / in
// one chain, the sums in order / now: N = 4200 1.24e-16 / 1.37e-16 / 1.02e-16, 9000
// 1.31e-16 / 1.32e-16 / 1.00e-16, 14000 1.18e-16 / 1.33e-16 / 0.98e-16 (1.07e-16 without
// FINE), 65536 3.9e-16 / 1.4e-16 / 1.1e-16; masses over many decades (lognormal, one of a
// hundred 1000 times as heavy) 14000 1.83e-16 / 2.1e-16 / 1.47e-16 (1.83e-16 without; at
// eps 1e-2 1.81e-16, 1.92e-16 without).
constexpr long long kStripFine64 = 16384;
template <int NI, bool EXCL, bool FINE>
__global__ void __launch_bounds__(kStripWarps * 32, 1)
    k_strip_f64(const IParticles ip, const JStream js, const StripPlan sp, const double eps2,
                double* act, double* rea, int* err) {
  constexpr int TB = NI;
  __shared__ double src[kStripWarps][4][32];
  extern __shared__ double strip_acc[];  // [kStripWarps][3][32 NI]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = warp * gridDim.x + blockIdx.x;
  grid_dependency_wait();
  launch_dependents();
  if (g >= sp.strips) return;
  int u = strip_start(sp, g);
  const int u_end = strip_start(sp, g + 1);
  const int from = (lane + 1) & 31;
  double* acc = strip_acc + warp * (96 * NI) + lane;
  const double *bx = src[warp][0], *by = src[warp][1], *bz = src[warp][2], *bm = src[warp][3];
  for (int r = strip_row(sp, u); u < u_end; ++r) {
    const int b0 = r * TB + (u - strip_prefix(sp, r));
    const int b1 = min(sp.batches, b0 + (u_end - u));
    u += b1 - b0;
    const long long ibase = (long long)r * (32 * NI) + lane;
    const int b_rea = (r + 1) * TB;
    const long long len = 96LL * (sp.batches - b_rea);  // reactions of this row block
    if (!NBR_IN((long long)(r + 1) * (32 * NI) - 1, ip.len, err) ||
        !NBR_IN(32LL * (((b1 - 1) | 3) + 1) - 1, js.len, err) ||
        !NBR_IN((long long)(g + r - sp.r0 + 1) * (96 * NI) - 1, sp.act_doubles, err) ||
        (len > 0 && !NBR_IN(strip_rea_off(sp, r) + len - 1, sp.reactions, err)))
      return;
    double* out = rea + strip_rea_off(sp, r) + lane - 96LL * b_rea;
    double xi[NI], yi[NI], zi[NI], mi[NI], ax[NI], ay[NI], az[NI];
#pragma unroll
    for (int k = 0; k < NI; ++k) {
      const long long i = ibase + 32 * k;
      xi[k] = ip.x[i]; yi[k] = ip.y[i]; zi[k] = ip.z[i]; mi[k] = ip.m[i];
      ax[k] = ay[k] = az[k] = 0.0;
      acc[32 * k] = acc[32 * NI + 32 * k] = acc[64 * NI + 32 * k] = 0.0;
    }
    long long j = 32LL * b0 + lane;
    double qx = js.x[j], qy = js.y[j], qz = js.z[j], qm = js.m[j];
#pragma unroll 1
    for (int b = b0; b < b1; ++b) {
      __syncwarp();
      src[warp][0][lane] = qx; src[warp][1][lane] = qy;
      src[warp][2][lane] = qz; src[warp][3][lane] = qm;
      __syncwarp();
      double xs = qx, ys = qy, zs = qz, ms = qm;
      j += 32;
      if (b + 1 < b1) { qx = js.x[j]; qy = js.y[j]; qz = js.z[j]; qm = js.m[j]; }
      double RX = 0.0, RY = 0.0, RZ = 0.0;
#pragma unroll 4
      for (int step = 0; step < 32; ++step) {
        const int jn = (lane + step + 1) & 31;  // the next step's source
        const double xn = bx[jn], yn = by[jn], zn = bz[jn], mn = bm[jn];
        double tx = RX, ty = RY, tz = RZ;  // FINE: the step's reaction alone
#pragma unroll
        for (int q0 = 0; q0 < NI; q0 += 2) {
          double dx[2], dy[2], dz[2], r2[2], y3[2];
#pragma unroll
          for (int q = 0; q < 2; ++q) dx[q] = xs - xi[q0 + q];
#pragma unroll
          for (int q = 0; q < 2; ++q) dy[q] = ys - yi[q0 + q];
#pragma unroll
          for (int q = 0; q < 2; ++q) dz[q] = zs - zi[q0 + q];
#pragma unroll
          for (int q = 0; q < 2; ++q) r2[q] = fma(dx[q], dx[q], eps2);
#pragma unroll
          for (int q = 0; q < 2; ++q) r2[q] = fma(dy[q], dy[q], r2[q]);
#pragma unroll
          for (int q = 0; q < 2; ++q) r2[q] = fma(dz[q], dz[q], r2[q]);
#pragma unroll
          for (int q = 0; q < 2; ++q) y3[q] = inv_cube<EXCL>(r2[q]);
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const double sj = ms * y3[q], si = mi[q0 + q] * y3[q];
            const bool first = FINE && q0 + q == 0;
            tx = first ? si * dx[q] : fma(si, dx[q], tx);
            ty = first ? si * dy[q] : fma(si, dy[q], ty);
            tz = first ? si * dz[q] : fma(si, dz[q], tz);
            az[q0 + q] = fma(sj, dz[q], az[q0 + q]);
            ay[q0 + q] = fma(sj, dy[q], ay[q0 + q]);
            ax[q0 + q] = fma(sj, dx[q], ax[q0 + q]);
          }
        }
        RX = __shfl_sync(0xffffffffu, FINE ? RX + tx : tx, from);
        RY = __shfl_sync(0xffffffffu, FINE ? RY + ty : ty, from);
        RZ = __shfl_sync(0xffffffffu, FINE ? RZ + tz : tz, from);
        xs = xn; ys = yn; zs = zn; ms = mn;
      }
      if (b >= b_rea) {
        double* o = out + 96LL * b;
        o[0] = -RX;
        o[32] = -RY;
        o[64] = -RZ;
      }
      if ((b & 3) == 3 || b + 1 == b1) {
#pragma unroll
        for (int k = 0; k < NI; ++k) {
          acc[32 * k] += ax[k]; acc[32 * NI + 32 * k] += ay[k]; acc[64 * NI + 32 * k] += az[k];
          ax[k] = ay[k] = az[k] = 0.0;
        }
      }
    }
    double* a = act + (long long)(g + r - sp.r0) * (96 * NI) + lane;
#pragma unroll
    for (int k = 0; k < 3 * NI; ++k) a[32 * k] = acc[32 * k];
  }
}

// The potential energy of the system over -G kInvDistScale: the units of the
// strips, each unordered pair once (in a block's own batches twice, at half the
// mass), with no reaction to carry: a step's source is read from the warp's
// staging buffer by all lanes.  Per pair 3 differences, 3 fma, 4 operations of
// inv_dist and 1 fma = 11, so 5.5 per ordered pair, against 11 in k_potential_f64,
// which also gives every particle's potential.  One sum per strip, lanes in
// xor order.  us per diagnostics call on B200, every ordered pair with
// rsqrt(double) / this: N = 2000 125 / 65, 16000 377 / 167, 65500 4198 / 1657, 262144
// 64535 / 24979 (81 % of the FP64 pipe).  8 receivers per lane in one CTA of 8
// warps per SM (two such CTAs spill: 27495); below kEnergyWideN 4 in two CTAs,
// for more units.
template <int NI, bool EXCL>
__global__ void __launch_bounds__(kStripWarps * 32, NI == 4 ? 2 : 1)
    k_strip_energy(const IParticles ip, const JStream js, const StripPlan sp, const double eps2,
                   double* sums, int* err) {
  constexpr int TB = NI;
  __shared__ double2 src[kStripWarps][32][2];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = warp * gridDim.x + blockIdx.x;
  if (g >= sp.strips) return;
  int u = strip_start(sp, g);
  const int u_end = strip_start(sp, g + 1);
  double total = 0.0;
  for (int r = strip_row(sp, u); u < u_end; ++r) {
    const int b0 = r * TB + (u - strip_prefix(sp, r));
    const int b1 = min(sp.batches, b0 + (u_end - u));
    u += b1 - b0;
    const long long ibase = (long long)r * (32 * NI) + lane;
    if (!NBR_IN((long long)(r + 1) * (32 * NI) - 1, ip.len, err) ||
        !NBR_IN(32LL * b1 - 1, js.len, err))
      return;
    double xi[NI], yi[NI], zi[NI], ph[NI];
#pragma unroll
    for (int k = 0; k < NI; ++k) {
      const long long i = ibase + 32 * k;
      xi[k] = ip.x[i]; yi[k] = ip.y[i]; zi[k] = ip.z[i];
      ph[k] = 0.0;
    }
    long long j = 32LL * b0 + lane;
    double qx = js.x[j], qy = js.y[j], qz = js.z[j], qm = js.m[j];
#pragma unroll 1
    for (int b = b0; b < b1; ++b) {
      const bool own = b < (r + 1) * TB;
      __syncwarp();
      src[warp][lane][0] = make_double2(qx, qy);
      src[warp][lane][1] = make_double2(qz, own ? 0.5 * qm : qm);
      __syncwarp();
      j += 32;
      if (b + 1 < b1) { qx = js.x[j]; qy = js.y[j]; qz = js.z[j]; qm = js.m[j]; }
      // Every pair by inv_dist, then, where a r2 was zero or subnormal, the
      // whole batch again with the limit's own arithmetic.  In the block's own
      // batches receiver kself of lane `step` is the source itself: no pair.
      const int kself = own ? b - r * TB : -1;
      double keep[NI];
#pragma unroll
      for (int k = 0; k < NI; ++k) keep[k] = ph[k];
      int lo = 0x7fffffff;
      auto pairs = [&](auto self_pair, auto limit, int step) {
        const double2 a = src[warp][step][0], c = src[warp][step][1];
#pragma unroll
        for (int k = 0; k < NI; ++k) {
          const double dx = a.x - xi[k], dy = a.y - yi[k], dz = c.x - zi[k];
          double r2 = fma(dx, dx, eps2);
          r2 = fma(dy, dy, r2);
          r2 = fma(dz, dz, r2);
          const bool self = decltype(self_pair)::value && k == kself && step == lane;
          const int hi = __double2hiint(r2);
          if (!decltype(limit)::value) lo = min(lo, self ? 0x7fffffff : hi);
          double v = decltype(limit)::value && hi < kTinyHi ? inv_dist_tiny<EXCL>(r2) : inv_dist(r2);
          if (self) v = 0.0;
          ph[k] = fma(c.y, v, ph[k]);
        }
      };
      const std::true_type yes;
      const std::false_type no;
      if (own) {
#pragma unroll 2
        for (int step = 0; step < 32; ++step) pairs(yes, no, step);
      } else {
#pragma unroll 4
        for (int step = 0; step < 32; ++step) pairs(no, no, step);
      }
      if (lo < kTinyHi) {
#pragma unroll
        for (int k = 0; k < NI; ++k) ph[k] = keep[k];
#pragma unroll 1
        for (int step = 0; step < 32; ++step) pairs(yes, yes, step);
      }
    }
#pragma unroll
    for (int k = 0; k < NI; ++k) total = fma(ip.m[ibase + 32 * k], ph[k], total);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) total += __shfl_xor_sync(0xffffffffu, total, off);
  if (lane == 0) sums[g] = total;
}

// Adds the partial sums of a batch's 32 particles, one per lane: its row block's
// strips, then the reactions from the row blocks before it, spread over the
// CTA's warps (a particle's chain of loads is what takes the time on a small
// system); the warps' sums are then added by halves, one warp per axis: a fixed
// order.  By mode: 0 runs the epilogue of the large kernels, 1 stores the sums
// into dst[d * ld + i], 2 adds them to it (a launch over some of the row blocks).
//
// What bounds it: on a small system the chain of loads, on a large one the bytes
// of the reactions in flight (0.8 GB at N = 262144 FP32C).  So up to two CTAs per
// SM in all each warp has eight row blocks' loads in flight; above that four, in
// 40 registers, so that three CTAs share an SM.  The reactions lie by (row
// block, batch), 384 or 768 bytes together, which strip and reduction move as
// one piece.  us per evaluation: before (one array per component, four row
// blocks, two CTAs) / two CTAs and eight / three CTAs and four: FP32C N = 4224
// 15.6 / 15.5 / 16.4, 12001 61.1 / 60.1 / 58.1, 65536 1385 / 1375 / 1366, 262144
// 21743 / 21576 / 21510; FP64 4224 21.4 / 21.1 / 22.0, 12001 112.4 / 112.4 / 110.1,
// 16000 180.6 / 181.9 / 181.2, 196608 25214 / 25072 / 25042.
// The last sums by halves, a warp per axis, instead of one warp in order: FP64 4224 21.2 /
// 20.8, 12001 110.3 / 111.0.
constexpr int kRedWarps = 16;

template <int PREC, int PER_SM>
__global__ void __launch_bounds__(32 * kRedWarps, PER_SM)
    k_strip_reduce(const IParticles ip, const Epilogue ep, const StripPlan sp, const double* act,
                   const void* rea_v, const double scale, const int mode, double* dst,
                   const long long ld) {
  using T = typename std::conditional<PREC == kFP32C, float, double>::type;
  __shared__ double part[kRedWarps][3][32];
  const int lane = threadIdx.x & 31, ph = threadIdx.x >> 5;
  const int b = blockIdx.x;                // batch of 32 particles
  const int rb = b / sp.tb;                // its row block
  const long long i = 32LL * b + lane;
  const double f = PREC == kFP32C ? scale * mass_mantissa(ip.m[0]) : scale;
  grid_dependency_wait();
  launch_dependents();
  if (!NBR_IN(i, ip.len, ep.err)) return;
  double sx = 0.0, sy = 0.0, sz = 0.0;
  if (rb >= sp.r0 && rb < sp.r1) {
    // the strips' action sums on this row block
    const int u0 = strip_prefix(sp, rb), u1 = strip_prefix(sp, rb + 1);
    const int g0 = strip_owner(sp, u0), g1 = strip_owner(sp, u1 - 1);
    const int rows_of = 32 * sp.tb;
    const double* a = act + (long long)(g0 + ph + rb - sp.r0) * (3 * rows_of) + (i - (long long)rb * rows_of);
#pragma unroll 4
    for (int g = g0 + ph; g <= g1; g += kRedWarps) {
      sx += a[0]; sy += a[rows_of]; sz += a[2 * rows_of];
      a += 3LL * kRedWarps * rows_of;
    }
  }
  // the reactions from the row blocks before its own
  const T* rea = reinterpret_cast<const T*>(rea_v);
  const int r_end = min(rb, sp.r1);
  constexpr int kRows = PER_SM == 2 ? 8 : 4;
#pragma unroll kRows
  for (int r = sp.r0 + ph; r < r_end; r += kRedWarps) {
    const T* a = rea + strip_rea_off(sp, r) + 96LL * (b - sp.tb * (r + 1)) + lane;
    sx += (double)a[0]; sy += (double)a[32]; sz += (double)a[64];
  }
  part[ph][0][lane] = sx; part[ph][1][lane] = sy; part[ph][2][lane] = sz;
  __syncthreads();
  if (ph > 2) return;  // warp d: the sum and the epilogue of axis d
  const int d = ph;
  const double* half = &part[0][d][lane];
  double s = sum_by_halves<kRedWarps / 2>(half, 96);
  __syncwarp();  // the other half's loads after these: 40 registers
  s = f * (s + sum_by_halves<kRedWarps / 2>(half + 48 * kRedWarps, 96));
  if (mode == 1) { dst[d * ld + i] = s; return; }
  if (mode == 2) { dst[d * ld + i] += s; return; }
  if (i >= ip.n) return;
  auto finish = [&](double* a_out, double* vel, const double* x, double* xn) {
    if (ep.mode == 0) {
      a_out[i] = (ep.want_force ? ep.G * ip.m[i] : ep.G) * s;
      return;
    }
    const double g = ep.G * s;
    a_out[i] = g;
    const double u = vel[i], v = u + ep.kick * g;
    vel[i] = v;
    xn[i] = x[i] + ep.drift * (ep.mode == 2 ? u : v);
  };
  if (d == 0) finish(ep.ax, ep.vx, ip.x, ep.xn);
  else if (d == 1) finish(ep.ay, ep.vy, ip.y, ep.yn);
  else finish(ep.az, ep.vz, ip.z, ep.zn);
}

}  // namespace

StripPlan strip_plan(int precision, long long n, int r0, int r1, int sms, int ni) {
  StripPlan p;
  p.tb = ni;
  p.batches = (int)((n + 31) / 32);
  p.rows = (int)((n + 32 * ni - 1) / (32 * ni));
  p.r0 = r0;
  p.r1 = std::min(r1, p.rows);
  p.units = strip_prefix(p, p.r1);
  p.strips = std::min(p.units, sms * kStripWarps);
  p.share = p.units / p.strips;
  p.longer = p.units % p.strips;
  p.act_doubles = ((long long)p.strips + p.r1 - p.r0) * 96 * ni;
  // the last row block's own batches end at or after the last batch
  p.reactions = strip_rea_off(p, p.r1) +
                (p.r1 == p.rows ? 96LL * ((long long)p.tb * p.rows - p.batches) : 0);
  p.doubles = p.act_doubles + (precision == kFP32C ? (p.reactions + 1) / 2 : p.reactions);
  return p;
}

// Receivers per lane for a whole system of n particles: the width whose
// strips a model finishes first.  More receivers per lane run a unit faster
// per pair, fewer make the units smaller, so that the longest strips are
// nearer to the mean.  A unit takes `unit` us of an SM with all its warps at
// work (from the rate at N = 262144); the last units of the longer strips, k
// warps of an SM at one unit each, take as long as two warps per
// scheduler, or one alone at `lone` of the full rate.  Over 33 sizes from
// 4224 to 65000 this gives each width's time to 0.6 % (FP64) and 1.5 % (FP32C)
// on average, with 11 to 13 us for the two launches and their latencies, and
// these three widths are within 0.3 % of the best of eleven (4 to 16
// receivers, 8 to 16 warps).
int strip_choose(int precision, long long n, int sms) {
  struct Width { int ni; double unit, lone; };
  static const Width w32[] = {{16, 1.534, 0.75}, {10, 0.997, 0.9}, {8, 0.844, 0.8}};
  static const Width w64[] = {{10, 1.962, 0.9}, {8, 1.589, 0.9}, {6, 1.217, 0.8}};
  int best = 0;
  double best_t = 0.0;
  for (const Width& w : precision == kFP32C ? w32 : w64) {
    const double rows = std::ceil((double)n / (32 * w.ni)), batches = std::ceil((double)n / 32);
    const double units = rows * batches - w.ni * rows * (rows - 1) / 2;
    const double strips = std::min(units, (double)sms * kStripWarps);
    const double share = std::floor(units / strips), longer = units - share * strips;
    const int last = (int)std::ceil((units < (double)sms * kStripWarps ? strips : longer) / sms);
    const double full = units < (double)sms * kStripWarps ? 0.0 : share * kStripWarps;
    const int layers = (last + 3) / 4;
    const double t = w.unit * (full + (layers == 1 ? 4.0 / w.lone : 4.0 * layers));
    if (!best || t < best_t) {
      best_t = t;
      best = w.ni;
    }
  }
  return best;
}

// Row blocks of each launch of an evaluation: all of them where the partial
// sums fit single_max (kN3SingleMaxDoubles), else launches of at most kN3SliceMaxDoubles
// (bands > 0: that many launches, for the tests).
std::vector<int> strip_bands(int precision, long long n, int sms, int ni, int bands,
                             long long single_max) {
  const int rows = (int)((n + 32 * ni - 1) / (32 * ni));
  std::vector<int> cut{0};
  if (bands > 0) {
    for (int k = 1; k <= bands; ++k) {
      const int r = (int)((long long)rows * k / bands);
      if (r > cut.back()) cut.push_back(r);
    }
    return cut;
  }
  // the reactions of rows r0 .. r1 - 1 as in strip_plan, without its 32-bit units
  auto doubles = [&](long long r0, long long r1) {
    const long long batches = (n + 31) / 32;
    const long long units = (r1 - r0) * batches - ni * ((r1 * (r1 + 1) - r0 * (r0 + 1)) / 2);
    return ((long long)sms * kStripWarps + r1 - r0) * 96 * ni +
           96 * (std::max(0LL, units) + ni) / (precision == kFP32C ? 2 : 1);
  };
  if (doubles(0, rows) <= single_max) {
    cut.push_back(rows);
    return cut;
  }
  while (cut.back() < rows) {
    int r = cut.back() + 1;
    while (r < rows && doubles(cut.back(), r + 1) <= kN3SliceMaxDoubles) ++r;
    cut.push_back(r);
  }
  return cut;
}

namespace {

template <int NI>
const void* strip_f32c(bool excl) {
  return excl ? (const void*)k_strip_f32c<NI, true> : (const void*)k_strip_f32c<NI, false>;
}
template <int NI>
const void* strip_f64(bool excl, bool fine) {
  if (fine) return excl ? (const void*)k_strip_f64<NI, true, true> : (const void*)k_strip_f64<NI, false, true>;
  return excl ? (const void*)k_strip_f64<NI, true, false> : (const void*)k_strip_f64<NI, false, false>;
}
const void* strip_fn(int precision, int ni, bool excl, long long n) {
  if (precision == kFP32C)
    return ni == 8 ? strip_f32c<8>(excl) : ni == 10 ? strip_f32c<10>(excl)
                                         : ni == 16 ? strip_f32c<16>(excl) : nullptr;
  const bool fine = n < kStripFine64;
  return ni == 6 ? strip_f64<6>(excl, fine) : ni == 8 ? strip_f64<8>(excl, fine)
                                            : ni == 10 ? strip_f64<10>(excl, fine) : nullptr;
}

// The action sums of every warp's row block.
size_t strip_smem(int ni) { return (size_t)kStripWarps * 96 * ni * sizeof(double); }

}  // namespace

cudaError_t launch_energy(long long n, double eps2, const IParticles& ip, const JStream& js, int* err,
                          double* sums, int sms, int* count, cudaStream_t st) {
  const int ni = n < kEnergyWideN ? 4 : 8, grid = (ni == 4 ? 2 : 1) * sms;
  const StripPlan p = strip_plan(kFP64, n, 0, 1 << 30, grid, ni);
  *count = p.strips;
  if (eps2 == 0.0) {
    if (ni == 4) k_strip_energy<4, true><<<grid, kStripWarps * 32, 0, st>>>(ip, js, p, 0.0, sums, err);
    else k_strip_energy<8, true><<<grid, kStripWarps * 32, 0, st>>>(ip, js, p, 0.0, sums, err);
  } else {
    if (ni == 4) k_strip_energy<4, false><<<grid, kStripWarps * 32, 0, st>>>(ip, js, p, eps2, sums, err);
    else k_strip_energy<8, false><<<grid, kStripWarps * 32, 0, st>>>(ip, js, p, eps2, sums, err);
  }
  return cudaGetLastError();
}

cudaError_t prepare_strips(int precision, long long n, int ni) {
  cudaError_t e = cudaSuccess;
  for (bool excl : {false, true}) {
    const void* fn = strip_fn(precision, ni, excl, n);
    if (!fn) return cudaErrorInvalidValue;
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)strip_smem(ni));
  }
  return e;
}

cudaError_t launch_strips(int precision, const StripPlan& p, double eps2, const IParticles& ip,
                          const JStream& js, const Epilogue& ep, double* scratch, int sms, int mode,
                          double* dst, long long ld, cudaStream_t st) {
  const void* fn = strip_fn(precision, p.tb, eps2 == 0.0, ip.n);
  if (!fn) return cudaErrorInvalidValue;
  IParticles a0 = ip;
  JStream a1 = js;
  StripPlan a2 = p;
  float e32 = (float)eps2;
  double e64 = eps2;
  double* act = scratch;
  void* rea = scratch + p.act_doubles;
  int* err = ep.err;
  void* args[] = {&a0, &a1, &a2, precision == kFP32C ? (void*)&e32 : (void*)&e64, &act, &rea, &err};
  cudaLaunchAttribute serial{};
  serial.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  serial.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(sms);
  cfg.blockDim = dim3(kStripWarps * 32);
  cfg.dynamicSmemBytes = strip_smem(p.tb);
  cfg.stream = st;
  cfg.attrs = &serial;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
  if (e != cudaSuccess) return e;
  cfg.gridDim = dim3(p.batches);
  cfg.blockDim = dim3(32 * kRedWarps);
  cfg.dynamicSmemBytes = 0;
  const void* sums = rea;
  const bool small = p.batches <= 2 * sms;
  if (precision == kFP32C)
    return cudaLaunchKernelEx(&cfg, small ? k_strip_reduce<kFP32C, 2> : k_strip_reduce<kFP32C, 3>, ip,
                              ep, p, (const double*)act, sums, 1.0 / ((double)kC53 - 1.0), mode, dst, ld);
  return cudaLaunchKernelEx(&cfg, small ? k_strip_reduce<kFP64, 2> : k_strip_reduce<kFP64, 3>, ip, ep,
                            p, (const double*)act, sums, kInvCubeScale, mode, dst, ld);
}

}  // namespace nbr
