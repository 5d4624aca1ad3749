// Shared device helpers for the accusim_b200 kernels (sm_100a).
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include "accusim_b200.h"

#define ACS_MAX_SPECIES 8

namespace acs {

constexpr int kBlock = 256;

__host__ __device__ inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// IEEE round-to-nearest FP64 operations that the compiler may not contract into FMAs. They give the
// reference's NumPy expressions bit for bit.
__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double div(double a, double b) { return __ddiv_rn(a, b); }

// d -= box * np.round(d / box)   (np.round: half to even == rint)
__device__ __forceinline__ double min_image(double d, double box) { return sub(d, mul(box, rint(div(d, box)))); }

// The same, bit for bit, without the division for almost every pair. A difference below 0.49 box (compared through
// the high words, on the integer pipe) has k = 0 and stays as it is. Otherwise t = d (1/box) differs from the IEEE
// quotient d / box by under 3e-16 |d / box|, and rint only changes at half-integers, so rint(t) is rint(d / box)
// unless t lies within 1e-9 of a half-integer (or |t| is huge); there the quotient decides as in the reference. rint
// by adding and subtracting 1.5 2^52 (round to nearest even, exact for |t| < 2^51): two additions at the full FP64
// rate, where the rint and trunc instructions run at a quarter of it or less.
static __device__ __noinline__ double min_image_quotient(double d, double box) { return min_image(d, box); }
__device__ __forceinline__ double image1(double d, double box, double inv_box, int near_hi) {
  if ((__double2hiint(d) & 0x7fffffff) < near_hi) return d;
  const double t = d * inv_box;
  const double k0 = sub(add(t, 6755399441055744.0), 6755399441055744.0);
  if (fabs(t - k0) < 0.5 - 1e-9 && fabs(t) < 1e6) return sub(d, mul(box, k0));
  return min_image_quotient(d, box);   // out of line: rare, and its registers stay out of the pair loops
}

// np.einsum("ij,ij->i") over 3 components, summed left to right without FMA.
__device__ __forceinline__ double norm2(double dx, double dy, double dz) {
  return add(add(mul(dx, dx), mul(dy, dy)), mul(dz, dz));
}

// A box with the constants the pair kernels' minimum image uses; an edge that is not a positive number takes the
// quotient everywhere.
struct ImageBox {
  double L[3], inv[3];
  // high words of 0.49 L (differences below it are their own minimum image) and, for image3_any, of 0.49999 L, 0.50001 L
  // and 1.49999 L (between the last two the image is one box away)
  int near_hi[3], below_hi[3], above_hi[3], limit_hi[3];
  int periodic;
};

inline ImageBox image_box(const double* edges3, int periodic) {
  ImageBox b;
  for (int k = 0; k < 3; ++k) {
    b.L[k] = edges3 ? edges3[k] : 0.0;
    b.inv[k] = b.L[k] != 0.0 ? 1.0 / b.L[k] : 0.0;
    const double L = b.L[k] > 0.0 && b.L[k] <= 1e300 ? b.L[k] : 0.0;
    auto high = [](double x) {
      uint64_t bits;
      memcpy(&bits, &x, 8);
      return (int)(bits >> 32);
    };
    b.near_hi[k] = high(0.49 * L);
    b.below_hi[k] = high(0.49999 * L);
    b.above_hi[k] = high(0.50001 * L) + 1;
    b.limit_hi[k] = high(1.49999 * L);
  }
  b.periodic = periodic && edges3;
  return b;
}

// Whether a difference is its own minimum image on every axis, by the high words alone.
__device__ __forceinline__ bool near_image(double dx, double dy, double dz, const ImageBox& b) {
  return (__double2hiint(dx) & 0x7fffffff) < b.near_hi[0] && (__double2hiint(dy) & 0x7fffffff) < b.near_hi[1] &&
         (__double2hiint(dz) & 0x7fffffff) < b.near_hi[2];
}

__device__ __forceinline__ void image3(double& dx, double& dy, double& dz, const ImageBox& b) {
  if (b.periodic) {
    dx = image1(dx, b.L[0], b.inv[0], b.near_hi[0]);
    dy = image1(dy, b.L[1], b.inv[1], b.near_hi[1]);
    dz = image1(dz, b.L[2], b.inv[2], b.near_hi[2]);
  }
}

// 1/x for normal positive x by Newton-Raphson from the hardware's FP64 reciprocal approximation (about 20 bits): after the
// first quadratic step (40 bits) the second's residual is exact in its FMA, so the result is the rounded reciprocal but for
// ties. x = 0 gives NaN through inf * 0.
__device__ __forceinline__ double recip(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(fma(-x, y, 1.0), y, y);
  return fma(fma(-x, y, 1.0), y, y);
}

// sqrt(x) and its reciprocal by Goldschmidt's coupled iteration (Markstein, "Software division and square root using
// Goldschmidt's algorithms", 2004) from the hardware's FP64 approximation (about 20 bits): one step gives 39 bits of both,
// then a residual that is exact in its FMA finishes each, so the root is the IEEE one and ir the rounded reciprocal of
// that root, but for ties. Two results for 10 operations. Zero, subnormal and huge x (rare) take the IEEE operations.
static __device__ __noinline__ double sqrt_recip_ieee(double x, double& ir) {
  const double r = sqrt(x);
  ir = 1.0 / r;
  return r;
}
__device__ __forceinline__ double sqrt_recip(double x, double& ir) {
  if ((unsigned)(__double2hiint(x) - 0x08000000) >= 0x70000000u) return sqrt_recip_ieee(x, ir);   // not in 2^[-895, 897)
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  double g = x * y, h = 0.5 * y;
  const double e = fma(-g, h, 0.5);
  g = fma(g, e, g);
  h = fma(h, e, h);
  const double r = fma(fma(-g, g, x), h, g), y1 = h + h;
  ir = fma(fma(-r, y1, 1.0), y1, y1);
  return r;
}

// The smallest double whose IEEE square root is at least r: r2 < square_reaching(r) decides as sqrt(r2) < r does.
inline double square_reaching(double r) {
  double t = r * r;
  while (t > 0.0 && sqrt(t) >= r) t = nextafter(t, 0.0);
  while (sqrt(t) < r) t = nextafter(t, HUGE_VAL);
  return t;
}

// erfc(x) and exp(-x^2), x = alpha r >= 0, from a Chebyshev series of exp(x^2) erfc(x) over the whole half line in a rational
// variable (the method of Shepherd and Laframboise, Math. Comp. 36, 1981). Here the variable vanishes with x: with
// s = x / (x + 2), exp(x^2) erfc(x) (x + 2) = 2 + s h(s), and h, computed in 50 digits to degree 24 over [0, 27.5] (the
// exponential is zero beyond), is within 1.4e-16, its coefficients' rounding. Below x = 0.6 the same h is summed as
// 1 + s (h / (x + 2) - 1), whose error goes to half a unit with x; above, as (2 + s h) / (x + 2).
// Its error in units of 2^-53 (10^5 points per range against quad precision, of this code transcribed with libm's
// exponential): root mean square 0.5 at x -> 0, 1.3 up to 2.4, 1.5 up to 5; largest 5.1 and 6.3, and 9 on the tail beyond.
// A series in (x - 3.75) / (x + 3.75) took the rounding of its argument near x = 0 (1.9, largest 7.2).
// The product alpha r is rounded too, a relative error that erfc and the exponential take 2 x^2 fold: its low part goes
// into the exponential for three operations. The force of one DSF pair (alpha rc = 2.4) is off by 1.6 to 1.8 units of its
// terms at all distances up to 0.8 rc, against 1.6 to 2.8 with erfc and exp of the rounded product, and 1.7 to 3.7 with the
// series above; of one Ewald pair (alpha rc = 4) by 1.2 to 1.6, against 1.3 to 8.9 and 1.6 to 15.
// One set of coefficients and no branch on ranges, so a warp's pairs stay together, and the exponential is the one the
// forces need anyway. 8000 ions' Ewald sum 418 -> 441 us, the 4096-ion force call 144.4 -> 146.3 us with this and
// sqrt_recip, for the accuracy.
__device__ __forceinline__ double erfc_exp(double alpha, double r, double& gauss) {
  double x = alpha * r;
  x = __double2hiint(x) < 0x408f4000 ? x : 1e3;   // both are zero from 39 on
  const double x2 = x * x;
  const double g = exp(-x2);
  // the roundings of alpha r (whose 2 x^2 fold is the largest error of a distant pair) and of x^2
  gauss = fma(-g, fma(x + x, fma(alpha, r, -x), fma(x, x, -x2)), g);
  const double w = recip(x + 2.0), s = x * w;
  const double t = fma(2.1454545454545455, s, -1.0), t2 = t * t;   // s in [0, 27.5 / 29.5] to [-1, 1]
  double a = -7.03276698885457419e-10;
  a = fma(a, t2, 3.69827855338635472e-09);
  a = fma(a, t2, 4.27993055151075388e-09);
  a = fma(a, t2, -9.77940454227550041e-08);
  a = fma(a, t2, 3.31218823208566288e-07);
  a = fma(a, t2, 3.32783527978017621e-07);
  a = fma(a, t2, -8.39035049546208681e-06);
  a = fma(a, t2, 4.51999891448717694e-05);
  a = fma(a, t2, -1.37057017009071884e-04);
  a = fma(a, t2, 3.94944399220502703e-05);
  a = fma(a, t2, 3.03160715558250648e-03);
  a = fma(a, t2, -1.16325487326915597e-02);
  a = fma(a, t2, -1.99641985249578879e+00);
  double b = -1.57096167960187793e-09;
  b = fma(b, t2, 1.41665436886721111e-08);
  b = fma(b, t2, -4.57254387984705977e-08);
  b = fma(b, t2, -2.97566004091487844e-08);
  b = fma(b, t2, 8.57659805297907151e-07);
  b = fma(b, t2, -3.35487926425173185e-06);
  b = fma(b, t2, 6.31148301325306036e-07);
  b = fma(b, t2, 7.58170834748642645e-05);
  b = fma(b, t2, -6.65704094465739086e-04);
  b = fma(b, t2, 4.75080620679196094e-03);
  b = fma(b, t2, -4.10826625607029136e-02);
  b = fma(b, t2, 5.45359367176469600e-01);
  const double h = fma(b, t, a);
  const bool small = __double2hiint(x) < 0x3fe33333;   // x < 0.6
  const double f = small ? fma(s, fma(h, w, -1.0), 1.0) : w * fma(s, h, 2.0);
  return f * gauss;
}

// An atom's position and one more value (species or charge) as one 32-byte sector, read by one 256-bit load: a pair
// loop that gathers from the caller's arrays touches up to four sectors per neighbour in four loads.
struct __align__(32) Packed {
  double x, y, z, w;
};

__device__ __forceinline__ Packed ld_packed(const Packed* p) {
  Packed v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}

// image3 for pairs that cross the box as often as not (all pairs of a periodic system): the choice between no shift and one
// box by the high words, one addition per axis; anything else (within 1e-5 of half a box, unwrapped atoms) by image3. The
// same results bit for bit.
__device__ __forceinline__ void image3_any(double& dx, double& dy, double& dz, const ImageBox& b) {
  const int hx = __double2hiint(dx) & 0x7fffffff, hy = __double2hiint(dy) & 0x7fffffff, hz = __double2hiint(dz) & 0x7fffffff;
  const bool nx = hx < b.below_hi[0], ny = hy < b.below_hi[1], nz = hz < b.below_hi[2];
  if ((nx || (hx >= b.above_hi[0] && hx < b.limit_hi[0])) && (ny || (hy >= b.above_hi[1] && hy < b.limit_hi[1])) &&
      (nz || (hz >= b.above_hi[2] && hz < b.limit_hi[2]))) {
    dx = sub(dx, nx ? 0.0 : copysign(b.L[0], dx));
    dy = sub(dy, ny ? 0.0 : copysign(b.L[1], dy));
    dz = sub(dz, nz ? 0.0 : copysign(b.L[2], dz));
  } else {
    image3(dx, dy, dz, b);
  }
}

// Neighbour-list slot: warp-interleaved so that a warp of consecutive atoms reads 128 contiguous bytes.
__host__ __device__ __forceinline__ int64_t nbr_slot(int64_t i, int k, int maxnb) {
  return (i >> 5) * (int64_t)maxnb * 32 + (int64_t)k * 32 + (i & 31);
}

// The screen of one candidate per lane against the warp's staged home atoms (hx, hy, hz: 32 negated coordinates each, 16-byte
// aligned, all 32 set): bit h of the result says r^2 <= lo for home atom h < nh (bits from nh on mean nothing), and
// `band` that some r^2 is not surely outside (mid - half, mid + half), the interval that needs the exact filter; a NaN is
// not. Four home atoms per round, two per packed FP32 operation (each half the IEEE scalar operation), one predicated bit
// each: about 8 instructions per home atom, where two ballots and two selects per home atom took 12 (the engine's 1M-atom
// list build 0.72 -> 0.59 ms with a bounded loop over each atom's accepted candidates).
__device__ __forceinline__ uint32_t screen_homes(const float4& o, const float* hx, const float* hy, const float* hz, int nh,
                                                 float lo, float mid, float half, bool& band) {
  const float2 px = make_float2(o.x, o.x), py = make_float2(o.y, o.y), pz = make_float2(o.z, o.z);
  const float2 m2 = make_float2(-mid, -mid);
  uint32_t m = 0u;
  bool b = false;
#pragma unroll 2
  for (int h = 0; h < nh; h += 4) {
    const float4 X = *reinterpret_cast<const float4*>(hx + h), Y = *reinterpret_cast<const float4*>(hy + h),
                 Z = *reinterpret_cast<const float4*>(hz + h);
    const float2 x0 = __fadd2_rn(px, make_float2(X.x, X.y)), x1 = __fadd2_rn(px, make_float2(X.z, X.w));
    const float2 y0 = __fadd2_rn(py, make_float2(Y.x, Y.y)), y1 = __fadd2_rn(py, make_float2(Y.z, Y.w));
    const float2 z0 = __fadd2_rn(pz, make_float2(Z.x, Z.y)), z1 = __fadd2_rn(pz, make_float2(Z.z, Z.w));
    const float2 q0 = __ffma2_rn(z0, z0, __ffma2_rn(y0, y0, __fmul2_rn(x0, x0)));
    const float2 q1 = __ffma2_rn(z1, z1, __ffma2_rn(y1, y1, __fmul2_rn(x1, x1)));
    const float2 t0 = __fadd2_rn(q0, m2), t1 = __fadd2_rn(q1, m2);
    uint32_t four = q0.x <= lo ? 1u : 0u;
    if (q0.y <= lo) four |= 2u;
    if (q1.x <= lo) four |= 4u;
    if (q1.y <= lo) four |= 8u;
    m |= four << h;
    b = b || !(fabsf(t0.x) >= half) || !(fabsf(t0.y) >= half) || !(fabsf(t1.x) >= half) || !(fabsf(t1.y) >= half);
  }
  band = b;
  return m;
}

// Transpose of a warp's 32 x 32 bits: bit c of lane r's result is bit r of lane c's value.
__device__ __forceinline__ uint32_t transpose_bits(uint32_t v, int lane) {
#pragma unroll
  for (int j = 16; j > 0; j >>= 1) {
    const uint32_t low = j == 16 ? 0x0000ffffu : j == 8 ? 0x00ff00ffu : j == 4 ? 0x0f0f0f0fu : j == 2 ? 0x33333333u : 0x55555555u;
    const uint32_t y = __shfl_xor_sync(0xffffffffu, v, j);
    const bool up = lane & j;
    const uint32_t keep = up ? ~low : low;
    v = (v & keep) | (__funnelshift_l(y, y, up ? 32 - j : j) & ~keep);
  }
  return v;
}

// Deterministic block reduction of W doubles per thread into partials[blockIdx][W]; the last block to
// finish (ticket) sums the partials into out[W] in a fixed order (thread t takes blocks t, t + blockDim, ..., then
// the same block reduction) and resets the ticket. The last block's sum is what the kernel's other blocks wait for:
// one thread walking the partials took 0.1 ms of the LJ force and 0.2 ms of the conserved sums at 4096 blocks (1M atoms);
// the whole block takes a few microseconds (10-step loop of the FP64 level at 1M atoms: 8.7 -> 7.6 ms).
template <int W>
__device__ __forceinline__ void block_sum(const double (&v)[W], double (*sh)[kBlock / 32], double (&out)[W]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    double x = v[w];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[w][wid] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) {
      double s = 0.0;
      for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += sh[w][k];
      out[w] = s;
    }
  }
}

template <int W>
__device__ void block_sum_finish(const double (&v)[W], double* partials, unsigned int* ticket, double* out) {
  __shared__ double sh[W][kBlock / 32];
  __shared__ bool last;
  double s[W];
  block_sum<W>(v, sh, s);
  if (gridDim.x == 1) {   // nothing to wait for
    if (threadIdx.x == 0) {
#pragma unroll
      for (int w = 0; w < W; ++w) out[w] = s[w];
    }
    return;
  }
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) partials[(int64_t)blockIdx.x * W + w] = s[w];
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int w = 0; w < W; ++w) s[w] = 0.0;
  for (unsigned int b = threadIdx.x; b < gridDim.x; b += blockDim.x) {
#pragma unroll
    for (int w = 0; w < W; ++w) s[w] += __ldcg(partials + (int64_t)b * W + w);
  }
  double r[W];
  block_sum<W>(s, sh, r);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 0; w < W; ++w) out[w] = r[w];
    *ticket = 0u;
  }
}

inline int launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? ACS_OK : ACS_ERR_CUDA;
}

}  // namespace acs
