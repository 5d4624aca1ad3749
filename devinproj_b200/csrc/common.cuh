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

// 1/x for normal positive x by Newton-Raphson from the hardware's FP64 reciprocal approximation (about 20 bits): two
// quadratic steps, the second's residual exact in its FMA, leave under 1 ulp. x = 0 gives NaN through inf * 0.
__device__ __forceinline__ double recip(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(fma(-x, y, 1.0), y, y);
  return fma(fma(-x, y, 1.0), y, y);
}

// 1/sqrt(x) for normal positive x: the hardware approximation (about 20 bits) and one step of the third-order iteration
// y (1 + e/2 + 3 e^2/8), e = 1 - x y^2; within 2 ulp.
__device__ __forceinline__ double recip_sqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(fma(0.375, e, 0.5), y * e, y);
}

// The smallest double whose IEEE square root is at least r: r2 < square_reaching(r) decides as sqrt(r2) < r does.
inline double square_reaching(double r) {
  double t = r * r;
  while (t > 0.0 && sqrt(t) >= r) t = nextafter(t, 0.0);
  while (sqrt(t) < r) t = nextafter(t, HUGE_VAL);
  return t;
}

// erfc(x) and exp(-x^2) for x >= 0. (1 + 2x) exp(x^2) erfc(x) is a smooth function of t = (x - k) / (x + k) over the
// whole half line (Shepherd and Laframboise, Math. Comp. 36, 1981): with k = 3.75 its Chebyshev series, computed here
// in extended precision to degree 23 and summed as two chains in t^2, is within 5.5e-17; the result is within 3 ulp of
// erfc (measured against 40 digits over [0, 8]). No ranges, so a warp's pairs stay together, and the exponential is the
// one the forces need anyway: about half of the operations of erfc and exp apart.
__device__ __forceinline__ double erfc_exp(double x, double& gauss) {
  x = fmin(x, 1e3);   // both are zero from 39 on
  const double s = x * x;
  const double g = exp(-s);
  gauss = fma(-g, fma(x, x, -s), g);   // the rounding of x^2
  const double u = fma(2.0, x, 1.0), w = x + 3.75;
  const double r = recip(u * w);
  const double t = (x - 3.75) * u * r, t2 = t * t;
  double a = -2.62310734713347593e-09;
  a = fma(a, t2, 3.19792667166680421e-08);
  a = fma(a, t2, -2.48571262480167447e-07);
  a = fma(a, t2, 1.74198215862248163e-06);
  a = fma(a, t2, -1.14380480333468935e-05);
  a = fma(a, t2, 5.16465297417741622e-05);
  a = fma(a, t2, 2.93714378044958009e-04);
  a = fma(a, t2, -9.74657968326526208e-03);
  a = fma(a, t2, -5.86933985766493402e-02);
  a = fma(a, t2, -1.08803930142444619e-01);
  a = fma(a, t2, 3.58541548547902569e-03);
  a = fma(a, t2, 1.23751263083782748e+00);
  double b = 3.11143338097992545e-10;
  b = fma(b, t2, -3.74421008096201827e-09);
  b = fma(b, t2, 2.32635087088591238e-08);
  b = fma(b, t2, -5.72182306032240859e-08);
  b = fma(b, t2, -9.73559896736774970e-07);
  b = fma(b, t2, 2.23842391550822306e-05);
  b = fma(b, t2, -2.90154080540841724e-04);
  b = fma(b, t2, 1.75562585289529543e-03);
  b = fma(b, t2, 2.83622774189564060e-02);
  b = fma(b, t2, 9.23043211603774838e-02);
  b = fma(b, t2, 8.22767384901452042e-02);
  b = fma(b, t2, -1.40240598585546966e-01);
  return fma(b, t, a) * (w * r) * gauss;
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
