// Shared device helpers for the accusim_b200 kernels (sm_100a).
#pragma once
#include <cuda_runtime.h>
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

// The same, bit for bit, with a multiply by 1/box in place of the division for almost every pair: t = d (1/box)
// differs from the IEEE quotient d / box by under 3e-16 |d / box|, and rint only changes at half-integers, so
// rint(t) is rint(d / box) unless t lies within 1e-9 of a half-integer (or |t| is huge); there the quotient
// decides as in the reference.
__device__ __forceinline__ double min_image(double d, double box, double inv_box) {
  const double t = d * inv_box;
  const double f = fabs(t - trunc(t));
  const double k = (fabs(f - 0.5) > 1e-9 && fabs(t) < 1e6) ? rint(t) : rint(div(d, box));
  return sub(d, mul(box, k));
}

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

struct Box3 {
  double L[3];
  double inv[3];   // 1 / L, for min_image's multiply
  int periodic;
};

// A box with the constants the pair kernels' minimum image uses; an edge that is not a positive number takes the
// quotient everywhere.
struct ImageBox {
  double L[3], inv[3];
  int near_hi[3];  // high word of 0.49 L: differences below it are their own minimum image
  int periodic;
};

inline ImageBox image_box(const double* edges3, int periodic) {
  ImageBox b;
  for (int k = 0; k < 3; ++k) {
    b.L[k] = edges3 ? edges3[k] : 0.0;
    b.inv[k] = b.L[k] != 0.0 ? 1.0 / b.L[k] : 0.0;
    const double near_d = b.L[k] > 0.0 && b.L[k] <= 1e300 ? 0.49 * b.L[k] : 0.0;
    uint64_t bits;
    memcpy(&bits, &near_d, 8);
    b.near_hi[k] = (int)(bits >> 32);
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

__device__ __forceinline__ void min_image3(double& dx, double& dy, double& dz, const Box3& b) {
  if (b.periodic) {
    dx = min_image(dx, b.L[0], b.inv[0]);
    dy = min_image(dy, b.L[1], b.inv[1]);
    dz = min_image(dz, b.L[2], b.inv[2]);
  }
}

// Neighbour-list slot: warp-interleaved so that a warp of consecutive atoms reads 128 contiguous bytes.
__host__ __device__ __forceinline__ int64_t nbr_slot(int64_t i, int k, int maxnb) {
  return (i >> 5) * (int64_t)maxnb * 32 + (int64_t)k * 32 + (i & 31);
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
