// FP64 Ewald summation on the device (accusim/forces.py:333-388): real-space erfc sum over minimum-image
// pairs inside rcut, reciprocal-space sum over the caller's k-vectors and weights, self term.
// Deterministic: every reduction runs in a fixed order.
#include <math.h>

#include <algorithm>

#include "accusim_b200_mlp.h"
#include "common.cuh"

using namespace acs;

namespace {

constexpr int kSChunks = 64;   // structure-factor partial sums per k-vector
constexpr int kTab = 17;       // e^{2 pi i m x / L} per axis, m = 0 .. 16
constexpr int kCube = 2 * kTab - 1;
constexpr int kAtoms = 32;     // atoms of a block: one per lane, the block's 8 warps share their partners or k-vectors
constexpr int kWarps = kBlock / 32;

struct EwaldPar {
  ImageBox box;
  double a, r2cut, c2a, pref_f, k;
  int K;
};

// What the k-vectors are. A k-vector set of the reference's form, 2 pi m / L with integers |m| <= 16, each with its mirror
// image, lets e^{i k r} be a product of three tabulated factors and needs half of the vectors; any other set takes
// sine and cosine per atom and vector. Decided on the device on each call, since the vectors are there.
struct KForm {
  int general;      // not such a set
};

__device__ __forceinline__ int cube_at(int x, int y, int z) {
  return ((x + kTab - 1) * kCube + (y + kTab - 1)) * kCube + (z + kTab - 1);
}

// Integer coordinates of every k-vector, packed (x + 16) | (y + 16) << 8 | (z + 16) << 16, and the cube's index of it; also
// packs positions and charges and clears the ticket.
__global__ void k_prepare(const double* __restrict__ pos, const double* __restrict__ q, int64_t n,
                          const double* __restrict__ kv, const __grid_constant__ EwaldPar P, Packed* __restrict__ pk,
                          int32_t* __restrict__ kn, int32_t* __restrict__ cube, KForm* form, unsigned int* ticket) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t == 0) *ticket = 0u;
  if (t < n) {
    Packed v;
    v.x = pos[3 * t];
    v.y = pos[3 * t + 1];
    v.z = pos[3 * t + 2];
    v.w = q[t];
    pk[t] = v;
  }
  if (t >= P.K) return;
  int m[3];
  bool ok = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double k = kv[3 * t + d], r = rint(k * P.box.L[d] / (2.0 * M_PI));
    ok = ok && fabs(r) < kTab && fabs(k - 2.0 * M_PI * r / P.box.L[d]) <= 4.5e-16 * fabs(k);
    m[d] = ok ? (int)r : 0;
  }
  if (!ok) {
    form->general = 1;
    return;
  }
  kn[t] = (m[0] + 16) | (m[1] + 16) << 8 | (m[2] + 16) << 16;
  cube[cube_at(m[0], m[1], m[2])] = (int32_t)t + 1;
}

// Every vector alone in its place of the cube (a repeated one is not) and with its mirror image; the weight of a pair.
__global__ void k_pair_vectors(const int32_t* __restrict__ kn, const int32_t* __restrict__ cube, int K,
                               const double* __restrict__ w, double* __restrict__ wfold, KForm* form) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K || form->general) return;
  const int x = (kn[k] & 255) - 16, y = (kn[k] >> 8 & 255) - 16, z = (kn[k] >> 16 & 255) - 16;
  const int mirror = cube[cube_at(-x, -y, -z)];
  if (cube[cube_at(x, y, z)] != k + 1 || mirror == 0) form->general = 1;
  // one vector of each pair stands for both
  const bool half = x > 0 || (x == 0 && (y > 0 || (y == 0 && z >= 0)));
  wfold[k] = !half ? 0.0 : (mirror == k + 1 || mirror == 0 ? w[k] : w[k] + w[mirror - 1]);
}

// table[atom][axis][m] = e^{2 pi i m x / L}
__global__ void k_phases(const Packed* __restrict__ pk, int64_t n, const __grid_constant__ EwaldPar P,
                         const KForm* __restrict__ form, double2* __restrict__ table) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * 3 * kTab || form->general) return;
  const int64_t i = t / (3 * kTab);
  const int r = (int)(t - i * 3 * kTab), d = r / kTab, m = r - d * kTab;
  const double* x = reinterpret_cast<const double*>(pk + i);
  double s, c;
  sincos(x[d] * (2.0 * M_PI * m / P.box.L[d]), &s, &c);
  table[t] = make_double2(c, s);
}

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(fma(-a.y, b.y, a.x * b.x), fma(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ double2 conj_if(double2 a, bool neg) { return make_double2(a.x, neg ? -a.y : a.y); }

// partial[c][k] = sum_{j in chunk c} q_j (cos, sin)(k . r_j)     (accusim/forces.py:382-383). A thread per k-vector, 32
// atoms at a time. The block's vectors share few pairs of the first two coordinates (runs along the last axis): the
// products q e^{ikx x} e^{iky y} of up to kRuns runs are formed once per atom in shared memory, and a vector adds the
// four real products with e^{ikz z}, 4 FP64 operations and two reads per atom and pair of mirrored vectors (three
// factors per vector, 10 operations and three reads: 69 us at 8000 ions and 7152 vectors, 50 here; a sine and cosine
// per atom and vector 226). More runs than that in a block form the three factors per vector.
constexpr int kRuns = 32;
__global__ void __launch_bounds__(kBlock) k_sfac_partial(const Packed* __restrict__ pk, int64_t n,
                                                         const double* __restrict__ kv, const int32_t* __restrict__ kn,
                                                         const double* __restrict__ wfold, int K,
                                                         const double2* __restrict__ table,
                                                         const KForm* __restrict__ form, double2* __restrict__ partial) {
  __shared__ double2 ez[kAtoms][kTab];
  __shared__ double2 exy[kAtoms][kRuns];
  __shared__ int codes[kRuns];
  __shared__ int before[kWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  const int c = blockIdx.y;
  const int64_t per = (n + kSChunks - 1) / kSChunks;
  const int64_t j0 = c * per, j1 = min(n, j0 + per);
  if (form->general) {
    if (k >= K) return;
    double re = 0.0, im = 0.0;
    const double kx = kv[3 * k], ky = kv[3 * k + 1], kz = kv[3 * k + 2];
    for (int64_t j = j0; j < j1; ++j) {
      const Packed o = ld_packed(pk + j);
      double s, co;
      sincos(o.x * kx + o.y * ky + o.z * kz, &s, &co);
      re += o.w * co;
      im += o.w * s;
    }
    partial[(int64_t)c * K + k] = make_double2(re, im);
    return;
  }
  const bool on = k < K && wfold[k] != 0.0;
  if (!__syncthreads_or(on)) return;   // a block of the mirrored half
  const int code = k < K ? kn[k] : 0x101010;
  const int x = (code & 255) - 16, y = (code >> 8 & 255) - 16, z = (code >> 16 & 255) - 16;
  // the runs of equal (x, y) among the block's vectors, numbered in order
  const bool first = on && (threadIdx.x == 0 || wfold[k - 1] == 0.0 || (kn[k - 1] & 0xffff) != (code & 0xffff));
  const unsigned bal = __ballot_sync(0xffffffffu, first);
  if (lane == 0) before[warp] = __popc(bal);
  __syncthreads();
  int run = __popc(bal & (0xffffffffu >> (31 - lane))) - 1, runs = 0;
  for (int w = 0; w < kWarps; ++w) {
    if (w < warp) run += before[w];
    runs += before[w];
  }
  const bool few = runs <= kRuns;
  if (few && first) codes[run] = code & 0xffff;
  double cc = 0.0, ss = 0.0, cs = 0.0, sc = 0.0;   // sums of the products of (re, im) of exy with (cos, sin) of ez
  for (int64_t b = j0; b < j1; b += kAtoms) {
    const int m = (int)min((int64_t)kAtoms, j1 - b);
    __syncthreads();
    for (int t = threadIdx.x; t < m * kTab; t += blockDim.x)
      ez[t / kTab][t % kTab] = table[(b + t / kTab) * 3 * kTab + 2 * kTab + t % kTab];
    if (few) {
      for (int t = threadIdx.x; t < m * runs; t += blockDim.x) {
        const int j = t / runs, r = t % runs, rx = (codes[r] & 255) - 16, ry = (codes[r] >> 8) - 16;
        const double2* tj = table + (b + j) * 3 * kTab;
        const double2 e = cmul(conj_if(tj[abs(rx)], rx < 0), conj_if(tj[kTab + abs(ry)], ry < 0));
        const double q = pk[b + j].w;
        exy[j][r] = make_double2(q * e.x, q * e.y);
      }
    }
    __syncthreads();
    if (on) {
      for (int j = 0; j < m; ++j) {
        double2 p;
        if (few) {
          p = exy[j][run];
        } else {
          const double2* tj = table + (b + j) * 3 * kTab;
          p = cmul(conj_if(tj[abs(x)], x < 0), conj_if(tj[kTab + abs(y)], y < 0));
          const double q = pk[b + j].w;
          p.x *= q;
          p.y *= q;
        }
        const double2 e = ez[j][abs(z)];
        cc = fma(p.x, e.x, cc);
        ss = fma(p.y, e.y, ss);
        cs = fma(p.x, e.y, cs);
        sc = fma(p.y, e.x, sc);
      }
    }
  }
  if (on) partial[(int64_t)c * K + k] = z < 0 ? make_double2(cc + ss, sc - cs) : make_double2(cc - ss, sc + cs);
}

// S'_k = w_k S_k (a pair's weight on the half that stands for both) and sum_k w |S|^2.
__global__ void __launch_bounds__(kBlock) k_sfac_sum(const double2* __restrict__ partial, int K,
                                                     const double* __restrict__ w, const double* __restrict__ wfold,
                                                     const KForm* __restrict__ form, double2* __restrict__ S,
                                                     double* parts, unsigned int* ticket, double* out) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  double e[1] = {0.0};
  if (k < K) {
    const bool general = form->general;
    const double wk = general ? w[k] : wfold[k];
    double re = 0.0, im = 0.0;
    if (general || wk != 0.0) {
#pragma unroll 8
      for (int c = 0; c < kSChunks; ++c) {
        const double2 p = partial[(int64_t)c * K + k];
        re += p.x;
        im += p.y;
      }
    }
    e[0] = wk * (re * re + im * im);
    S[k] = make_double2(wk * re, wk * im);
  }
  block_sum_finish<1>(e, parts, ticket, out);
}

// One real-space pair: the force of j on i over d, coef (f_i -= coef d), and its energy without the charges' product.
__device__ __forceinline__ double ewald_pair(const EwaldPar& P, double r2, double qq, double& er) {
  double ir, gauss;
  const double r = sqrt_recip(r2, ir);
  er = erfc_exp(P.a, r, gauss) * ir;
  const double i2 = ir * ir, ir2 = fma(fma(-r2, i2, 1.0), i2, i2);   // 1/r^2 without the rounding of r twice
  return qq * fma(P.c2a, gauss, er) * ir2;
}

// Real space, every pair once: a block takes 8 tiles of 32 atoms (a tile per warp, an atom per lane) against every
// gridDim.y-th tile from its first on. A warp meets a later tile by rotating its atoms, with the force gathered on them,
// through the lanes: 32 rounds of 32 different pairs, after which the forces on the tile are home; those of the block's
// warps are added in warp order and stored per block, so every sum has a fixed order. Its own tile a warp takes both
// ways round. Bound by FP64 issue, some 95 operations per round whether few or all of its pairs are inside rcut; the
// rotation (14 shuffles) hides behind them. 8000 ions: 0.29 ms in 111 parts of a block row (0.27 before the pair
// terms were as exact as now, 0.29 then in 56 parts, 0.34 in 28: a block's share of the triangle shrinks along the rows);
// the pairs from both sides, a lane per atom (k_ewald_real), 0.55; the whole sum went from 9.75 ms (one thread per atom
// for all pairs and vectors) to 0.44.
__global__ void __launch_bounds__(kBlock, 3) k_ewald_tiles(const Packed* __restrict__ pk, int64_t n,
                                                           const __grid_constant__ EwaldPar P,
                                                           Packed* __restrict__ ipart, double* __restrict__ jpart) {
  __shared__ double onto[2][3][kWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tiles = (n + 31) / 32, ti = (int64_t)blockIdx.x * kWarps + warp;
  const int64_t i = ti * 32 + lane;
  const bool have_i = i < n;
  const Packed me = ld_packed(pk + min(i, n - 1));
  double fx = 0.0, fy = 0.0, fz = 0.0, u = 0.0;
  int buf = 0;
  for (int64_t tj = (int64_t)blockIdx.x * kWarps + blockIdx.y; tj < tiles; tj += gridDim.y, buf ^= 1) {
    double jx = 0.0, jy = 0.0, jz = 0.0;
    if (tj >= ti && ti < tiles) {   // warp-uniform
      const int64_t j0 = tj * 32;
      const bool own = tj == ti;
      Packed o = ld_packed(pk + min(j0 + lane, n - 1));
      for (int t = 0; t < 32; ++t) {
        const int64_t j = j0 + ((lane + t) & 31);
        double dx = sub(o.x, me.x), dy = sub(o.y, me.y), dz = sub(o.z, me.z);
        image3_any(dx, dy, dz, P.box);
        const double r2 = norm2(dx, dy, dz);
        if (r2 < P.r2cut && have_i && j < n && j != i) {
          double er;
          const double qq = me.w * o.w, coef = ewald_pair(P, r2, qq, er);
          u = fma(own ? 0.5 * qq : qq, er, u);
          fx = fma(-coef, dx, fx);
          fy = fma(-coef, dy, fy);
          fz = fma(-coef, dz, fz);
          jx = fma(coef, dx, jx);
          jy = fma(coef, dy, jy);
          jz = fma(coef, dz, jz);
        }
        const int from = (lane + 1) & 31;
        o.x = __shfl_sync(0xffffffffu, o.x, from);
        o.y = __shfl_sync(0xffffffffu, o.y, from);
        o.z = __shfl_sync(0xffffffffu, o.z, from);
        o.w = __shfl_sync(0xffffffffu, o.w, from);
        jx = __shfl_sync(0xffffffffu, jx, from);
        jy = __shfl_sync(0xffffffffu, jy, from);
        jz = __shfl_sync(0xffffffffu, jz, from);
      }
      if (own) jx = jy = jz = 0.0;   // its pairs were met from both sides
    }
    onto[buf][0][warp][lane] = jx;
    onto[buf][1][warp][lane] = jy;
    onto[buf][2][warp][lane] = jz;
    __syncthreads();   // the other buffer's readers passed this barrier after reading
    if (warp < 3) {
      double s = 0.0;
      for (int w = 0; w < kWarps; ++w) s += onto[buf][warp][w][lane];
      const int64_t j = tj * 32 + lane;
      if (j < n) jpart[((int64_t)blockIdx.x * 3 + warp) * n + j] = s;
    }
  }
  if (have_i) {
    Packed out;
    out.x = fx;
    out.y = fy;
    out.z = fz;
    out.w = u;
    ipart[(int64_t)blockIdx.y * n + i] = out;
  }
}

// Real space without the tiles' buffer (more than kTileAtoms atoms): every pair from both sides, a lane per atom against
// one chunk of partners.
__global__ void __launch_bounds__(kBlock, 4) k_ewald_real(const Packed* __restrict__ pk, int64_t n,
                                                          const __grid_constant__ EwaldPar P, Packed* __restrict__ ipart) {
  __shared__ double part[4][kWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * kAtoms + lane;
  const int64_t per = (n + gridDim.y - 1) / gridDim.y;
  const int64_t j0 = blockIdx.y * per, j1 = min(n, j0 + per);
  const Packed me = ld_packed(pk + min(i, n - 1));
  double fx = 0.0, fy = 0.0, fz = 0.0, u = 0.0;
  Packed next{};
  if (j0 + warp < j1) next = ld_packed(pk + j0 + warp);
  for (int64_t j = j0 + warp; j < j1; j += kWarps) {
    const Packed o = next;
    if (j + kWarps < j1) next = ld_packed(pk + j + kWarps);
    double dx = sub(o.x, me.x), dy = sub(o.y, me.y), dz = sub(o.z, me.z);
    image3_any(dx, dy, dz, P.box);
    const double r2 = norm2(dx, dy, dz);
    if (!(r2 < P.r2cut) || j == i) continue;
    double er;
    const double qq = me.w * o.w, coef = ewald_pair(P, r2, qq, er);
    u = fma(0.5 * qq, er, u);
    fx = fma(-coef, dx, fx);
    fy = fma(-coef, dy, fy);
    fz = fma(-coef, dz, fz);
  }
  part[0][warp][lane] = fx;
  part[1][warp][lane] = fy;
  part[2][warp][lane] = fz;
  part[3][warp][lane] = u;
  __syncthreads();
  if (warp == 0 && i < n) {
    double v[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int c = 0; c < 4; ++c)
      for (int w = 0; w < kWarps; ++w) v[c] += part[c][w][lane];
    Packed out;
    out.x = v[0];
    out.y = v[1];
    out.z = v[2];
    out.w = v[3];
    ipart[(int64_t)blockIdx.y * n + i] = out;
  }
}

// Reciprocal forces, sum_k w_k Im(conj(S_k) e^{i k.r_i}) k (accusim/forces.py:385-386) over one share of the vectors (in
// units of 2 pi / L with the tables). A lane per atom; the block's warps take k-vectors in turn, in runs along the last
// axis (the product of the first two factors is kept while the run lasts), tables in shared memory, 9 FP64 operations
// per atom and pair of mirrored vectors.
__global__ void __launch_bounds__(kBlock) k_ewald_recip(const Packed* __restrict__ pk, int64_t n,
                                                        const double* __restrict__ kv, const int32_t* __restrict__ kn,
                                                        const double2* __restrict__ S, int K,
                                                        const double2* __restrict__ table,
                                                        const KForm* __restrict__ form, Packed* __restrict__ gpart) {
  extern __shared__ double2 tab[];   // [3 * kTab][kAtoms]
  __shared__ double part[3][kWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i0 = (int64_t)blockIdx.x * kAtoms, i = i0 + lane;
  double gx = 0.0, gy = 0.0, gz = 0.0;
  if (form->general) {
    const Packed me = ld_packed(pk + min(i, n - 1));
    for (int k = blockIdx.y * kWarps + warp; k < K; k += kWarps * gridDim.y) {
      const double kx = kv[3 * k], ky = kv[3 * k + 1], kz = kv[3 * k + 2];
      double s, co;
      sincos(me.x * kx + me.y * ky + me.z * kz, &s, &co);
      const double2 Sk = S[k];
      const double t = Sk.x * s - Sk.y * co;
      gx += t * kx;
      gy += t * ky;
      gz += t * kz;
    }
  } else {
    const int m = (int)min((int64_t)kAtoms, n - i0);
    for (int t = threadIdx.x; t < m * 3 * kTab; t += blockDim.x)
      tab[t % (3 * kTab) * kAtoms + t / (3 * kTab)] = table[i0 * 3 * kTab + t];
    __syncthreads();
    int run = -1;
    double2 xy = make_double2(0.0, 0.0);
    double sum = 0.0;   // over the run's vectors
    auto close = [&]() {
      gx = fma((double)((run & 255) - 16), sum, gx);
      gy = fma((double)((run >> 8 & 255) - 16), sum, gy);
      sum = 0.0;
    };
    for (int b = 32 * (blockIdx.y * kWarps + warp); b < K; b += kBlock * gridDim.y) {
      const int mine = b + lane < K ? kn[b + lane] : 0;
      const double2 Sm = b + lane < K ? S[b + lane] : make_double2(0.0, 0.0);
      unsigned live = __ballot_sync(0xffffffffu, Sm.x != 0.0 || Sm.y != 0.0);   // the mirrored half is zero
      while (live) {
        const int q = __ffs(live) - 1;
        live &= live - 1u;
        const int code = __shfl_sync(0xffffffffu, mine, q);
        const double2 Sk = __ldg(S + b + q);
        const int z = (code >> 16 & 255) - 16;
        if ((code & 0xffff) != run) {
          if (run >= 0) close();
          run = code & 0xffff;
          const int x = (run & 255) - 16, y = (run >> 8 & 255) - 16;
          xy = cmul(conj_if(tab[abs(x) * kAtoms + lane], x < 0), conj_if(tab[(kTab + abs(y)) * kAtoms + lane], y < 0));
        }
        const double2 e = cmul(xy, conj_if(tab[(2 * kTab + abs(z)) * kAtoms + lane], z < 0));
        const double t = fma(Sk.x, e.y, -Sk.y * e.x);
        sum += t;
        gz = fma((double)z, t, gz);
      }
    }
    if (run >= 0) close();
  }
  part[0][warp][lane] = gx;
  part[1][warp][lane] = gy;
  part[2][warp][lane] = gz;
  __syncthreads();
  if (warp == 0 && i < n) {
    Packed out;
    double g[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int c = 0; c < 3; ++c)
      for (int w = 0; w < kWarps; ++w) g[c] += part[c][w][lane];
    out.x = g[0];
    out.y = g[1];
    out.z = g[2];
    out.w = 0.0;
    gpart[(int64_t)blockIdx.y * n + i] = out;
  }
}

// Sums the parts: 4 pi / V q_i times the reciprocal shares, the real-space shares, and what earlier blocks' tiles put onto
// the atom; a warp of the block takes every 8th part.
__global__ void __launch_bounds__(kBlock) k_ewald_sum(const Packed* __restrict__ pk, int64_t n,
                                                      const __grid_constant__ EwaldPar P, const KForm* __restrict__ form,
                                                      const Packed* __restrict__ gpart, int shares,
                                                      const Packed* __restrict__ ipart, int chunks,
                                                      const double* __restrict__ jpart, double* __restrict__ force,
                                                      double* partials, unsigned int* ticket, double* energy_real) {
  __shared__ double part[4][kWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * kAtoms + lane;
  double f[4] = {0.0, 0.0, 0.0, 0.0};
  if (i < n) {
    const double pre = P.pref_f * pk[i].w;
    for (int c = warp; c < shares; c += kWarps) {
      const Packed g = ld_packed(gpart + (int64_t)c * n + i);
      const bool general = form->general;
      f[0] += pre * (general ? 1.0 : 2.0 * M_PI / P.box.L[0]) * g.x;
      f[1] += pre * (general ? 1.0 : 2.0 * M_PI / P.box.L[1]) * g.y;
      f[2] += pre * (general ? 1.0 : 2.0 * M_PI / P.box.L[2]) * g.z;
    }
    for (int c = warp; c < chunks; c += kWarps) {
      const Packed r = ld_packed(ipart + (int64_t)c * n + i);
      f[0] += r.x;
      f[1] += r.y;
      f[2] += r.z;
      f[3] += r.w;
    }
    if (jpart) {
      const int64_t blocks = i / 32 / kWarps + 1;   // blocks whose first tile is not after the atom's
      for (int64_t b = warp; b < blocks; b += kWarps) {
#pragma unroll
        for (int c = 0; c < 3; ++c) f[c] += jpart[(b * 3 + c) * n + i];
      }
    }
  }
#pragma unroll
  for (int c = 0; c < 4; ++c) part[c][warp][lane] = f[c];
  __syncthreads();
  double u[1] = {0.0};
  if (warp == 0 && i < n) {
#pragma unroll
    for (int c = 0; c < 4; ++c)
      for (int w = 1; w < kWarps; ++w) f[c] += part[c][w][lane];
    force[3 * i] = P.k * f[0];
    force[3 * i + 1] = P.k * f[1];
    force[3 * i + 2] = P.k * f[2];
    u[0] = f[3];
  }
  block_sum_finish<1>(u, partials, ticket, energy_real);
}

inline size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

// The tiles' buffer, 3 n doubles per 256 atoms, stays under 256 MB up to here.
constexpr int64_t kTileAtoms = 49152;

// Parts a block row is split into, for about `rounds` blocks on each of 148 x 3 places, at most `most`.
int split_of(int64_t rows, int64_t rounds, int64_t most) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(most, ceil_div(444 * rounds, std::max<int64_t>(rows, 1))));
}
int real_chunks(int64_t n) {
  return n <= kTileAtoms ? split_of(ceil_div(n, kBlock), 8, std::min<int64_t>(128, ceil_div(n, 32)))
                         : split_of(ceil_div(n, kAtoms), 4, 64);
}
int recip_shares(int64_t n) { return split_of(ceil_div(n, kAtoms), 3, 16); }

struct EwaldWork {
  size_t pk, partial, S, kn, wfold, cube, table, ipart, jpart, gpart, eparts, sparts, flags, bytes;
};

EwaldWork work_of(int64_t n, int32_t K) {
  EwaldWork w;
  size_t at = 0;
  auto take = [&](size_t b) {
    const size_t o = at;
    at += a256(b);
    return o;
  };
  w.pk = take((size_t)n * sizeof(Packed));
  w.ipart = take((size_t)n * sizeof(Packed) * real_chunks(n));
  w.jpart = take(n <= kTileAtoms ? (size_t)ceil_div(n, kBlock) * 3 * n * 8 : 0);
  w.gpart = take((size_t)n * sizeof(Packed) * recip_shares(n));
  w.partial = take((size_t)kSChunks * K * 16);
  w.S = take((size_t)K * 16);
  w.kn = take((size_t)K * 4);
  w.wfold = take((size_t)K * 8);
  w.table = take((size_t)n * 3 * kTab * 16);
  w.eparts = take((size_t)ceil_div(n, kAtoms) * 8);
  w.sparts = take((size_t)ceil_div(K, kBlock) * 8);
  w.cube = take((size_t)kCube * kCube * kCube * 4 + sizeof(KForm));   // cleared together
  w.flags = w.cube + (size_t)kCube * kCube * kCube * 4;
  take(256);                                                           // ticket, after the flags' block
  w.bytes = at + 256;
  return w;
}

}  // namespace

extern "C" {

size_t acs_ewald_work_bytes(int64_t n, int32_t K) {
  return work_of(std::max<int64_t>(n, 1), std::max(K, 1)).bytes;
}

int acs_ewald_fp64(const double* pos, const double* q, int64_t n, const double* box3, const double* kvec,
                   const double* kw, int32_t K, double alpha, double rcut, double k_coul, double* force,
                   double* energy3_dev, void* work, size_t work_bytes, void* stream) {
  if (n < 1 || !pos || !q || !box3 || !kvec || !kw || K < 1 || !force || !energy3_dev || !(rcut > 0.0) ||
      !(alpha > 0.0))
    return ACS_ERR_ARG;
  if (work_bytes < acs_ewald_work_bytes(n, K) || !work) return ACS_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  char* base = (char*)(((uintptr_t)work + 255) & ~(uintptr_t)255);
  const EwaldWork w = work_of(n, K);
  Packed* pk = (Packed*)(base + w.pk);
  Packed* ipart = (Packed*)(base + w.ipart);
  double* jpart = n <= kTileAtoms ? (double*)(base + w.jpart) : nullptr;
  Packed* gpart = (Packed*)(base + w.gpart);
  double2* partial = (double2*)(base + w.partial);
  double2* S = (double2*)(base + w.S);
  int32_t* kn = (int32_t*)(base + w.kn);
  double* wfold = (double*)(base + w.wfold);
  double2* table = (double2*)(base + w.table);
  double* eparts = (double*)(base + w.eparts);
  double* sparts = (double*)(base + w.sparts);
  int32_t* cube = (int32_t*)(base + w.cube);
  KForm* form = (KForm*)(base + w.flags);
  unsigned int* ticket = (unsigned int*)(base + a256(w.flags + sizeof(KForm)));
  EwaldPar P;
  P.box = image_box(box3, 1);
  P.a = alpha;
  P.r2cut = square_reaching(rcut);
  P.c2a = 2.0 * alpha / sqrt(M_PI);
  const double V = box3[0] * box3[1] * box3[2];
  P.pref_f = 4.0 * M_PI / V;
  P.k = k_coul;
  P.K = K;
  if (cudaMemsetAsync(cube, 0, w.flags + sizeof(KForm) - w.cube, s) != cudaSuccess) return ACS_ERR_CUDA;
  k_prepare<<<(int)ceil_div(std::max<int64_t>(n, K), kBlock), kBlock, 0, s>>>(pos, q, n, kvec, P, pk, kn, cube, form,
                                                                              ticket);
  k_pair_vectors<<<(int)ceil_div(K, kBlock), kBlock, 0, s>>>(kn, cube, K, kw, wfold, form);
  k_phases<<<(int)ceil_div(n * 3 * kTab, kBlock), kBlock, 0, s>>>(pk, n, P, form, table);
  k_sfac_partial<<<dim3((unsigned)ceil_div(K, kBlock), kSChunks), kBlock, 0, s>>>(pk, n, kvec, kn, wfold, K, table, form,
                                                                                  partial);
  k_sfac_sum<<<(int)ceil_div(K, kBlock), kBlock, 0, s>>>(partial, K, kw, wfold, form, S, sparts, ticket,
                                                         energy3_dev + 1);   // scaled on the host
  const int chunks = real_chunks(n), shares = recip_shares(n);
  if (jpart)
    k_ewald_tiles<<<dim3((unsigned)ceil_div(n, kBlock), chunks), kBlock, 0, s>>>(pk, n, P, ipart, jpart);
  else
    k_ewald_real<<<dim3((unsigned)ceil_div(n, kAtoms), chunks), kBlock, 0, s>>>(pk, n, P, ipart);
  k_ewald_recip<<<dim3((unsigned)ceil_div(n, kAtoms), shares), kBlock, sizeof(double2) * 3 * kTab * kAtoms, s>>>(
      pk, n, kvec, kn, S, K, table, form, gpart);
  k_ewald_sum<<<(int)ceil_div(n, kAtoms), kBlock, 0, s>>>(pk, n, P, form, gpart, shares, ipart, chunks, jpart, force,
                                                          eparts, ticket, energy3_dev);
  return launch_status();
}

}  // extern "C"
