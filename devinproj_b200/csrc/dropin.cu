// FP64 drop-in kernels: cell grid, full neighbour list, LJ and DSF forces, VelocityVerlet, reductions.
//
// These back the reference-shaped plug-ins (LennardJones / DampedShiftedCoulomb / VelocityVerlet) when
// called one force evaluation at a time. Arithmetic follows the reference's FP64 NumPy expressions
// (accusim/forces.py:119-175, :279-321, :408-452; accusim/integrators.py:25-31); the pair filter and
// the integrator use non-contracted IEEE operations so their decisions and updates are bit-identical.
#include <math.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "common.cuh"

using namespace acs;

namespace {

struct GridDev {
  double lo[3], span[3];
  ImageBox box;
  int nc[3];
  double rc2;
};

GridDev to_dev(const acs_grid* g) {
  GridDev d;
  for (int k = 0; k < 3; ++k) {
    d.lo[k] = g->lo[k];
    d.span[k] = g->span[k];
    d.nc[k] = g->ncell[k];
  }
  d.box = image_box(g->box, g->periodic);
  d.rc2 = g->rc2;
  return d;
}

// cell = clip(int((pos - lo) / span * ncell), 0, ncell - 1)   (accusim/forces.py:290-291)
__device__ __forceinline__ int bin1(double x, double lo, double span, int nc) {
  double t = mul(div(sub(x, lo), span), (double)nc);
  if (!(t >= 1.0)) return 0;  // also catches NaN
  if (t >= (double)(nc - 1)) return nc - 1;
  return (int)t;
}

__device__ __forceinline__ int cell_index(const double* __restrict__ pos, int64_t i, const GridDev& g) {
  const int c0 = bin1(pos[3 * i + 0], g.lo[0], g.span[0], g.nc[0]);
  const int c1 = bin1(pos[3 * i + 1], g.lo[1], g.span[1], g.nc[1]);
  const int c2 = bin1(pos[3 * i + 2], g.lo[2], g.span[2], g.nc[2]);
  return (c0 * g.nc[1] + c1) * g.nc[2] + c2;
}

// place: the atom's arrival number in its cell.
__global__ void k_bin(const double* __restrict__ pos, int64_t n, GridDev g, int32_t* __restrict__ cell_of,
                      int32_t* __restrict__ place, int32_t* __restrict__ count) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cell_index(pos, i, g);
  cell_of[i] = c;
  place[i] = atomicAdd(&count[c], 1);
}

// Three-phase exclusive scan over int32 (chunk of 4096 per 1024-thread block).
constexpr int kScanThreads = 1024, kScanPer = 4, kScanChunk = kScanThreads * kScanPer;

__device__ int block_exclusive_scan(int v, int* total) {
  __shared__ int warp_sums[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;
  __syncthreads();
  if (wid == 0) {
    int w = (lane < (int)(blockDim.x >> 5)) ? warp_sums[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    warp_sums[lane] = w;
  }
  __syncthreads();
  int excl = x - v + (wid > 0 ? warp_sums[wid - 1] : 0);
  if (total) *total = warp_sums[(blockDim.x >> 5) - 1];
  __syncthreads();
  return excl;
}

__global__ void k_scan_chunks(const int32_t* __restrict__ in, int32_t* __restrict__ out, int64_t len,
                              int32_t* __restrict__ chunk_sums) {
  int64_t base = (int64_t)blockIdx.x * kScanChunk + (int64_t)threadIdx.x * kScanPer;
  int v[kScanPer];
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    v[k] = (base + k < len) ? in[base + k] : 0;
    s += v[k];
  }
  int total;
  int e = block_exclusive_scan(s, &total);
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    if (base + k < len) out[base + k] = e;
    e += v[k];
  }
  if (threadIdx.x == 0) chunk_sums[blockIdx.x] = total;
}

__global__ void k_scan_sums(int32_t* __restrict__ sums, int64_t nchunks, int32_t* __restrict__ grand_total) {
  // one block; serial over groups of 1024 chunk sums with a running carry
  __shared__ int carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t b = 0; b < nchunks; b += blockDim.x) {
    int64_t idx = b + threadIdx.x;
    int v = idx < nchunks ? sums[idx] : 0;
    int total;
    int e = block_exclusive_scan(v, &total);
    if (idx < nchunks) sums[idx] = e + carry;
    __syncthreads();
    if (threadIdx.x == 0) carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0 && grand_total) *grand_total = carry;
}

__global__ void k_scan_add(int32_t* __restrict__ out, int64_t len, const int32_t* __restrict__ sums) {
  int64_t base = (int64_t)blockIdx.x * kScanChunk;
  int add_v = sums[blockIdx.x];
  for (int k = threadIdx.x; k < kScanChunk; k += blockDim.x)
    if (base + k < len) out[base + k] += add_v;
}

__global__ void k_scatter(const int32_t* __restrict__ cell_of, const int32_t* __restrict__ place, int64_t n,
                          const int32_t* __restrict__ start, int32_t* __restrict__ unsorted) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) unsorted[start[cell_of[i]] + place[i]] = (int32_t)i;
}

// Counting, scan and scatter of up to kBinAtoms atoms into fewer than kBinCells cells by one block, the counts in shared
// memory: in small systems the launches of the general path (six and a clear) are most of its time. Whole list build of 864
// atoms 41 -> 23 us, 4096 ions 54 -> 37, 8000 ions 74 -> 56 (one block 11 us against 13 in seven launches).
constexpr int kBinAtoms = 8192, kBinCells = 8192;
__global__ void __launch_bounds__(1024) k_bin_block(const double* __restrict__ pos, int n,
                                                    const __grid_constant__ GridDev g, int nc,
                                                    int32_t* __restrict__ cell_of, int32_t* __restrict__ start,
                                                    int32_t* __restrict__ unsorted) {
  constexpr int kA = kBinAtoms / 1024, kC = kBinCells / 1024;
  __shared__ int count[kBinCells];
  for (int c = threadIdx.x; c < kBinCells; c += 1024) count[c] = 0;
  __syncthreads();
  int cell[kA], place[kA];
#pragma unroll
  for (int q = 0; q < kA; ++q) {
    const int i = threadIdx.x + 1024 * q;
    cell[q] = i < n ? cell_index(pos, i, g) : 0;
    if (i < n) {
      cell_of[i] = cell[q];
      place[q] = atomicAdd(&count[cell[q]], 1);
    }
  }
  __syncthreads();
  int v[kC], sum = 0, total;
#pragma unroll
  for (int q = 0; q < kC; ++q) {
    v[q] = count[kC * threadIdx.x + q];
    sum += v[q];
  }
  int ex = block_exclusive_scan(sum, &total);   // its barriers separate the reads above from the writes below
#pragma unroll
  for (int q = 0; q < kC; ++q) {
    const int c = kC * threadIdx.x + q;
    count[c] = ex;
    if (c <= nc) start[c] = ex;   // from nc on: n
    ex += v[q];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kA; ++q) {
    const int i = threadIdx.x + 1024 * q;
    if (i < n) unsorted[count[cell[q]] + place[q]] = i;
  }
}

// FP32 screen of the list build. Positions are held in units of the list radius from the grid's corner, one float4 per
// atom in cell order (w: atom index bits). Against the FP64 distance the FP32 one of two such positions is off by less
// than `err` per axis (both roundings, the image shift's and the subtraction's, for coordinates up to the grid's
// largest extent; four times the sum of the bounds), so r^2 <= lo is a pair, r^2 >= hi is none, and the band between
// is decided by the reference's FP64 expression. A position outside the grid (a caller's unwrapped atom, binned into an
// edge cell) or not finite is stored as NaN, which puts all its candidates into the band.
struct Screen {
  double scale, extent[3];
  float L[3], inv[3];   // periodic box in list radii
  float lo, hi;
};

// For pairs with r^2 < limit2 (at most the grid's radius squared).
Screen screen_of(const acs_grid* g, double limit2) {
  Screen f;
  f.scale = 1.0 / g->rc;
  double most = 0.0;
  for (int k = 0; k < 3; ++k) {
    f.extent[k] = g->span[k] * f.scale;
    most = std::max(most, f.extent[k]);
    f.L[k] = (float)(g->box[k] * f.scale);
    f.inv[k] = 1.0f / f.L[k];
  }
  const double r2 = limit2 * f.scale * f.scale, err = 1.2e-6 * most;
  const double band = std::max(1e-4 * r2, 2.0 * 1.7321 * sqrt(r2) * err + 3.0 * err * err);
  f.lo = (float)(r2 - band);
  f.hi = (float)(r2 + band);
  return f;
}

// Atoms of a cell in ascending index order, so list order is deterministic run to run: every atom's rank among
// its cell's atoms (the scatter's arbitrary order in `unsorted`) gives the place of its screen position. A thread per
// atom; the reads of a cell's members are shared by the cell's atoms through L1.
__global__ void k_rank_cells(const double* __restrict__ pos, const int32_t* __restrict__ cell_of, int64_t n, GridDev g,
                             Screen f, const int32_t* __restrict__ start, const int32_t* __restrict__ unsorted,
                             float4* __restrict__ screen) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int c = cell_of[i];
  const int s = start[c], e = start[c + 1];
  int rank = 0;
  for (int b = s; b < e; ++b) rank += unsorted[b] < (int32_t)i;
  float x[3];
  bool inside = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double t = (pos[3 * i + d] - g.lo[d]) * f.scale;
    inside = inside && t >= -0.01 && t <= f.extent[d] + 0.01;
    x[d] = (float)t;
  }
  screen[s + rank] = make_float4(inside ? x[0] : __int_as_float(0x7fffffff), x[1], x[2], __int_as_float((int32_t)i));
}

// The reference's FP64 filter of one pair.
__device__ __noinline__ bool exact_pair(const double* __restrict__ pos, int64_t i, int64_t j, const GridDev& g) {
  double dx = sub(pos[3 * j], pos[3 * i]), dy = sub(pos[3 * j + 1], pos[3 * i + 1]), dz = sub(pos[3 * j + 2], pos[3 * i + 2]);
  image3(dx, dy, dz, g.box);
  return norm2(dx, dy, dz) < g.rc2;
}

// The 27-cell stencil of cell (c0, c1, c2) as 9 rows of up to 3 cells along the last axis, whose atoms are consecutive
// in cell order; a row that wraps is two stretches with different images. Lane l < 18 holds the first slot and length
// of stretch l (row l / 2: offsets a, b; first or second part) and its image, the stencil's wraps per axis as
// (x + 1) + 3 (y + 1) + 9 (z + 1). Stretches in lane order, slots in order, are the stencil order.
__device__ __forceinline__ void stencil_stretch(const GridDev& g, const int32_t* __restrict__ start, int c, int lane,
                                                int& k0, int& len, int& image) {
  k0 = len = 0;
  image = 13;
  if (lane >= 18) return;
  const int c2 = c % g.nc[2], c1 = (c / g.nc[2]) % g.nc[1], c0 = c / (g.nc[2] * g.nc[1]);
  const int a = lane / 6 - 1, b = (lane / 2) % 3 - 1, part = lane & 1;
  const bool per = g.box.periodic;
  int x = c0 + a, y = c1 + b, wx = 0, wy = 0, wz = 0;
  bool on = true;
  if (per) {
    on = (g.nc[0] >= 3 || a == 0) && (g.nc[1] >= 3 || b == 0);
    wx = x < 0 ? -1 : (x >= g.nc[0] ? 1 : 0);
    wy = y < 0 ? -1 : (y >= g.nc[1] ? 1 : 0);
    x -= wx * g.nc[0];
    y -= wy * g.nc[1];
  } else {
    on = x >= 0 && x < g.nc[0] && y >= 0 && y < g.nc[1];
  }
  int z0 = c2 - 1, z1 = c2 + 1;   // inclusive
  if (!per || g.nc[2] < 3) {
    z0 = max(z0, 0);
    z1 = min(z1, g.nc[2] - 1);
    on = on && part == 0;
  } else if (z0 < 0) {            // the wrapped cell first, as the stencil order has it
    if (part == 0) { z0 = z1 = g.nc[2] - 1; wz = -1; } else { z0 = 0; }
  } else if (z1 >= g.nc[2]) {
    if (part == 0) { z1 = g.nc[2] - 1; } else { z0 = z1 = 0; wz = 1; }
  } else {
    on = on && part == 0;
  }
  if (!on) return;
  const int row = (x * g.nc[1] + y) * g.nc[2];
  k0 = start[row + z0];
  len = start[row + z1 + 1] - k0;
  image = (wx + 1) + 3 * (wy + 1) + 9 * (wz + 1);
}

__device__ __forceinline__ void list_end(int32_t i, int cnt, int maxnb, int32_t* __restrict__ nnb, acs_dev_status* status) {
  nnb[i] = cnt;
  if (cnt > maxnb) {
    atomicOr(&status->flags, ACS_FLAG_OVERFLOW);
    atomicMax(&status->need_nbr, cnt);
  }
}

// Neighbour lists, a warp per atom in cell order: the warp tests 32 candidates at a time by the FP32 screen and a ballot
// keeps the accepted ones in stencil order, ascending index within a cell. WRAP: a periodic axis has fewer than 4
// cells, so the image is found per pair instead of from the stencil offset (with 3 cells both images of a pair whose
// images are in doubt lie outside the radius). kU loads in flight.
// Bound by instruction issue (about 30 per 32 candidates) and, in small systems, by the latency of one atom's chain. A
// thread per atom testing every candidate in FP64 took, for the whole build, 305 us at 864 LJ atoms (now 23), 355 at
// 16,384 (69) and 643 at 8000 ions with 250 neighbours (56).
template <bool WRAP, int kU>
__global__ void __launch_bounds__(kBlock) k_list_atoms(const double* __restrict__ pos, int64_t n,
                                                       const __grid_constant__ GridDev g, Screen f,
                                                       const int32_t* __restrict__ cell_of,
                                                       const int32_t* __restrict__ start,
                                                       const float4* __restrict__ screen, int maxnb,
                                                       int32_t* __restrict__ nbr, int32_t* __restrict__ nnb,
                                                       acs_dev_status* status) {
  const int lane = threadIdx.x & 31;
  const int64_t slot = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (slot >= n) return;
  const float4 me = screen[slot];
  const int32_t i = __float_as_int(me.w);
  int k0, len, image;
  stencil_stretch(g, start, cell_of[i], lane, k0, len, image);
  unsigned work = __ballot_sync(0xffffffffu, len > 0);
  const unsigned below = (1u << lane) - 1u;
  int32_t* __restrict__ row = nbr + nbr_slot(i, 0, maxnb);
  int cnt = 0;
  while (work) {
    const int st = __ffs(work) - 1;
    work &= work - 1u;
    const int s0 = __shfl_sync(0xffffffffu, k0, st), s1 = s0 + __shfl_sync(0xffffffffu, len, st);
    float mx = me.x, my = me.y, mz = me.z;
    if (!WRAP) {   // the candidates' image shift, taken off this atom
      const int im = __shfl_sync(0xffffffffu, image, st);
      mx -= (float)(im % 3 - 1) * f.L[0];
      my -= (float)((im / 3) % 3 - 1) * f.L[1];
      mz -= (float)(im / 9 - 1) * f.L[2];
    }
    for (int base = s0; base < s1; base += 32 * kU) {
      float4 o[kU];
#pragma unroll
      for (int v = 0; v < kU; ++v) {
        const int k = base + 32 * v + lane;
        o[v] = make_float4(3e30f, 3e30f, 3e30f, 0.f);   // past the end: r^2 overflows, outside
        if (k < s1) o[v] = __ldg(screen + k);
      }
#pragma unroll
      for (int v = 0; v < kU; ++v) {
        if (base + 32 * v >= s1) break;
        const int k = base + 32 * v + lane;
        float dx = o[v].x - mx, dy = o[v].y - my, dz = o[v].z - mz;
        if (WRAP) {
          dx -= f.L[0] * rintf(dx * f.inv[0]);
          dy -= f.L[1] * rintf(dy * f.inv[1]);
          dz -= f.L[2] * rintf(dz * f.inv[2]);
        }
        const float q = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        const int32_t j = __float_as_int(o[v].w);
        bool in = k < s1 && q <= f.lo;
        const bool band = k < s1 && !(q <= f.lo) && !(q >= f.hi);
        if (__any_sync(0xffffffffu, band)) {
          if (band) in = exact_pair(pos, i, j, g);
        }
        in = in && k != slot;
        const unsigned bal = __ballot_sync(0xffffffffu, in);
        const int at = cnt + __popc(bal & below);
        if (in && at < maxnb) row[(int64_t)at * 32] = j;
        cnt += __popc(bal);
      }
    }
  }
  if (lane == 0) list_end(i, cnt, maxnb, nnb, status);
}

// Neighbour lists, a lane per atom in cell order, for cells with few atoms (sparse_cells): bound by the latency of a
// stencil's cell starts and candidates, with up to 1024 atoms of an SM in flight. The same lists entry by entry. Whole build
// of 10^6 atoms in random order at 0.2, 0.7 and 1.6 atoms a cell: 193, 214, 264 us; a warp per atom 930, 1184, 1297. The
// stencil's starts read together into registers took 220, 283, 375 (104 registers).
template <bool WRAP>
__global__ void __launch_bounds__(kBlock) k_list_sparse(const double* __restrict__ pos, int64_t n,
                                                        const __grid_constant__ GridDev g, Screen f,
                                                        const int32_t* __restrict__ cell_of,
                                                        const int32_t* __restrict__ start,
                                                        const float4* __restrict__ screen, int maxnb,
                                                        int32_t* __restrict__ nbr, int32_t* __restrict__ nnb,
                                                        acs_dev_status* status) {
  const int64_t slot = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= n) return;
  const float4 me = screen[slot];
  const int32_t i = __float_as_int(me.w);
  int32_t* __restrict__ row = nbr + nbr_slot(i, 0, maxnb);
  int cnt = 0;
  const int c = cell_of[i];
#pragma unroll 1
  for (int st = 0; st < 18; ++st) {
    int k0, len, im;
    stencil_stretch(g, start, c, st, k0, len, im);
    float mx = me.x, my = me.y, mz = me.z;
    if (!WRAP) {
      mx -= (float)(im % 3 - 1) * f.L[0];
      my -= (float)((im / 3) % 3 - 1) * f.L[1];
      mz -= (float)(im / 9 - 1) * f.L[2];
    }
    for (int k = k0; k < k0 + len; ++k) {
      const float4 o = __ldg(screen + k);
      float dx = o.x - mx, dy = o.y - my, dz = o.z - mz;
      if (WRAP) {
        dx -= f.L[0] * rintf(dx * f.inv[0]);
        dy -= f.L[1] * rintf(dy * f.inv[1]);
        dz -= f.L[2] * rintf(dz * f.inv[2]);
      }
      const float q = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
      if (q >= f.hi || k == slot) continue;
      const int32_t j = __float_as_int(o.w);
      if (!(q <= f.lo) && !exact_pair(pos, i, j, g)) continue;
      if (cnt < maxnb) row[(int64_t)cnt * 32] = j;
      ++cnt;
    }
  }
  list_end(i, cnt, maxnb, nnb, status);
}

// Neighbour lists, a warp per home cell (32 of its atoms at a time), for systems with cells enough to fill the chip: the
// stencil's candidates are read, shifted to their image and culled against the home atoms' bounding box once for all
// home atoms, packed to full batches of 32 in shared memory, and each batch is screened against two home atoms per
// packed FP32 operation; ballots give a home atom's accepted candidates, which its lane then writes. The same lists entry
// by entry. Boxes with 4 or more cells on every periodic axis. Whole build of the 1,048,576-atom LJ fluid (78 neighbours
// of 516 candidates): 2.73 ms by a thread per atom in FP64, 1.97 by a warp per atom, 0.71 here, where the lists' 4-byte
// stores, one sector each, are most of the rest; with the atoms in random order 4.97, 2.35 and 2.51. 80 registers and 36
// bytes spilled.
__global__ void __launch_bounds__(kBlock) k_list_cells(const double* __restrict__ pos, const __grid_constant__ GridDev g,
                                                       Screen f, int64_t ncells, const int32_t* __restrict__ start,
                                                       const float4* __restrict__ screen, int maxnb,
                                                       int32_t* __restrict__ nbr, int32_t* __restrict__ nnb,
                                                       acs_dev_status* status) {
  constexpr int kWarps = kBlock / 32;
  __shared__ __align__(8) float hnx[kWarps][32], hny[kWarps][32], hnz[kWarps][32];   // home positions, negated
  __shared__ float4 buf[kWarps][64];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int64_t c = (int64_t)blockIdx.x * kWarps + wib;
  if (c >= ncells) return;
  const int h0 = start[c], hn = start[c + 1] - h0;
  if (32 * (int)blockIdx.y >= hn) return;
  int k0, len, image;
  stencil_stretch(g, start, (int)c, lane, k0, len, image);
  const unsigned work0 = __ballot_sync(0xffffffffu, len > 0);
  for (int hb = 32 * blockIdx.y; hb < hn; hb += 32 * gridDim.y) {
    const int nh = min(32, hn - hb);
    const float4 me = screen[h0 + hb + min(lane, nh - 1)];
    const int32_t i = __float_as_int(me.w);
    __syncwarp();
    hnx[wib][lane] = -me.x;
    hny[wib][lane] = -me.y;
    hnz[wib][lane] = -me.z;
    // bounding box of the home atoms; one that is NaN (decided in FP64) turns the culling off
    float lx = me.x, ly = me.y, lz = me.z, ux = me.x, uy = me.y, uz = me.z;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lx = fminf(lx, __shfl_xor_sync(0xffffffffu, lx, o));
      ly = fminf(ly, __shfl_xor_sync(0xffffffffu, ly, o));
      lz = fminf(lz, __shfl_xor_sync(0xffffffffu, lz, o));
      ux = fmaxf(ux, __shfl_xor_sync(0xffffffffu, ux, o));
      uy = fmaxf(uy, __shfl_xor_sync(0xffffffffu, uy, o));
      uz = fmaxf(uz, __shfl_xor_sync(0xffffffffu, uz, o));
    }
    const float reach = __any_sync(0xffffffffu, isnan(me.x)) ? __int_as_float(0x7f800000) : f.hi;
    int32_t* __restrict__ row = nbr + nbr_slot(i, 0, maxnb);
    int cnt = 0, nbuf = 0;
    unsigned work = work0;
    int k = 0, s1 = 0;   // this lane's next raw candidate and the end of its stretch
    float sx = 0.f, sy = 0.f, sz = 0.f;
    float4 raw;
    bool more, live = false;
    // the next 32 raw candidates; warp-uniform result: whether there were any
    auto next = [&]() {
      const bool done = __shfl_sync(0xffffffffu, k, 0) >= s1;
      if (done) {
        if (!work) return false;
        const int st = __ffs(work) - 1;
        work &= work - 1u;
        const int s0 = __shfl_sync(0xffffffffu, k0, st);
        s1 = s0 + __shfl_sync(0xffffffffu, len, st);
        const int im = __shfl_sync(0xffffffffu, image, st);
        sx = (float)(im % 3 - 1) * f.L[0];
        sy = (float)((im / 3) % 3 - 1) * f.L[1];
        sz = (float)(im / 9 - 1) * f.L[2];
        k = s0 + lane;
      }
      live = k < s1;
      if (live) raw = __ldg(screen + k);
      k += 32;
      return true;
    };
    more = next();
    while (true) {
      if (more) {   // append this chunk's survivors, in order; the next chunk's loads fly while a batch is screened
        float4 o = make_float4(raw.x + sx, raw.y + sy, raw.z + sz, raw.w);
        const float gx = fmaxf(fmaxf(lx - o.x, o.x - ux), 0.f), gy = fmaxf(fmaxf(ly - o.y, o.y - uy), 0.f),
                    gz = fmaxf(fmaxf(lz - o.z, o.z - uz), 0.f);
        const bool keep = live && (isnan(o.x) || !(fmaf(gz, gz, fmaf(gy, gy, gx * gx)) >= reach));
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (keep) buf[wib][nbuf + __popc(bal & below)] = o;
        nbuf += __popc(bal);
        more = next();
      }
      if (nbuf == 0 && !more) break;
      if (nbuf < 32 && more) continue;
      const int nk = min(32, nbuf);
      __syncwarp();
      float4 cur = make_float4(3e30f, 3e30f, 3e30f, 0.f);
      if (lane < nk) cur = buf[wib][lane];
      uint32_t m_in = 0u, m_out = 0u;
      const float2 px = make_float2(cur.x, cur.x), py = make_float2(cur.y, cur.y), pz = make_float2(cur.z, cur.z);
#pragma unroll 2
      for (int h = 0; h < nh; h += 2) {
        const float2 x = __fadd2_rn(px, *reinterpret_cast<const float2*>(&hnx[wib][h]));
        const float2 y = __fadd2_rn(py, *reinterpret_cast<const float2*>(&hny[wib][h]));
        const float2 z = __fadd2_rn(pz, *reinterpret_cast<const float2*>(&hnz[wib][h]));
        const float2 q = __ffma2_rn(z, z, __ffma2_rn(y, y, __fmul2_rn(x, x)));
        const unsigned i0 = __ballot_sync(0xffffffffu, q.x <= f.lo), o0 = __ballot_sync(0xffffffffu, q.x >= f.hi);
        const unsigned i1 = __ballot_sync(0xffffffffu, q.y <= f.lo), o1 = __ballot_sync(0xffffffffu, q.y >= f.hi);
        if (lane == h) {
          m_in = i0;
          m_out = o0;
        }
        if (lane == h + 1) {
          m_in = i1;
          m_out = o1;
        }
      }
      const uint32_t valid = lane < nh ? 0xffffffffu >> (32 - nk) : 0u;
      m_in &= valid;
      uint32_t m_band = valid & ~m_in & ~m_out;
      if (__any_sync(0xffffffffu, m_band != 0u)) {
        while (m_band) {
          const int t = __ffs(m_band) - 1;
          m_band &= m_band - 1u;
          if (exact_pair(pos, i, __float_as_int(buf[wib][t].w), g)) m_in |= 1u << t;
        }
      }
      while (m_in) {   // list order; the atom itself is left out
        const int t = __ffs(m_in) - 1;
        m_in &= m_in - 1u;
        const int32_t j = __float_as_int(buf[wib][t].w);
        if (j != i) {
          if (cnt < maxnb) row[(int64_t)cnt * 32] = j;
          ++cnt;
        }
      }
      __syncwarp();   // the survivors beyond this batch move to the front
      const int rest = nbuf - nk;
      float4 mv = make_float4(0.f, 0.f, 0.f, 0.f);
      if (lane < rest) mv = buf[wib][nk + lane];
      __syncwarp();
      if (lane < rest) buf[wib][lane] = mv;
      nbuf = rest;
    }
    if (lane < nh) list_end(i, cnt, maxnb, nnb, status);
  }
}

// One pair into the histogram below: its distance by the reference's FP64 expression and its bin by NumPy's rule.
__device__ __forceinline__ void count_pair(const double* __restrict__ pos, const int32_t* __restrict__ sp, int64_t i, int64_t j,
                                           const GridDev& g, int species, int bins, double rmax, double step, double per_bin,
                                           unsigned int* sh_hist) {
  double dx = sub(pos[3 * j], pos[3 * i]), dy = sub(pos[3 * j + 1], pos[3 * i + 1]), dz = sub(pos[3 * j + 2], pos[3 * i + 2]);
  image3_any(dx, dy, dz, g.box);
  const double r = __dsqrt_rn(norm2(dx, dy, dz));
  if (r <= rmax && (species < 0 || sp[j] == species)) {
    int idx = min((int)(r * per_bin), bins - 1);
    if (r < mul((double)idx, step)) idx -= 1;
    const double upper = idx + 1 == bins ? rmax : mul((double)(idx + 1), step);
    if (r >= upper && idx != bins - 1) idx += 1;
    atomicAdd(&sh_hist[idx], 1u);
  }
}

// Pair-distance histogram of accusim/analysis.py:7-24 (rdf): pairs i < j, both of `species` (all when < 0),
// minimum-image r by the reference's FP64 expression, binned by NumPy's uniform-bin rule on [0, rmax]
// (numpy histogram: index = int((r / rmax) * bins), the right edge into the last bin, then one step down if
// r < edge[index] or up if r >= edge[index + 1] below the last bin, with edge[k] = k * (rmax / bins) and
// edge[bins] = rmax; the steps make the index the same for a quotient rounded otherwise). Per-block shared-memory
// counts, integer atomics: exact and order-independent.
// A warp per atom over the later atoms of its stencil, in cell order (each pair once): the FP32 screen drops what is
// surely farther than rmax (5 of 6 candidates), the rest queue in shared memory and are measured 32 at a time, so the
// FP64 square roots run on full warps. 32,000 LJ atoms to 4.4 sigma: 1.37 ms by a thread per atom over all candidates
// in FP64, 0.12 here. WRAP as for k_list_atoms.
template <bool WRAP>
__global__ void __launch_bounds__(kBlock) k_rdf(const double* __restrict__ pos, const int32_t* __restrict__ sp, int64_t n,
                                                const __grid_constant__ GridDev g, Screen f,
                                                const int32_t* __restrict__ cell_of, const int32_t* __restrict__ start,
                                                const float4* __restrict__ screen, int species, int bins, double rmax,
                                                double step, unsigned long long* __restrict__ hist) {
  extern __shared__ unsigned int sh_hist[];
  __shared__ int2 queue[kBlock / 32][64];
  for (int b = threadIdx.x; b < bins; b += blockDim.x) sh_hist[b] = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const double per_bin = bins / rmax;
  int queued = 0;
  auto measure = [&](int m) {   // the first m queued pairs
    if (lane < m) {
      const int2 p = queue[wib][lane];
      count_pair(pos, sp, p.x, p.y, g, species, bins, rmax, step, per_bin, sh_hist);
    }
  };
  for (int64_t slot = (int64_t)blockIdx.x * (kBlock / 32) + wib; slot < n; slot += (int64_t)gridDim.x * (kBlock / 32)) {
    const float4 me = screen[slot];
    const int32_t i = __float_as_int(me.w);
    if (species >= 0 && sp[i] != species) continue;
    int k0, len, image;
    stencil_stretch(g, start, cell_of[i], lane, k0, len, image);
    const int past = k0 + len;
    k0 = max(k0, (int)min(slot + 1, (int64_t)past));   // later atoms only
    unsigned work = __ballot_sync(0xffffffffu, k0 < past);
    while (work) {
      const int st = __ffs(work) - 1;
      work &= work - 1u;
      const int s0 = __shfl_sync(0xffffffffu, k0, st), s1 = __shfl_sync(0xffffffffu, past, st);
      float mx = me.x, my = me.y, mz = me.z;
      if (!WRAP) {
        const int im = __shfl_sync(0xffffffffu, image, st);
        mx -= (float)(im % 3 - 1) * f.L[0];
        my -= (float)((im / 3) % 3 - 1) * f.L[1];
        mz -= (float)(im / 9 - 1) * f.L[2];
      }
      for (int base = s0; base < s1; base += 32) {
        const int k = base + lane;
        float4 o = make_float4(3e30f, 3e30f, 3e30f, 0.f);
        if (k < s1) o = __ldg(screen + k);
        float dx = o.x - mx, dy = o.y - my, dz = o.z - mz;
        if (WRAP) {
          dx -= f.L[0] * rintf(dx * f.inv[0]);
          dy -= f.L[1] * rintf(dy * f.inv[1]);
          dz -= f.L[2] * rintf(dz * f.inv[2]);
        }
        const float q = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        const bool maybe = k < s1 && !(q >= f.hi);
        const unsigned bal = __ballot_sync(0xffffffffu, maybe);
        if (maybe) queue[wib][queued + __popc(bal & below)] = make_int2(i, __float_as_int(o.w));
        queued += __popc(bal);
        __syncwarp();
        if (queued >= 32) {
          measure(32);
          queued -= 32;
          const int2 rest = queue[wib][32 + lane];
          __syncwarp();
          queue[wib][lane] = rest;
          __syncwarp();
        }
      }
    }
  }
  measure(queued);
  __syncthreads();
  for (int b = threadIdx.x; b < bins; b += blockDim.x)
    if (sh_hist[b]) atomicAdd(&hist[b], (unsigned long long)sh_hist[b]);
}

// The same counts for cells with few atoms (sparse_cells): a lane per atom, each walking its own stencil, the pairs in the
// warp's queue. 10^6 atoms at 0.2, 0.7 and 3.3 a cell: 191, 198, 294 us; a warp per atom 527, 676, 790; a lane per atom that
// measured its own pairs at once, on divergent FP64 code, 312, 585, 1195.
template <bool WRAP>
__global__ void __launch_bounds__(kBlock) k_rdf_sparse(const double* __restrict__ pos, const int32_t* __restrict__ sp, int64_t n,
                                                       const __grid_constant__ GridDev g, Screen f,
                                                       const int32_t* __restrict__ cell_of,
                                                       const int32_t* __restrict__ start,
                                                       const float4* __restrict__ screen, int species, int bins, double rmax,
                                                       double step, unsigned long long* __restrict__ hist) {
  extern __shared__ unsigned int sh_hist[];
  __shared__ int2 queue[kBlock / 32][64];
  for (int b = threadIdx.x; b < bins; b += blockDim.x) sh_hist[b] = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const double per_bin = bins / rmax;
  int queued = 0;
  for (int64_t base = (int64_t)blockIdx.x * blockDim.x + 32 * wib; base < n; base += (int64_t)gridDim.x * blockDim.x) {
    const int64_t slot = base + lane;
    const float4 me = screen[min(slot, n - 1)];
    const int32_t i = __float_as_int(me.w);
    const bool on = slot < n && (species < 0 || sp[i] == species);
    const int c = cell_of[i], c2 = c % g.nc[2];
    const bool wraps = __any_sync(0xffffffffu, c2 == 0 || c2 == g.nc[2] - 1);
#pragma unroll 1
    for (int st = 0; st < 18; st += wraps ? 1 : 2) {
      int k0, len, im;
      stencil_stretch(g, start, c, st, k0, len, im);
      const int end = on ? k0 + len : 0;
      float mx = me.x, my = me.y, mz = me.z;
      if (!WRAP) {
        mx -= (float)(im % 3 - 1) * f.L[0];
        my -= (float)((im / 3) % 3 - 1) * f.L[1];
        mz -= (float)(im / 9 - 1) * f.L[2];
      }
      for (int k = (int)max((int64_t)k0, slot + 1); __any_sync(0xffffffffu, k < end); ++k) {   // later atoms only
        float4 o = make_float4(3e30f, 3e30f, 3e30f, 0.f);
        if (k < end) o = __ldg(screen + k);
        float dx = o.x - mx, dy = o.y - my, dz = o.z - mz;
        if (WRAP) {
          dx -= f.L[0] * rintf(dx * f.inv[0]);
          dy -= f.L[1] * rintf(dy * f.inv[1]);
          dz -= f.L[2] * rintf(dz * f.inv[2]);
        }
        const bool maybe = k < end && !(fmaf(dz, dz, fmaf(dy, dy, dx * dx)) >= f.hi);
        const unsigned bal = __ballot_sync(0xffffffffu, maybe);
        if (maybe) queue[wib][queued + __popc(bal & below)] = make_int2(i, __float_as_int(o.w));
        queued += __popc(bal);
        __syncwarp();
        if (queued >= 32) {
          const int2 p = queue[wib][lane];
          count_pair(pos, sp, p.x, p.y, g, species, bins, rmax, step, per_bin, sh_hist);
          queued -= 32;
          const int2 rest = queue[wib][32 + lane];
          __syncwarp();
          queue[wib][lane] = rest;
          __syncwarp();
        }
      }
    }
  }
  if (lane < queued) {
    const int2 p = queue[wib][lane];
    count_pair(pos, sp, p.x, p.y, g, species, bins, rmax, step, per_bin, sh_hist);
  }
  __syncthreads();
  for (int b = threadIdx.x; b < bins; b += blockDim.x)
    if (sh_hist[b]) atomicAdd(&hist[b], (unsigned long long)sh_hist[b]);
}

__global__ void k_pairs(const int32_t* __restrict__ nbr, const int32_t* __restrict__ nnb, int64_t n, int maxnb,
                        int32_t* pi, int32_t* pj, int64_t cap, unsigned long long* count) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int m = min(nnb[i], maxnb);
  for (int k = 0; k < m; ++k) {
    int j = nbr[nbr_slot(i, k, maxnb)];
    if (i < j) {
      unsigned long long w = atomicAdd(count, 1ull);
      if ((int64_t)w < cap) {
        pi[w] = (int32_t)i;
        pj[w] = j;
      }
    }
  }
}

__device__ __forceinline__ bool moved(double dx, double dy, double dz, const ImageBox& box, double half_skin2) {
  image3(dx, dy, dz, box);
  return !(norm2(dx, dy, dz) < half_skin2);   // NaN also forces a rebuild, as in the reference
}

// One block's answer for up to kMovedAtoms atoms, without the clear that the grid's needs before it: a small system's
// skin test is launches. The loads of a thread's atoms go out together (4096 atoms: 5.9 us one after the other, 5.3 so; the
// grid's kernel takes 3.1, and the clear).
constexpr int kMovedAtoms = 4096;
__global__ void __launch_bounds__(1024) k_displacement_block(const double* __restrict__ pos,
                                                             const double* __restrict__ pos0, int n, ImageBox box,
                                                             double half_skin2, int32_t* flag) {
  constexpr int kA = kMovedAtoms / 1024;
  double d[kA][3];
#pragma unroll
  for (int q = 0; q < kA; ++q) {
    const int i = threadIdx.x + 1024 * q;
#pragma unroll
    for (int c = 0; c < 3; ++c) d[q][c] = i < n ? sub(pos[3 * i + c], pos0[3 * i + c]) : 0.0;
  }
  bool any = false;
#pragma unroll
  for (int q = 0; q < kA; ++q)
    if ((int)threadIdx.x + 1024 * q < n) any = any || moved(d[q][0], d[q][1], d[q][2], box, half_skin2);
  const int r = __syncthreads_or(any);
  if (threadIdx.x == 0) *flag = r ? 1 : 0;
}

__global__ void k_displacement(const double* __restrict__ pos, const double* __restrict__ pos0, int64_t n, ImageBox box,
                               double half_skin2, int32_t* flag) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && moved(sub(pos[3 * i], pos0[3 * i]), sub(pos[3 * i + 1], pos0[3 * i + 1]), sub(pos[3 * i + 2], pos0[3 * i + 2]),
                     box, half_skin2))
    *flag = 1;
}

// ------------------------------------------------------------------------------------ forces --
struct LJTab {
  int ns;
  double eps[ACS_MAX_SPECIES * ACS_MAX_SPECIES];
  double sig2[ACS_MAX_SPECIES * ACS_MAX_SPECIES];
  double rc2[ACS_MAX_SPECIES * ACS_MAX_SPECIES];
  double shift6;  // src6**2 - src6, src6 = (1/cutoff**2)**3
};

struct DSFPar {
  double a, rc, rc2, k, c, erc, erc_rc, fshift, self_coef;
};

// Packs positions with the species index (sp) or the charge (q) and clears the energy reduction's ticket.
__global__ void k_pack(const double* __restrict__ pos, const int32_t* __restrict__ sp, const double* __restrict__ q,
                       int64_t n, Packed* __restrict__ out, unsigned int* ticket) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *ticket = 0u;
  if (i >= n) return;
  Packed v;
  v.x = pos[3 * i];
  v.y = pos[3 * i + 1];
  v.z = pos[3 * i + 2];
  v.w = sp ? __hiloint2double(0, sp[i]) : q[i];
  out[i] = v;
}

// How the pair kernels split their work: a block of 256 threads takes 256 / phases atoms, and the `phases` threads of
// an atom (256 / phases apart in the block) share its neighbours, entry k going to phase k mod phases. Consecutive
// threads are consecutive atoms, so a list row is read in whole sectors for every split up to 32 (8 atoms a row).
struct PairSplit {
  int log2_phases, atoms;   // phases = 1 << log2_phases, atoms = 256 >> log2_phases
  int64_t blocks;
};

// About how many neighbours an atom has in its list (all atoms without one), from the density and the cutoff alone: the
// split decides the order of an atom's sum, which must not depend on the buffer the caller gave the list (its capacity).
// A list holds the neighbours to the cutoff plus a skin, 1.4 times those inside in the usual 0.3 of 2.5. Without a box the
// density is not known: few, but more than a gas has.
double pairs_per_atom(int64_t n, bool list, const double* box3, double rc) {
  if (!list) return (double)n;
  if (!box3) return std::min((double)n, 24.0);
  const double V = fabs(box3[0] * box3[1] * box3[2]);
  return V > 0.0 ? std::min((double)n, 1.4 * 4.0 / 3.0 * M_PI * rc * rc * rc * ((double)n / V)) : (double)n;
}

// The fewest phases (at most 32) that give kHalfFilled threads; then more, up to `threads` and kMostThreads in all, while
// each thread keeps `entries` of an atom's pairs. 151,552 threads are resident: half of them hide the latency of a call
// with few pairs, and more only add blocks whose sums meet at the end (LJ gas, 0.3 entries an atom: 12,000 atoms 11.3 us
// with 96,000 threads, 13.6 with 192,000). A thread with few entries is all prologue. DSF terms are long enough to want
// several waves, if there are pairs: 32,768 ions with 351 entries 141 us at 131,072 threads, 118 at 262,144, 112 at
// 524,288; 175,616 ions 678, 595, 544; 64,000 with 78 entries 83, 72, 72 us at 128,000, 256,000 and 512,000; with 22
// entries 33, 31, 35; with 0.3 entries 12, 15, 21 (a thread per atom, as it was before the split: 17). LJ with 79 entries
// an atom does not: 32,000 atoms 18.5 us at 128,000 threads, 21.6 at 256,000, 21.5 at 64,000; 12,000 atoms 17.7 at 96,000,
// 19.7 at 192,000; 55,296 atoms 25.5 at 110,592, 28.0 at 221,184, 35.0 at 55,296; 1,048,576 atoms 0.355 ms with one
// phase, 0.372 with two, 0.430 with four. With 351 entries it does: 110,592 ions 135 us with four phases, 157 with two,
// 147 with eight; 175,616 ions 210 with four, 300 with one.
constexpr int64_t kMostThreads = 1 << 20, kHalfFilled = 75776, kDsfThreads = 524288;
constexpr double kLjEntries = 56.0, kDsfEntries = 8.0;
PairSplit pair_split(int64_t n, double pairs, int64_t threads, double entries) {
  PairSplit s;
  s.log2_phases = 0;
  while (s.log2_phases < 5 && (n << s.log2_phases) < kHalfFilled) ++s.log2_phases;
  while (s.log2_phases < 5 && (n << s.log2_phases) < threads && (n << (s.log2_phases + 1)) <= kMostThreads &&
         pairs >= entries * (2 << s.log2_phases))
    ++s.log2_phases;
  s.atoms = kBlock >> s.log2_phases;
  s.blocks = ceil_div(n, s.atoms);
  return s;
}

// Whether the gathers are worth a launch that packs the atoms first. In small systems, and in larger ones with few pairs, it
// costs more than it gives: 400 atoms 11.0 us packed, 9.5 from the caller's arrays, at any density; 4000 atoms with 78
// entries 13.5, 12.7 (with 345 entries 19.8, 18.9); 12,000 with 33 entries 13.5, 12.7, with 78 17.6, 17.0, with 344 36.1,
// 40.5; 26,000 with 0.3 entries 11.2, 9.9, with 78 21.9, 24.9; DSF at the same sizes 10.0, 8.6; 15.6, 14.6 (30.2, 29.9);
// 17.6, 16.6, 25.9, 24.8, 60.7, 63.7; 10.9, 9.4, 38.7, 40.1. The same results bit for bit.
bool pack_gathers(int64_t n, double pairs) { return n >= 32768 || (n >= 6000 && (double)n * pairs >= 1e6); }

// Sums the phases' values of every atom of the block in phase order; the result is in phase 0's threads.
__device__ __forceinline__ void sum_phases(const PairSplit& sp, double (&v)[4]) {
  if (sp.log2_phases == 0) return;
  __shared__ double part[4][kBlock];
#pragma unroll
  for (int c = 0; c < 4; ++c) part[c][threadIdx.x] = v[c];
  __syncthreads();
  if ((int)threadIdx.x >= sp.atoms) return;
  for (int ph = 1; ph < (1 << sp.log2_phases); ++ph) {
#pragma unroll
    for (int c = 0; c < 4; ++c) v[c] += part[c][ph * sp.atoms + threadIdx.x];
  }
}

// LJ forces and energy, FP64. At 1M atoms (78 list entries each) the gathers bound it: L1 serves one 32-byte record per
// cycle, 0.29 ms for 82M entries, and the kernel takes 0.30 (one thread per atom over the caller's arrays, with branches
// around each pair and three rounding instructions per minimum image: 0.67). Three gathers and the next list entries
// in flight at 64 registers; more of either loses the occupancy that hides the FP64 chains (0.32 to 0.44 measured). An
// 864-atom box: 52 -> 5.8 us; 256 atoms without a list: 92 -> 6.8. PACKED gathers one 256-bit record per neighbour,
// otherwise from the caller's arrays (pack_gathers; the entry point without a work buffer). The list variants spill 8
// (ONE) to 24 bytes at the 64 registers that four blocks per SM leave. ONE: a single species, its constants in registers;
// else the species-pair tables are staged in shared memory (a kernel parameter indexed per thread serialises).
template <bool DENSE, bool PACKED, bool ONE>
__global__ void __launch_bounds__(kBlock, 4) k_lj64(const double* __restrict__ pos, const int32_t* __restrict__ sp,
                                                  const Packed* __restrict__ pk, int64_t n, ImageBox box,
                                                  const int32_t* __restrict__ nbr, const int32_t* __restrict__ nnb,
                                                  int maxnb, const __grid_constant__ LJTab t, PairSplit split,
                                                  double* __restrict__ force, double* partials, unsigned int* ticket,
                                                  double* energy) {
  __shared__ double tab[3][ONE ? 1 : ACS_MAX_SPECIES * ACS_MAX_SPECIES];
  if (!ONE) {
    for (int q = threadIdx.x; q < t.ns * t.ns; q += blockDim.x) {
      tab[0][q] = t.eps[q];
      tab[1][q] = t.sig2[q];
      tab[2][q] = t.rc2[q];
    }
    __syncthreads();
  }
  const int a = threadIdx.x & (split.atoms - 1), phase = threadIdx.x >> (8 - split.log2_phases);
  const int phases = 1 << split.log2_phases;
  const int64_t i = (int64_t)blockIdx.x * split.atoms + a;
  constexpr int kU = 3;
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  if (i < n) {
    Packed me;
    if (PACKED) {
      me = ld_packed(pk + i);
    } else {
      me.x = pos[3 * i];
      me.y = pos[3 * i + 1];
      me.z = pos[3 * i + 2];
    }
    const int si = ONE ? 0 : (PACKED ? __double2loint(me.w) : sp[i]) * t.ns;
    const double s1 = t.sig2[0], c1 = t.rc2[0];
    // One block of U neighbours, without branches but for the boundary's minimum images: the terms of a neighbour
    // outside the cutoff (3 in 10 list entries) are formed and dropped by a zero 1/r^2, so the U chains of dependent
    // FP64 operations overlap; the energy shift is counted apart.
    double cnt = 0.0;   // neighbours inside (ONE), or their sum of epsilon
    auto block = [&](const Packed* o, const bool* ok, auto tag) {
      constexpr int W = decltype(tag)::value;
      double d[W][3];
      bool near = true;
#pragma unroll
      for (int q = 0; q < W; ++q) {
        d[q][0] = sub(o[q].x, me.x);
        d[q][1] = sub(o[q].y, me.y);
        d[q][2] = sub(o[q].z, me.z);
        near = near && near_image(d[q][0], d[q][1], d[q][2], box);
      }
      if (!near) {
#pragma unroll
        for (int q = 0; q < W; ++q) image3(d[q][0], d[q][1], d[q][2], box);
      }
#pragma unroll
      for (int q = 0; q < W; ++q) {
        const double r2 = norm2(d[q][0], d[q][1], d[q][2]);
        const int p = ONE ? 0 : si + __double2loint(o[q].w);
        const double e = ONE ? 1.0 : tab[0][p];
        const bool in = ok[q] && r2 < (ONE ? c1 : tab[2][p]) && e > 0.0;
        const double ir2 = in ? recip(r2) : 0.0;
        const double sr2 = (ONE ? s1 : tab[1][p]) * ir2;
        const double sr6 = sr2 * sr2 * sr2;
        const double w = fma(sr6, sr6, -sr6);
        v[3] = ONE ? v[3] + w : fma(e, w, v[3]);
        if (in) cnt += e;
        // 2 sr6^2 - sr6 in one rounding: formed from w it took two, and one pair's force was up to 6% further off (root
        // mean square, 1.06 against 0.99 units of 2^-53 of its terms at 1.2 to 1.5 sigma)
        const double c = (ONE ? ir2 : e * ir2) * fma(sr6 + sr6, sr6, -sr6);
        if (in) {   // not 0 * d: an atom that is not finite has no neighbours and must not reach their sums
          v[0] = fma(c, d[q][0], v[0]);
          v[1] = fma(c, d[q][1], v[1]);
          v[2] = fma(c, d[q][2], v[2]);
        }
      }
    };
    auto gather = [&](int32_t j) {
      Packed o;
      if (PACKED) {
        o = ld_packed(pk + j);
      } else {
        o.x = pos[3 * (int64_t)j];
        o.y = pos[3 * (int64_t)j + 1];
        o.z = pos[3 * (int64_t)j + 2];
        o.w = ONE ? 0.0 : __hiloint2double(0, sp[j]);
      }
      return o;
    };
    const int32_t* __restrict__ row = DENSE ? nullptr : nbr + nbr_slot(i, 0, maxnb);
    const int64_t m = DENSE ? n : (int64_t)min(nnb[i], maxnb);
    // list entry kq of this atom (-1 past the end); all atoms in turn without a list
    auto entry = [&](int64_t kq) -> int32_t {
      if (DENSE) return kq < m && kq != i ? (int32_t)kq : -1;
      return kq < m ? __ldcs(row + kq * 32) : -1;
    };
    int32_t jn[kU];
#pragma unroll
    for (int q = 0; q < kU; ++q) jn[q] = entry(phase + q * phases);
    for (int64_t k = phase; k < m; k += kU * phases) {
      bool ok[kU];
      Packed o[kU];
#pragma unroll
      for (int q = 0; q < kU; ++q) {   // a missing entry gathers the atom itself and is left out
        ok[q] = jn[q] >= 0;
        o[q] = gather(ok[q] ? jn[q] : (int32_t)i);
      }
#pragma unroll
      for (int q = 0; q < kU; ++q) jn[q] = entry(k + (kU + q) * phases);   // the next block's entries
      block(o, ok, std::integral_constant<int, kU>{});
    }
    const double e0 = ONE ? t.eps[0] : 1.0;
    v[3] = 4.0 * e0 * (v[3] - t.shift6 * cnt);
    v[0] *= -24.0 * e0;
    v[1] *= -24.0 * e0;
    v[2] *= -24.0 * e0;
    if (ONE && !(e0 > 0.0)) v[0] = v[1] = v[2] = v[3] = 0.0;
  }
  sum_phases(split, v);
  if (i < n && phase == 0) {
    force[3 * i] = v[0];
    force[3 * i + 1] = v[1];
    force[3 * i + 2] = v[2];
  }
  double u[1] = {phase == 0 ? 0.5 * v[3] : 0.0};
  block_sum_finish<1>(u, partials, ticket, energy);
}

template <bool PACKED, bool ONE>
void launch_lj64(const double* pos, const int32_t* sp, const Packed* pk, int64_t n, const ImageBox& b, const int32_t* nbr,
                 const int32_t* nnb, int maxnb, const LJTab& t, const PairSplit& split, double* force, double* partials,
                 unsigned int* ticket, double* energy, cudaStream_t s) {
  if (nbr)
    k_lj64<false, PACKED, ONE><<<(int)split.blocks, kBlock, 0, s>>>(pos, sp, pk, n, b, nbr, nnb, maxnb, t, split, force,
                                                                    partials, ticket, energy);
  else
    k_lj64<true, PACKED, ONE><<<(int)split.blocks, kBlock, 0, s>>>(pos, sp, pk, n, b, nullptr, nullptr, 0, t, split,
                                                                   force, partials, ticket, energy);
}

double lj_pairs_per_atom(int64_t n, bool list, const double* box3, int n_species, const double* eps_tab,
                         const double* sig_tab, double cutoff) {
  double sig = 0.0;   // the largest of a pair that interacts
  for (int a = 0; a < n_species * n_species; ++a)
    if (eps_tab[a] > 0.0) sig = std::max(sig, sig_tab[a]);
  return pairs_per_atom(n, list, box3, cutoff * sig);
}

LJTab lj_tables(int n_species, const double* eps_tab, const double* sig_tab, double cutoff) {
  LJTab t;
  t.ns = n_species;
  for (int a = 0; a < n_species * n_species; ++a) {
    t.eps[a] = eps_tab[a];
    t.sig2[a] = sig_tab[a] * sig_tab[a];                       // sig ** 2
    const double rc = cutoff * sig_tab[a];
    t.rc2[a] = rc * rc;                                        // (cutoff * sig) ** 2
  }
  const double c2 = cutoff * cutoff;
  const double src6 = (1.0 / c2) * (1.0 / c2) * (1.0 / c2);
  t.shift6 = src6 * src6 - src6;
  return t;
}

// DSF forces and energy, FP64, the gather and the list entry after it in flight (PACKED as for k_lj64). Bound
// by FP64 issue: about 90 FP64 operations per list entry (two thirds of the entries lie inside the cutoff, but nearly
// every warp holds one that does), half the pipe's rate on 64,000 ions. 4096 ions (351 list entries each): 430 us with
// one thread per atom, sqrt, erfc, exp and two divisions a pair, 34 with the split, 28 with erfc_exp; 64,000 ions:
// 640, 301 and 229.
template <bool DENSE, bool PACKED>
__global__ void __launch_bounds__(kBlock, 4) k_dsf64(const double* __restrict__ pos, const double* __restrict__ q,
                                                      const Packed* __restrict__ pk, int64_t n, ImageBox box,
                                                      const int32_t* __restrict__ nbr, const int32_t* __restrict__ nnb,
                                                      int maxnb, const int32_t* __restrict__ ex_start,
                                                      const int32_t* __restrict__ ex_idx, DSFPar P, PairSplit split,
                                                      double* __restrict__ force, double* partials,
                                                      unsigned int* ticket, double* energy) {
  const int a = threadIdx.x & (split.atoms - 1), phase = threadIdx.x >> (8 - split.log2_phases);
  const int phases = 1 << split.log2_phases;
  const int64_t i = (int64_t)blockIdx.x * split.atoms + a;
  double v[4] = {0.0, 0.0, 0.0, 0.0};
  double qi = 0.0;
  if (i < n) {
    auto gather = [&](int64_t j) {
      if (PACKED) return ld_packed(pk + j);
      Packed o;
      o.x = pos[3 * j];
      o.y = pos[3 * j + 1];
      o.z = pos[3 * j + 2];
      o.w = q[j];
      return o;
    };
    const Packed me = gather(i);
    qi = me.w;
    const int xs = ex_start ? ex_start[i] : 0, xe = ex_start ? ex_start[i + 1] : 0;
    const int32_t* __restrict__ row = DENSE ? nullptr : nbr + nbr_slot(i, 0, maxnb);
    const int64_t m = DENSE ? n : (int64_t)min(nnb[i], maxnb);
    // list entry k of this atom, the atom itself past the end; all atoms in turn without a list
    auto entry = [&](int64_t k) { return k < m ? (DENSE ? (int32_t)k : __ldcs(row + k * 32)) : (int32_t)i; };
    int32_t jn = entry(phase);
    for (int64_t k = phase; k < m; k += phases) {
      const int32_t j = jn;
      const Packed o = gather(j);
      jn = entry(k + phases);
      double dx = sub(o.x, me.x), dy = sub(o.y, me.y), dz = sub(o.z, me.z);
      if (!near_image(dx, dy, dz, box)) image3(dx, dy, dz, box);
      const double r2 = norm2(dx, dy, dz);
      if (!(r2 < P.rc2) || (DENSE && j == i)) continue;
      bool excluded = false;
      for (int x = xs; x < xe; ++x) excluded |= ex_idx[x] == j;
      if (excluded) continue;
      const double qq = qi * o.w;
      double ir;
      const double r = sqrt_recip(r2, ir);
      double gauss;
      const double er = erfc_exp(P.a, r, gauss) * ir;
      v[3] = fma(qq, er - P.erc_rc + P.fshift * (r - P.rc), v[3]);
      const double fv = qq * (fma(fma(P.c, gauss, er), ir, -P.fshift) * ir);
      v[0] = fma(-fv, dx, v[0]);
      v[1] = fma(-fv, dy, v[1]);
      v[2] = fma(-fv, dz, v[2]);
    }
  }
  sum_phases(split, v);
  double u[1] = {0.0};
  if (i < n && phase == 0) {
    force[3 * i] = P.k * v[0];
    force[3 * i + 1] = P.k * v[1];
    force[3 * i + 2] = P.k * v[2];
    u[0] = P.k * (0.5 * v[3] - qi * qi * P.self_coef);
  }
  block_sum_finish<1>(u, partials, ticket, energy);
}

// ------------------------------------------------------------------------------- integrator --
__global__ void k_kick(double* __restrict__ vel, const double* __restrict__ acc, int64_t n3, double h) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n3) vel[i] = add(vel[i], mul(h, acc[i]));  // vel += (0.5*dt) * acc
}

// pos %= box with NumPy's remainder: r = fmod(x, L); r += L if r and L differ in sign.
__device__ __forceinline__ double py_mod(double x, double L) {
  double r = fmod(x, L);
  if (r != 0.0) {
    if ((L < 0.0) != (r < 0.0)) r = add(r, L);
  } else {
    r = copysign(0.0, L);
  }
  return r;
}

// Calls f(element, atom, axis, q) for the 768 components of each block's 256 atoms, three per thread, 256 apart: the arrays
// stream, where an atom per thread reads and writes 24-byte strides.
template <class F>
__device__ __forceinline__ void for_components(int64_t n, F&& f) {
  const int64_t i0 = (int64_t)blockIdx.x * kBlock;
  const int m = (int)min((int64_t)kBlock, n - i0) * 3;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int l = threadIdx.x + kBlock * q;
    if (l < m) f(3 * i0 + l, i0 + l / 3, l % 3, q);
  }
}

// pos += dt vel, pos %= L. In (0, L) the remainder is x itself, in (L, 2L) and (-L, 0) one exact or IEEE subtraction or
// addition, as py_mod's fmod has it; its loop is left to the others. A thread's loads
// go out together: a small system takes 3.2 us so, 4.4 with each store before the next component's load, 3.1 with an atom
// per thread; 1M atoms 8.3, 10.1 and 19 us (L2 holds part of them; from HBM the bytes take 11.5).
__global__ void k_drift_wrap(double* __restrict__ pos, const double* __restrict__ vel, int64_t n, double dt, ImageBox box) {
  double p[3], v[3];
  for_components(n, [&](int64_t e, int64_t, int, int q) {
    p[q] = pos[e];
    v[q] = vel[e];
  });
  for_components(n, [&](int64_t e, int64_t, int d, int q) {
    double x = add(p[q], mul(dt, v[q]));
    if (box.periodic) {
      const double L = d == 0 ? box.L[0] : d == 1 ? box.L[1] : box.L[2];
      if (!(x > 0.0 && x < L)) x = x > L && x < 2.0 * L ? sub(x, L) : (x < 0.0 && x > -L ? add(x, L) : py_mod(x, L));
    }
    pos[e] = x;
  });
}

// Langevin O-step: vel = c1 * vel + sig[atom] * noise (accusim/integrators.py:66-67, no FMA).
__global__ void k_langevin_ou(double* __restrict__ vel, const double* __restrict__ noise,
                              const double* __restrict__ sig, int64_t n3, double c1) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n3) vel[i] = add(mul(c1, vel[i]), mul(sig[i / 3], noise[i]));
}

struct MassTab {
  double m[ACS_MAX_SPECIES];
};

__global__ void k_accel(double* __restrict__ acc, const double* __restrict__ force, const int32_t* __restrict__ sp,
                        const __grid_constant__ MassTab mt, int64_t n) {
  for_components(n, [&](int64_t e, int64_t i, int, int) { acc[e] = div(force[e], mt.m[sp[i]]); });   // 1M atoms 20 -> 11 us
}

__global__ void __launch_bounds__(kBlock) k_conserved(const double* __restrict__ pos, const double* __restrict__ vel,
                                                       const int32_t* __restrict__ sp, MassTab mt, int64_t n,
                                                       double* partials, unsigned int* ticket, double* out) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  if (i < n) {
    const double m = mt.m[sp[i]];
    const double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
    const double vx = vel[3 * i], vy = vel[3 * i + 1], vz = vel[3 * i + 2];
    v[0] = 0.5 * (m * (vx * vx) + m * (vy * vy) + m * (vz * vz));
    const double px = m * vx, py = m * vy, pz = m * vz;
    v[1] = px;
    v[2] = py;
    v[3] = pz;
    v[4] = y * pz - z * py;
    v[5] = z * px - x * pz;
    v[6] = x * py - y * px;
  }
  block_sum_finish<7>(v, partials, ticket, out);
}

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

inline int64_t grid_cells(const acs_grid* g) { return (int64_t)g->ncell[0] * g->ncell[1] * g->ncell[2]; }

// CPython float floor division (Objects/floatobject.c float_divmod), as used by `span // rc`.
double py_floordiv(double a, double b) {
  double mod = fmod(a, b);
  double dv = (a - mod) / b;
  if (mod != 0.0) {
    if ((b < 0) != (mod < 0)) dv -= 1.0;
  }
  double fl;
  if (dv != 0.0) {
    fl = floor(dv);
    if (dv - fl > 0.5) fl += 1.0;
  } else {
    fl = copysign(0.0, a / b);
  }
  return fl;
}

constexpr int kRdfMaxBins = 8192;   // shared-memory counts per block

// Cell binning shared by the list build and the pair histogram: atoms counted into cells, exclusive scan,
// scatter, deterministic in-cell order (ascending atom index).
struct CellBins {
  int32_t *cell_of, *start;
  float4* screen;   // cell order
};
int bin_cells(const double* pos, int64_t n, const acs_grid* g, void* work, cudaStream_t s, CellBins& cb) {
  const int64_t nc = grid_cells(g);
  const int64_t nchunks = ceil_div(nc + 1, kScanChunk);
  char* w = (char*)(((uintptr_t)work + 255) & ~(uintptr_t)255);
  cb.screen = (float4*)w; w += align256((size_t)n * 16);
  cb.cell_of = (int32_t*)w; w += align256(n * 4);
  int32_t* count = (int32_t*)w; w += align256((nc + 1) * 4);
  cb.start = (int32_t*)w; w += align256((nc + 1) * 4);
  int32_t* unsorted = (int32_t*)w; w += align256(n * 4);
  int32_t* place = (int32_t*)w; w += align256(n * 4);
  int32_t* sums = (int32_t*)w;
  GridDev gd = to_dev(g);
  const int nb = (int)ceil_div(n, kBlock);
  if (n <= kBinAtoms && nc < kBinCells) {
    k_bin_block<<<1, 1024, 0, s>>>(pos, (int)n, gd, (int)nc, cb.cell_of, cb.start, unsorted);
  } else {
    if (cudaMemsetAsync(count, 0, (nc + 1) * 4, s) != cudaSuccess) return 1;
    k_bin<<<nb, kBlock, 0, s>>>(pos, n, gd, cb.cell_of, place, count);
    k_scan_chunks<<<(int)nchunks, kScanThreads, 0, s>>>(count, cb.start, nc + 1, sums);
    k_scan_sums<<<1, kScanThreads, 0, s>>>(sums, nchunks, nullptr);
    k_scan_add<<<(int)nchunks, 256, 0, s>>>(cb.start, nc + 1, sums);
    k_scatter<<<nb, kBlock, 0, s>>>(cb.cell_of, place, n, cb.start, unsorted);
  }
  k_rank_cells<<<nb, kBlock, 0, s>>>(pos, cb.cell_of, n, gd, screen_of(g, g->rc2), cb.start, unsorted, cb.screen);
  return 0;
}

// Whether a lane per atom on its own stencil beats a warp per atom (k_list_sparse, k_rdf_sparse): where cells hold few
// atoms, a warp's 32 lanes meet stretches of a few candidates, if there are atoms enough to fill the chip. List build, warp
// against lane per atom, at 0.7 and 3.4 atoms a cell: 16,000 atoms 58, 58 against 53, 70 us; 32,000 76, 82 against 52, 66;
// 250,000 322, 362 against 84, 123; 10^6 1184, 1338 against 214, 371 (a thread per atom testing every
// candidate in FP64 499, 1184). At 4.6 a cell the warp per cell takes over (32,000 atoms 60 against 80). Histogram: 32,000
// atoms 58, 63 against 58, 78; 64,000 79, 89 against 58, 85; 10^6 676, 790 against 198, 294 (in FP64 530, 1344).
constexpr int64_t kSparseList = 20000, kSparseRdf = 50000;
bool sparse_cells(int64_t n, int64_t nc, int64_t least) { return n >= least && n < 4 * nc; }

}  // namespace

// ===================================================================================== C ABI ==
extern "C" {

int acs_abi_version(void) { return ACS_ABI_VERSION; }

const char* acs_status_string(int s) {
  switch (s) {
    case ACS_OK: return "ok";
    case ACS_ERR_ARG: return "bad argument";
    case ACS_ERR_WORKSPACE: return "workspace too small";
    case ACS_ERR_CUDA: return "CUDA runtime error";
    case ACS_ERR_LIST_OVERFLOW: return "neighbour list capacity exceeded";
    case ACS_ERR_NONFINITE: return "non-finite force or position";
    case ACS_ERR_TIMEOUT: return "device barrier wait timed out";
    case ACS_ERR_UNSUPPORTED: return "unsupported size or mode";
    case ACS_ERR_NO_DEVICE: return "no CUDA device";
    default: return "unknown status";
  }
}

int acs_device_info(int* sm_count, int* cc_major, int* cc_minor) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return ACS_ERR_NO_DEVICE;
  cudaDeviceProp p;
  if (cudaGetDeviceProperties(&p, dev) != cudaSuccess) return ACS_ERR_NO_DEVICE;
  if (sm_count) *sm_count = p.multiProcessorCount;
  if (cc_major) *cc_major = p.major;
  if (cc_minor) *cc_minor = p.minor;
  return ACS_OK;
}

int acs_grid_setup(acs_grid* g, const double* box3, int periodic, const double* lo3, const double* hi3, double rc) {
  if (!g || !(rc > 0.0) || (!box3 && (!lo3 || !hi3))) return ACS_ERR_ARG;
  for (int k = 0; k < 3; ++k) {
    double lo, span;
    if (box3) {
      lo = 0.0;
      span = box3[k];
    } else {
      lo = lo3[k];
      span = std::max(hi3[k] - lo, rc);
    }
    if (!(span > 0.0)) return ACS_ERR_ARG;
    double nc = std::max(py_floordiv(span, rc), 1.0);
    if (nc > 2097152.0) return ACS_ERR_UNSUPPORTED;
    int ic = (int)nc;
    if (periodic && box3 && ic < 3) ic = 1;
    g->lo[k] = lo;
    g->span[k] = span;
    g->box[k] = box3 ? box3[k] : 0.0;
    g->ncell[k] = ic;
  }
  if (grid_cells(g) > (int64_t)INT32_MAX / 2) return ACS_ERR_UNSUPPORTED;
  g->periodic = (periodic && box3) ? 1 : 0;
  g->rc = rc;
  g->rc2 = rc * rc;
  return ACS_OK;
}

size_t acs_nlist_work_bytes(int64_t n, const acs_grid* g) {
  if (!g || n < 0) return 0;
  const int64_t nc = grid_cells(g);
  const int64_t nchunks = ceil_div(nc + 1, kScanChunk);
  return 256 + align256((size_t)n * 16) + align256(n * 4) + 2 * align256((nc + 1) * 4) + 2 * align256(n * 4) +
         align256((nchunks + 1) * 4);
}

int acs_nlist_build(const double* pos, int64_t n, const acs_grid* g, int32_t maxnb, int32_t* nbr, int32_t* nnb,
                    void* work, size_t work_bytes, acs_dev_status* status, void* stream) {
  if (!g || n < 0 || maxnb < 1 || n > INT32_MAX || (n > 0 && (!pos || !nbr || !nnb || !work || !status)))
    return ACS_ERR_ARG;
  if (work_bytes < acs_nlist_work_bytes(n, g)) return ACS_ERR_WORKSPACE;
  if (n == 0) return ACS_OK;
  cudaStream_t s = (cudaStream_t)stream;
  CellBins cb;
  if (bin_cells(pos, n, g, work, s, cb)) return ACS_ERR_CUDA;
  const GridDev gd = to_dev(g);
  const Screen f = screen_of(g, g->rc2);
  const int64_t nc = grid_cells(g);
  const bool wrap = g->periodic && (g->ncell[0] < 4 || g->ncell[1] < 4 || g->ncell[2] < 4);
  // From 1024 cells on a warp per cell wins (16,384 LJ atoms, 857 cells: both 72 us for the whole build; 55,296 atoms:
  // 87 us against 144; 1,048,576: 0.71 ms against 1.97; 4000 atoms in 125 cells: 72 against 42), if the cells hold
  // atoms to share the staging.
  if (!wrap && nc >= 1024 && n >= 4 * nc) {
    const unsigned chunks = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ceil_div(2 * n, 32 * nc), 64));
    k_list_cells<<<dim3((unsigned)ceil_div(nc, kBlock / 32), chunks), kBlock, 0, s>>>(pos, gd, f, nc, cb.start, cb.screen,
                                                                                     maxnb, nbr, nnb, status);
  } else if (sparse_cells(n, nc, kSparseList)) {
    (wrap ? k_list_sparse<true> : k_list_sparse<false>)<<<(int)ceil_div(n, kBlock), kBlock, 0, s>>>(
        pos, n, gd, f, cb.cell_of, cb.start, cb.screen, maxnb, nbr, nnb, status);
  } else {
    // 4 loads in flight where a stretch of 3 cells fills them (4096 ions in 27 cells: 53 us with 1, 49 with 2, 45 with 4),
    // else 2 (8000 ions in 216 cells: 41, 36, 39)
    const bool long_rows = 3 * n >= 256 * nc;
    auto kernel = wrap ? (long_rows ? k_list_atoms<true, 4> : k_list_atoms<true, 2>)
                       : (long_rows ? k_list_atoms<false, 4> : k_list_atoms<false, 2>);
    kernel<<<(int)ceil_div(n, kBlock / 32), kBlock, 0, s>>>(
        pos, n, gd, f, cb.cell_of, cb.start, cb.screen, maxnb, nbr, nnb, status);
  }
  return launch_status();
}

size_t acs_rdf_work_bytes(int64_t n, const acs_grid* g) { return acs_nlist_work_bytes(n, g); }

int acs_rdf_hist(const double* pos, const int32_t* sp, int64_t n, const acs_grid* g, int32_t species, int32_t bins,
                 double rmax, unsigned long long* hist, void* work, size_t work_bytes, void* stream) {
  if (!g || n < 0 || n > INT32_MAX || bins < 1 || bins > kRdfMaxBins || !(rmax > 0.0) || !hist ||
      (n > 0 && (!pos || !work || (species >= 0 && !sp))))
    return ACS_ERR_ARG;
  if (!g->periodic || !(g->rc >= rmax)) return ACS_ERR_ARG;   // cells no narrower than rmax, periodic box
  if (work_bytes < acs_rdf_work_bytes(n, g)) return ACS_ERR_WORKSPACE;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemsetAsync(hist, 0, sizeof(unsigned long long) * bins, s) != cudaSuccess) return ACS_ERR_CUDA;
  if (n == 0) return ACS_OK;
  CellBins cb;
  if (bin_cells(pos, n, g, work, s, cb)) return ACS_ERR_CUDA;
  const bool wrap = g->ncell[0] < 4 || g->ncell[1] < 4 || g->ncell[2] < 4;
  // one round of blocks (up to 4 on each of 148 SMs), so that a block's counts are added to the result once
  const int blocks = (int)std::min<int64_t>(592, ceil_div(n, kBlock / 32));
  const bool sparse = sparse_cells(n, grid_cells(g), kSparseRdf);
  auto kernel = sparse ? (wrap ? k_rdf_sparse<true> : k_rdf_sparse<false>) : (wrap ? k_rdf<true> : k_rdf<false>);
  kernel<<<blocks, kBlock, sizeof(unsigned int) * bins, s>>>(
      pos, sp, n, to_dev(g), screen_of(g, square_reaching(nextafter(rmax, HUGE_VAL))), cb.cell_of,
      cb.start, cb.screen, species, bins, rmax, rmax / bins, hist);
  return launch_status();
}

int acs_nlist_pairs(const int32_t* nbr, const int32_t* nnb, int64_t n, int32_t maxnb, int32_t* pi, int32_t* pj,
                    int64_t cap, unsigned long long* count_dev, void* stream) {
  if (n < 0 || maxnb < 1 || !count_dev || (n > 0 && (!nbr || !nnb)) || (cap > 0 && (!pi || !pj))) return ACS_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (cudaMemsetAsync(count_dev, 0, sizeof(unsigned long long), s) != cudaSuccess) return ACS_ERR_CUDA;
  if (n == 0) return ACS_OK;
  k_pairs<<<(int)ceil_div(n, kBlock), kBlock, 0, s>>>(nbr, nnb, n, maxnb, pi, pj, cap, count_dev);
  return launch_status();
}

int acs_nlist_displacement(const double* pos, const double* pos0, int64_t n, const double* box3, int periodic,
                           double half_skin2, int32_t* flag_dev, void* stream) {
  if (n < 0 || !flag_dev || (n > 0 && (!pos || !pos0))) return ACS_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const ImageBox box = image_box(box3, periodic);
  if (n > 0 && n <= kMovedAtoms) {
    k_displacement_block<<<1, 1024, 0, s>>>(pos, pos0, (int)n, box, half_skin2, flag_dev);
    return launch_status();
  }
  if (cudaMemsetAsync(flag_dev, 0, 4, s) != cudaSuccess) return ACS_ERR_CUDA;
  if (n == 0) return ACS_OK;
  k_displacement<<<(int)ceil_div(n, kBlock), kBlock, 0, s>>>(pos, pos0, n, box, half_skin2, flag_dev);
  return launch_status();
}

// Energy partials (one per block of the pair kernels), ticket, packed positions; 256 bytes to align them in the
// caller's buffer.
static int64_t force_blocks(int64_t n) {   // the most of any split: more than one phase ends at kMostThreads
  n = std::max<int64_t>(n, 1);
  return std::max(ceil_div(n, kBlock), std::min<int64_t>(ceil_div(n, kBlock / 32), kMostThreads / kBlock));
}
size_t acs_force_work_bytes(int64_t n) {
  return align256(force_blocks(n) * 8) + 256 + align256((size_t)std::max<int64_t>(n, 1) * sizeof(Packed)) + 256;
}

// Carves a force call's work buffer and clears the ticket; with `packed`, by the packing kernel, which it launches.
static int force_setup(const double* pos, const int32_t* sp, const double* q, int64_t n, void* work, size_t work_bytes,
                       const PairSplit& split, bool packed, double** partials, unsigned int** ticket, Packed** pk,
                       cudaStream_t s) {
  if (work_bytes < acs_force_work_bytes(n) || !work) return ACS_ERR_WORKSPACE;
  char* w = (char*)(((uintptr_t)work + 255) & ~(uintptr_t)255);
  *partials = (double*)w; w += align256(force_blocks(n) * 8);
  *ticket = (unsigned int*)w; w += 256;
  *pk = (Packed*)w;
  if (!packed)   // one block adds up without the ticket
    return split.blocks == 1 || cudaMemsetAsync(*ticket, 0, 4, s) == cudaSuccess ? ACS_OK : ACS_ERR_CUDA;
  k_pack<<<(int)ceil_div(n, kBlock), kBlock, 0, s>>>(pos, sp, q, n, *pk, *ticket);
  return launch_status();
}

static int reduce_setup(void* work, size_t work_bytes, size_t need, int64_t nblocks, int width, double** partials,
                        unsigned int** ticket, cudaStream_t s) {
  if (work_bytes < need) return ACS_ERR_WORKSPACE;
  *partials = (double*)work;
  *ticket = (unsigned int*)((char*)work + align256(nblocks * width * 8));
  return cudaMemsetAsync(*ticket, 0, 4, s) == cudaSuccess ? ACS_OK : ACS_ERR_CUDA;
}

int acs_lj_fp64(const double* pos, const int32_t* sp, int64_t n, const double* box3, int periodic,
                const int32_t* nbr, const int32_t* nnb, int32_t maxnb, int32_t n_species, const double* eps_tab,
                const double* sig_tab, double cutoff, double* force, double* energy_dev, void* work,
                size_t work_bytes, void* stream) {
  if (n < 1 || n > INT32_MAX || !pos || !sp || !force || !energy_dev || !eps_tab || !sig_tab || n_species < 1 ||
      n_species > ACS_MAX_SPECIES || !(cutoff > 0.0) || (nbr && (!nnb || maxnb < 1)))
    return ACS_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  double* partials;
  unsigned int* ticket;
  Packed* pk;
  const double pairs = lj_pairs_per_atom(n, nbr, box3, n_species, eps_tab, sig_tab, cutoff);
  const PairSplit split = pair_split(n, pairs, kMostThreads, kLjEntries);
  const bool packed = pack_gathers(n, pairs);
  int st = force_setup(pos, sp, nullptr, n, work, work_bytes, split, packed, &partials, &ticket, &pk, s);
  if (st) return st;
  const LJTab t = lj_tables(n_species, eps_tab, sig_tab, cutoff);
  const ImageBox b = image_box(box3, periodic);
  auto launch = n_species == 1 ? (packed ? launch_lj64<true, true> : launch_lj64<false, true>)
                               : (packed ? launch_lj64<true, false> : launch_lj64<false, false>);
  launch(pos, sp, pk, n, b, nbr, nnb, maxnb, t, split, force, partials, ticket, energy_dev, s);
  return launch_status();
}

int acs_dsf_fp64(const double* pos, const double* q, int64_t n, const double* box3, int periodic,
                 const int32_t* nbr, const int32_t* nnb, int32_t maxnb, const int32_t* ex_start,
                 const int32_t* ex_idx, double alpha, double rcut, double k, double* force, double* energy_dev,
                 void* work, size_t work_bytes, void* stream) {
  if (n < 1 || n > INT32_MAX || !pos || !q || !force || !energy_dev || !(rcut > 0.0) || !(alpha >= 0.0) ||
      (nbr && (!nnb || maxnb < 1)) || (ex_start && !ex_idx))
    return ACS_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  double* partials;
  unsigned int* ticket;
  Packed* pk;
  const double pairs = pairs_per_atom(n, nbr, box3, rcut);
  const PairSplit split = pair_split(n, pairs, kDsfThreads, kDsfEntries);
  const bool packed = pack_gathers(n, pairs);
  int st = force_setup(pos, nullptr, q, n, work, work_bytes, split, packed, &partials, &ticket, &pk, s);
  if (st) return st;
  DSFPar P;
  P.a = alpha;
  P.rc = rcut;
  P.rc2 = square_reaching(rcut);
  P.k = k;
  P.c = 2.0 * alpha / sqrt(M_PI);
  P.erc = erfc(alpha * rcut);
  P.erc_rc = P.erc / rcut;
  P.fshift = P.erc / (rcut * rcut) + P.c * exp(-((alpha * rcut) * (alpha * rcut))) / rcut;
  P.self_coef = P.erc / (2.0 * rcut) + alpha / sqrt(M_PI);
  const ImageBox b = image_box(box3, periodic);
  auto kernel = nbr ? (packed ? k_dsf64<false, true> : k_dsf64<false, false>)
                    : (packed ? k_dsf64<true, true> : k_dsf64<true, false>);
  kernel<<<(int)split.blocks, kBlock, 0, s>>>(pos, q, pk, n, b, nbr, nnb, maxnb, ex_start, ex_idx, P, split, force, partials,
                                              ticket, energy_dev);
  return launch_status();
}

int acs_vv_kick(double* vel, const double* acc, int64_t n, double half_dt, void* stream) {
  if (n < 0 || (n > 0 && (!vel || !acc))) return ACS_ERR_ARG;
  if (n == 0) return ACS_OK;
  k_kick<<<(int)ceil_div(3 * n, kBlock), kBlock, 0, (cudaStream_t)stream>>>(vel, acc, 3 * n, half_dt);
  return launch_status();
}

int acs_vv_drift_wrap(double* pos, const double* vel, int64_t n, double dt, const double* box3, int periodic,
                      void* stream) {
  if (n < 0 || (n > 0 && (!pos || !vel))) return ACS_ERR_ARG;
  if (n == 0) return ACS_OK;
  k_drift_wrap<<<(int)ceil_div(n, kBlock), kBlock, 0, (cudaStream_t)stream>>>(pos, vel, n, dt,
                                                                                image_box(box3, periodic));
  return launch_status();
}

int acs_langevin_ou(double* vel, const double* noise, const double* sig, int64_t n, double c1, void* stream) {
  if (n < 0 || (n > 0 && (!vel || !noise || !sig))) return ACS_ERR_ARG;
  if (n == 0) return ACS_OK;
  k_langevin_ou<<<(int)ceil_div(3 * n, kBlock), kBlock, 0, (cudaStream_t)stream>>>(vel, noise, sig, 3 * n, c1);
  return launch_status();
}

int acs_vv_accel(double* acc, const double* force, const int32_t* sp, const double* species_mass, int32_t n_species,
                 int64_t n, void* stream) {
  if (n < 0 || (n > 0 && (!acc || !force || !sp || !species_mass)) || n_species < 1 || n_species > ACS_MAX_SPECIES)
    return ACS_ERR_ARG;
  if (n == 0) return ACS_OK;
  MassTab mt;
  for (int a = 0; a < ACS_MAX_SPECIES; ++a) mt.m[a] = a < n_species ? species_mass[a] : 1.0;
  k_accel<<<(int)ceil_div(n, kBlock), kBlock, 0, (cudaStream_t)stream>>>(acc, force, sp, mt, n);
  return launch_status();
}

size_t acs_reduce_work_bytes(int64_t n) { return align256(std::max<int64_t>(ceil_div(n, kBlock), 1) * 7 * 8) + 256; }

int acs_reduce_conserved(const double* pos, const double* vel, const int32_t* sp, const double* species_mass,
                         int32_t n_species, int64_t n, double* out_dev, void* work, size_t work_bytes, void* stream) {
  if (n < 1 || !pos || !vel || !sp || !species_mass || !out_dev || n_species < 1 || n_species > ACS_MAX_SPECIES)
    return ACS_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const int64_t nb = ceil_div(n, kBlock);
  double* partials;
  unsigned int* ticket;
  int st = reduce_setup(work, work_bytes, acs_reduce_work_bytes(n), nb, 7, &partials, &ticket, s);
  if (st) return st;
  MassTab mt;
  for (int a = 0; a < ACS_MAX_SPECIES; ++a) mt.m[a] = a < n_species ? species_mass[a] : 0.0;
  k_conserved<<<(int)nb, kBlock, 0, s>>>(pos, vel, sp, mt, n, partials, ticket, out_dev);
  return launch_status();
}

}  // extern "C"

// ============================================================= allocation-free LJ force entry point ==
// Some callers cannot allocate device memory when they need forces: code that owns every byte of the GPU
// through its own pool, real-time loops that forbid allocation after start-up, or plug-in hosts that hand
// out only input and output buffers. acs_lj_fp64_noalloc serves them: it runs the same FP64 LJ kernel as
// acs_lj_fp64, but its reduction scratch (one FP64 partial per block plus a completion counter) lives in the
// fixed device array below instead of a caller-provided work buffer, and it always gathers from the caller's arrays.
//
// The array is 64 KiB + 256 B and exists on every GPU that loads this library until the process exits; it bounds
// n at kNoAllocMaxAtoms = 2,097,152 atoms: a block takes 256 atoms, or fewer (down to 8) while the atoms' threads
// stay within kMostThreads. All calls share it, so calls whose work overlaps on the
// GPU (different streams, or different host threads on one device) race and corrupt each other's energy;
// serialise them. The completion counter is cleared at the start of every call; the partials are fully
// overwritten by each call.
namespace {

constexpr int64_t kNoAllocMaxBlocks = 8192;                   // 8192 partials of 8 bytes = 64 KiB
constexpr int64_t kNoAllocMaxAtoms = kNoAllocMaxBlocks * kBlock;  // 2,097,152
static_assert(kMostThreads / kBlock <= kNoAllocMaxBlocks && 2 * kHalfFilled <= kMostThreads, "partials of every split");
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocMaxBlocks * 8 + 256];

// The address is looked up once per CUDA context (the primary context of each device, or any context a driver-API
// caller makes current): a symbol's address belongs to the context the module was loaded into, so a cache keyed
// by the device alone would hand a non-primary context, or a primary context re-created after cudaDeviceReset,
// an address it cannot use.
struct NoAllocEntry {
  int dev;
  void* ctx;
  void* ptr;
};
constexpr int kNoAllocCache = 64;
std::mutex g_noalloc_mutex;
NoAllocEntry g_noalloc_cache[kNoAllocCache];
int g_noalloc_used = 0;

// cuCtxGetCurrent through the runtime's driver entry point (no link against libcuda); null if unavailable.
using CtxGetCurrentFn = int (*)(void**);
CtxGetCurrentFn ctx_get_current() {
  static CtxGetCurrentFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return (CtxGetCurrentFn)p;
  }();
  return fn;
}

// Device address of g_noalloc_scratch in the current context, looked up on the first call in that context.
// Before the runtime has made a context current, the symbol lookup itself initialises the device's primary
// context, which is then the current one.
int noalloc_scratch(void** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) return ACS_ERR_NO_DEVICE;
  CtxGetCurrentFn get = ctx_get_current();
  void* ctx = nullptr;
  if (!get || get(&ctx) != 0) return ACS_ERR_CUDA;
  std::lock_guard<std::mutex> lock(g_noalloc_mutex);
  for (int k = 0; ctx && k < g_noalloc_used; ++k) {
    if (g_noalloc_cache[k].dev == dev && g_noalloc_cache[k].ctx == ctx) {
      *out = g_noalloc_cache[k].ptr;
      return ACS_OK;
    }
  }
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) return ACS_ERR_CUDA;
  if (!ctx && (get(&ctx) != 0 || !ctx)) return ACS_ERR_CUDA;
  if (g_noalloc_used < kNoAllocCache) g_noalloc_cache[g_noalloc_used++] = NoAllocEntry{dev, ctx, p};
  *out = p;
  return ACS_OK;
}

}  // namespace

extern "C" int acs_lj_fp64_noalloc(const double* pos, const int32_t* sp, int64_t n, const double* box3, int periodic,
                                   const int32_t* nbr, const int32_t* nnb, int32_t maxnb, int32_t n_species,
                                   const double* eps_tab, const double* sig_tab, double cutoff, double* force,
                                   double* energy_dev, void* stream) {
  if (n > kNoAllocMaxAtoms) return ACS_ERR_UNSUPPORTED;
  if (n < 1 || !pos || !sp || !force || !energy_dev || !eps_tab || !sig_tab || n_species < 1 ||
      n_species > ACS_MAX_SPECIES || !(cutoff > 0.0) || (nbr && (!nnb || maxnb < 1)))
    return ACS_ERR_ARG;
  void* scratch = nullptr;
  int st = noalloc_scratch(&scratch);
  if (st) return st;
  cudaStream_t s = (cudaStream_t)stream;
  double* partials = (double*)scratch;
  unsigned int* ticket = (unsigned int*)((char*)scratch + kNoAllocMaxBlocks * 8);
  if (cudaMemsetAsync(ticket, 0, 4, s) != cudaSuccess) return ACS_ERR_CUDA;
  const LJTab t = lj_tables(n_species, eps_tab, sig_tab, cutoff);
  const PairSplit split =
      pair_split(n, lj_pairs_per_atom(n, nbr, box3, n_species, eps_tab, sig_tab, cutoff), kMostThreads, kLjEntries);
  const ImageBox b = image_box(box3, periodic);
  if (n_species == 1)   // the same arithmetic as acs_lj_fp64, bit for bit
    launch_lj64<false, true>(pos, sp, nullptr, n, b, nbr, nnb, maxnb, t, split, force, partials, ticket, energy_dev, s);
  else
    launch_lj64<false, false>(pos, sp, nullptr, n, b, nbr, nnb, maxnb, t, split, force, partials, ticket, energy_dev, s);
  return launch_status();
}
