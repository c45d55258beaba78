// SPH particle relaxation and density on a periodic box (l3es/relax.py:16-178,
// l3es/utils.py:169-218, relaxation block of l3es/combined.py:132-142) for sm_103a.
//
// Particles: n per axis at rest (spacing dx = L / n, mass dx^dim, reference density 1),
// quintic spline kernel with smoothing length dx and cutoff 3 dx, Tait EoS with gamma 1
// and sound speed 10 u_ref.
//
// Neighbour search is a cell list rebuilt on every call:
//   k_sph_bin      wrap (optionally after an Euler predictor), cell id, cell counts
//   k_sph_scan     exclusive scan of the counts (one CTA)
//   k_sph_scatter  slot per particle (atomic, unordered)
//   k_sph_order    stable order inside each cell (rank by input index), so that neighbour
//                  sums run in a fixed order and results are bitwise reproducible; stores
//                  cell-local FP32 coordinates
//   k_sph_density  rho = m sum_j W(|r_ij|)            (kSphLanes lanes per particle, cell order)
//   k_sph_accel    pressure + transport-velocity (and viscous) accelerations
// Cells are cubes of side L / floor(n / 3) >= cutoff, so a 3^dim stencil holds every
// neighbour. Pair geometry is FP32 from cell-local coordinates (offsets below one cell
// side, so the FP32 rounding of a pair distance is ~1e-7 of dx); each lane sums its
// neighbours' FP32 terms in float-float (Ff, error-free FP32 additions: FP64 arithmetic
// is scarce on this GPU and FP64 accumulators kept its FP64 pipe 73-85% busy), the lanes
// combine in FP64, and the density-to-pressure step (rho - 1) is FP64.
#include <cuda_runtime.h>

#include <cmath>
#include <string>
#include <type_traits>

#include "l3es_internal.h"
#include "particle_kernels.cuh"

namespace l3es {

constexpr int kSphThreads = 128;
// Lanes per particle in the neighbour sums: lane q visits candidates q, q + 8, ... of every
// stencil cell and the lanes' FP64 partial sums are added by a fixed shuffle tree, so the
// summation order stays fixed (bitwise reproducible). With one thread per particle a 32^3
// relaxation call kept ~7 warps per SM, each walking ~900 candidates one load after the
// other.
constexpr int kSphLanes = 8;

struct SphGeom {
  double L;      // box side
  double inv_cs; // cells per unit length (nc / L)
  double cs_d;   // cell side L / nc (cell origins; nc * cs_d == L up to FP64 rounding)
  float cs;      // cell side (stencil offsets)
  float Lf;      // box side (FP32, for the nc == 1 minimum image)
  int nc;        // cells per axis (1: every particle is a candidate, minimum image)
  float inv_h;   // 1 / dx
  float cut2;    // (3 dx)^2
};

__device__ __forceinline__ int cell_coord(double x, const SphGeom& g) {
  int c = (int)(x * g.inv_cs);
  return c < 0 ? 0 : (c >= g.nc ? g.nc - 1 : c);
}

// Morris (1997) quintic spline without its normalisation sigma:
//   w(q) = (3-q)_+^5 - 6 (2-q)_+^5 + 15 (1-q)_+^5,  dw/dq = -5 (3-q)_+^4 + 30 (2-q)_+^4 - 75 (1-q)_+^4
__device__ __forceinline__ float quintic_w(float q) {
  const float q3 = fmaxf(0.f, 3.f - q), q2 = fmaxf(0.f, 2.f - q), q1 = fmaxf(0.f, 1.f - q);
  const float a = q3 * q3, b = q2 * q2, c = q1 * q1;
  return a * a * q3 - 6.f * (b * b * q2) + 15.f * (c * c * q1);
}
__device__ __forceinline__ float quintic_dw(float q) {
  const float q3 = fmaxf(0.f, 3.f - q), q2 = fmaxf(0.f, 2.f - q), q1 = fmaxf(0.f, 1.f - q);
  const float a = q3 * q3, b = q2 * q2, c = q1 * q1;
  return -5.f * (a * a) + 30.f * (b * b) - 75.f * (c * c);
}

template <int DIM>
__device__ __forceinline__ int cell_index(const int* ci, int nc) {
  int c = 0;
#pragma unroll
  for (int d = 0; d < DIM; ++d) c = c * nc + ci[d];
  return c;
}

// wrapped position (after x += dt * u when u != null), its cell, cell counts
template <int DIM>
__global__ void __launch_bounds__(kSphThreads)
k_sph_bin(const double* __restrict__ r, const double* __restrict__ u, double dt, long long np, SphGeom g,
          double* __restrict__ xw, int* __restrict__ cell, int* __restrict__ count) {
  pdl_begin();
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= np) return;
  int ci[DIM];
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    double x = r[j * DIM + d];
    if (u) x += dt * u[j * DIM + d];
    x = wrap_period(x, g.L);
    xw[j * DIM + d] = x;
    ci[d] = cell_coord(x, g);
  }
  const int c = cell_index<DIM>(ci, g.nc);
  cell[j] = c;
  atomicAdd(count + c, 1);
}

// exclusive scan of ncell counts by one CTA of 1024 threads: each thread sums a
// contiguous segment, the segment sums are scanned with warp shuffles
__global__ void __launch_bounds__(1024)
k_sph_scan(const int* __restrict__ count, int ncell, int* __restrict__ start, int* __restrict__ cursor) {
  pdl_begin();
  __shared__ int warp_sum[32];
  const int seg = (ncell + 1023) / 1024;
  const int b = threadIdx.x * seg, e = min(ncell, b + seg);
  int s = 0;
  for (int i = b; i < e; ++i) s += count[i];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[w] = incl;
  __syncthreads();
  if (w == 0) {
    int v = warp_sum[lane], iv = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, iv, o);
      if (lane >= o) iv += t;
    }
    warp_sum[lane] = iv - v;
  }
  __syncthreads();
  int run = warp_sum[w] + incl - s;
  for (int i = b; i < e; ++i) {
    start[i] = run;
    cursor[i] = run;
    run += count[i];
  }
  if (threadIdx.x == 1023) start[ncell] = run;
}

__global__ void __launch_bounds__(kSphThreads)
k_sph_scatter(const int* __restrict__ cell, long long np, int* __restrict__ cursor, int* __restrict__ perm0) {
  pdl_begin();
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j < np) perm0[atomicAdd(cursor + cell[j], 1)] = (int)j;
}

// slot of particle perm0[s] = cell start + number of cell members with a smaller input
// index; cell-local FP32 coordinates (and the velocity, when given) in that order
template <int DIM>
__global__ void __launch_bounds__(kSphThreads)
k_sph_order(const int* __restrict__ perm0, const int* __restrict__ cell, const int* __restrict__ start,
            const double* __restrict__ xw, const double* __restrict__ u, long long np, SphGeom g,
            int* __restrict__ perm, float4* __restrict__ xs, float4* __restrict__ us) {
  pdl_begin();
  const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= np) return;
  const int j = perm0[s];
  const int c = cell[j];
  const int b = start[c], e = start[c + 1];
  int rank = 0;
  for (int m = b; m < e; ++m) rank += perm0[m] < j;
  const int t = b + rank;
  perm[t] = j;
  float loc[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int d = 0; d < DIM; ++d) {
    const double x = xw[(long long)j * DIM + d];
    // its cell on axis d
    const int q = d == DIM - 1 ? c % g.nc : d == DIM - 2 ? c / g.nc % g.nc : c / (g.nc * g.nc);
    loc[d] = (float)(x - (double)q * g.cs_d);
  }
  xs[t] = make_float4(loc[0], loc[1], loc[2], 0.f);
  if (us) {
    float v[3] = {0.f, 0.f, 0.f};
#pragma unroll
    for (int d = 0; d < DIM; ++d) v[d] = (float)u[(long long)j * DIM + d];
    us[t] = make_float4(v[0], v[1], v[2], 0.f);
  }
}

// Visits every neighbour of a particle (cell-local position xi in cell ci) by its kSphLanes
// lanes: f(slot j, dx, dy, dz, r^2) for pairs with r^2 < cut2, the particle itself included
// (r = 0). Cells of the 3^dim stencil are wrapped; the displacement r_i - r_j is formed
// from cell-local coordinates and the stencil offset. Lane q takes candidates q, q + 8, ...
// of every cell, cells in a fixed order, so a lane's sum runs in a fixed order.
// One candidate in eight is a neighbour. A lane first lists its neighbours (slot and cell of
// the stencil, in its own column of shared memory) and runs f over the list afterwards, in
// the same order: with f inside the candidate loop nearly every turn of a warp ran it for
// the few lanes that had a neighbour. The cells' slot ranges are fetched once by the lanes
// together, and a cell's first five candidates per lane are in flight at once. A list that
// could overflow (14 neighbours per lane on average) is worked off before the next cell.
// A relaxation call of 32^3 particles: 237 us with f in the candidate loop (density 78,
// acceleration 152 us), 199 us with lists; 17^3 118 -> 91 us.
constexpr int kSphList = 32;
constexpr int kSphTurns = 5;  // candidates per lane in flight: a cell of a lattice holds about 33
struct SphLists {
  int slot[kSphList][kSphThreads];
  unsigned char cell[kSphList][kSphThreads];
};

// displacement of xi from xj, a particle of the cell at offset (ox, oy, oz), and its square
template <int DIM>
__device__ __forceinline__ float4 pair_displacement(const float4 xi, int ox, int oy, int oz, const float4 xj,
                                                    const SphGeom& g) {
  const float px = xi.x - (float)ox * g.cs, py = xi.y - (float)oy * g.cs, pz = xi.z - (float)oz * g.cs;
  const float dx = px - xj.x, dy = py - xj.y, dz = DIM == 3 ? pz - xj.z : 0.f;
  return make_float4(dx, dy, dz, dx * dx + dy * dy + dz * dz);
}

// One cell (nc == 1): every particle is a candidate, at the minimum image.
template <int DIM, class P, class F>
__device__ __forceinline__ void for_all_pairs(bool live, const float4 xi, const SphGeom& g,
                                              const int* __restrict__ start, const float4* __restrict__ xs, int lane,
                                              P&& fetch, F&& f) {
  const int e = live ? start[1] : 0;
  for (int jj = start[0] + lane; jj < e; jj += kSphLanes) {
    const float4 xj = xs[jj];
    float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = DIM == 3 ? xi.z - xj.z : 0.f;
    dx -= g.Lf * rintf(dx / g.Lf);
    dy -= g.Lf * rintf(dy / g.Lf);
    if (DIM == 3) dz -= g.Lf * rintf(dz / g.Lf);
    const float r2 = dx * dx + dy * dy + dz * dz;
    if (r2 < g.cut2) f(jj, dx, dy, dz, r2, fetch(jj));
  }
}

// stencil cell k (x offset varying fastest)
template <int DIM>
__device__ __forceinline__ void stencil_offset(int k, int& ox, int& oy, int& oz) {
  ox = k % 3 - 1;
  oy = k / 3 % 3 - 1;
  oz = DIM == 3 ? k / 9 - 1 : 0;
}

// (nc >= 3) fetch(j): what f wants of slot j beside its displacement. keep(i, j, code):
// called with f, the lane's i-th neighbour.
template <int DIM, class P, class F, class K>
__device__ __forceinline__ void for_neighbours(bool live, const float4 xi, const int3 ci, const SphGeom& g,
                                               const int* __restrict__ start, const float4* __restrict__ xs, int lane,
                                               SphLists& lists, P&& fetch, F&& f, K&& keep) {
  const int nc = g.nc, tid = threadIdx.x, base = (tid & 31) - lane;
  constexpr int cells = DIM == 3 ? 27 : 9;
  constexpr int S = DIM == 3 ? 4 : 2;  // cells whose range a lane fetches: lane, lane + 8, ...
  int rb[S], re[S];
  auto wrap = [nc](int c) { return c < 0 ? c + nc : (c >= nc ? c - nc : c); };
#pragma unroll
  for (int q = 0; q < S; ++q) {
    const int k = lane + q * kSphLanes;
    rb[q] = re[q] = 0;
    if (live && k < cells) {
      int ox, oy, oz;
      stencil_offset<DIM>(k, ox, oy, oz);
      const int cx = wrap(ci.x + ox), cy = wrap(ci.y + oy);
      const int c = DIM == 3 ? (cx * nc + cy) * nc + wrap(ci.z + oz) : cx * nc + cy;
      rb[q] = start[c];
      re[q] = start[c + 1];
    }
  }
  int cnt = 0, done = 0;
#pragma unroll 1
  for (int k = 0; k <= cells; ++k) {  // the turn after the last cell works the rest off
    int b = rb[0], e = re[0];
#pragma unroll
    for (int q = 1; q < S; ++q)
      if (k / kSphLanes == q) {
        b = rb[q];
        e = re[q];
      }
    b = __shfl_sync(0xffffffffu, b, base + k % kSphLanes);
    e = __shfl_sync(0xffffffffu, e, base + k % kSphLanes);
    if (k == cells) e = b;
    int ox, oy, oz;
    stencil_offset<DIM>(k, ox, oy, oz);
    const unsigned char code = (unsigned char)((ox + 1) | (oy + 1) << 2 | (oz + 1) << 4);
    do {
      if (k == cells || cnt > kSphList - kSphTurns) {
        int jc = cnt > 0 ? lists.slot[0][tid] : 0, oc = cnt > 0 ? lists.cell[0][tid] : 0;
        float4 xc = xs[jc];
        auto pc = fetch(jc);
#pragma unroll 1
        for (int i = 0; i < cnt; ++i) {  // the next neighbour's operands while this one's pair is formed
          const int jn = i + 1 < cnt ? lists.slot[i + 1][tid] : 0, on = i + 1 < cnt ? lists.cell[i + 1][tid] : 0;
          const float4 xn = i + 1 < cnt ? xs[jn] : make_float4(0.f, 0.f, 0.f, 0.f);
          const auto pn = fetch(jn);
          const float4 d = pair_displacement<DIM>(xi, (oc & 3) - 1, (oc >> 2 & 3) - 1, (oc >> 4) - 1, xc, g);
          f(jc, d.x, d.y, d.z, d.w, pc);
          keep(done + i, jc, oc);
          jc = jn;
          oc = on;
          xc = xn;
          pc = pn;
        }
        done += cnt;
        cnt = 0;
      }
      float4 xj[kSphTurns];
#pragma unroll
      for (int i = 0; i < kSphTurns; ++i) {
        const int jj = b + lane + i * kSphLanes;
        xj[i] = jj < e ? xs[jj] : make_float4(1e30f, 0.f, 0.f, 0.f);  // far from everything
      }
#pragma unroll
      for (int i = 0; i < kSphTurns; ++i) {
        const int jj = b + lane + i * kSphLanes;
        if (jj < e && pair_displacement<DIM>(xi, ox, oy, oz, xj[i], g).w < g.cut2) {
          lists.slot[cnt][tid] = jj;
          lists.cell[cnt][tid] = code;
          ++cnt;
        }
      }
      b += kSphTurns * kSphLanes;
    } while (b < e);
  }
  keep(done, -1, 0);
}

// Neighbours that the density pass leaves for the acceleration pass of the same call, so
// that the search (27 cells, eight candidates for one neighbour) runs once: entry k of
// lane q of slot i at nb[k stride + 8 i + q] (slot | stencil cell << kSphCodeShift; a warp
// reads 32 neighbouring words), counts at n. A lane with more than `cap` of them searches
// again. The order is the search's, so the sums are the same to the bit. A relaxation call of
// 32^3 particles 199 -> 175 us, 9^3 80 -> 49, 160^2 (2D) 92 -> 83.
struct SphKept {
  unsigned* nb;  // null: not kept
  int* n;
  long long stride;
  int cap;
};
constexpr int kSphCodeShift = 26;
constexpr int kSphKept3d = 32, kSphKept2d = 12;  // about 14 and 4 per lane on a lattice
constexpr size_t kSphKeptBytes = (size_t)1 << 30;  // plans above it (10^6 particles in 3D) search twice

// the pairs of one lane without lists, in the order of for_neighbours
template <int DIM, class P, class F>
__device__ __forceinline__ void for_neighbours_direct(const float4 xi, const int3 ci, const SphGeom& g,
                                                   const int* __restrict__ start, const float4* __restrict__ xs,
                                                   int lane, P&& fetch, F&& f) {
  const int nc = g.nc;
  auto wrap = [nc](int c) { return c < 0 ? c + nc : (c >= nc ? c - nc : c); };
  constexpr int cells = DIM == 3 ? 27 : 9;
  for (int k = 0; k < cells; ++k) {
    int ox, oy, oz;
    stencil_offset<DIM>(k, ox, oy, oz);
    const int cx = wrap(ci.x + ox), cy = wrap(ci.y + oy);
    const int c = DIM == 3 ? (cx * nc + cy) * nc + wrap(ci.z + oz) : cx * nc + cy;
    for (int j = start[c] + lane; j < start[c + 1]; j += kSphLanes) {
      const float4 d = pair_displacement<DIM>(xi, ox, oy, oz, xs[j], g);
      if (d.w < g.cut2) f(j, d.x, d.y, d.z, d.w, fetch(j));
    }
  }
}

// the pairs of one lane from its kept list
template <int DIM, class P, class F>
__device__ __forceinline__ void for_kept(const float4 xi, const SphGeom& g, const float4* __restrict__ xs,
                                         const unsigned* __restrict__ nb, long long stride, int n, P&& fetch, F&& f) {
  constexpr int U = 2;  // pairs whose operands are in flight beside the two being formed
  unsigned cc[U];
  float4 xc[U];
  decltype(fetch(0)) pc[U];
  auto load = [&](int i, int q) {
    cc[q] = i < n ? nb[i * stride] : 0u;
    const int j = (int)(cc[q] & ((1u << kSphCodeShift) - 1));
    xc[q] = xs[j];
    pc[q] = fetch(j);
  };
#pragma unroll
  for (int q = 0; q < U; ++q) load(q, q);
#pragma unroll 1
  for (int i = 0; i < n; i += U) {
    unsigned c0[U];
    float4 x0[U];
    decltype(fetch(0)) p0[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      c0[q] = cc[q];
      x0[q] = xc[q];
      p0[q] = pc[q];
      load(i + U + q, q);
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const int o = (int)(c0[q] >> kSphCodeShift);
      const float4 d = pair_displacement<DIM>(xi, (o & 3) - 1, (o >> 2 & 3) - 1, (o >> 4) - 1, x0[q], g);
      if (i + q < n) f((int)(c0[q] & ((1u << kSphCodeShift) - 1)), d.x, d.y, d.z, d.w, p0[q]);
    }
  }
}

// cell coordinates of the particle at slot i
template <int DIM>
__device__ __forceinline__ int3 slot_cell(long long i, const int* __restrict__ perm, const int* __restrict__ cell,
                                          int nc) {
  const int c = cell[perm[i]], q = c / nc;
  return DIM == 3 ? make_int3(q / nc, q % nc, c % nc) : make_int3(q, c % nc, 0);
}

// The lanes' float-float sums of F values per particle, in FP64: (particle of the block,
// value) at sums[particle F + value]. The tree is that of a butterfly over the lanes. FP64 is
// scarce on this GPU, so the sums meet in shared memory and whole warps add them: lanes 0-3
// and 4-7 of a value by a thread each, instead of every lane adding every value; the
// acceleration pass' wraps and divisions follow with a thread per particle and component (a
// lane per particle made each warp run them three times for four live lanes). With the cells
// read instead of formed again from FP64 positions, and the wraps' quotients made only where
// they are not zero: a relaxation call of 32^3 particles 175 -> 118 us, 160^2 (2D) 83 -> 47.
constexpr int kSphGroup = kSphThreads / kSphLanes;  // particles per block
template <int F>
struct SphSums {
  float2 lane[F][kSphThreads];
  double half[2][kSphGroup * F];
};
template <int F>
__device__ __forceinline__ void block_sums(const Ff (&part)[F], SphSums<F>& m) {
#pragma unroll
  for (int f = 0; f < F; ++f) m.lane[f][threadIdx.x] = make_float2(part[f].hi, part[f].lo);
  __syncthreads();
  for (int task = threadIdx.x; task < 2 * kSphGroup * F; task += kSphThreads) {
    const int h = task / (kSphGroup * F), v = task % (kSphGroup * F);
    const float2* l = &m.lane[v % F][v / F * kSphLanes + 4 * h];
    auto d = [&](int q) { return (double)l[q].x + (double)l[q].y; };
    m.half[h][v] = (d(0) + d(1)) + (d(2) + d(3));
  }
  __syncthreads();
}

// rho[slot] = m sigma sum_j w(r_ij / h); rp[slot] = (rho, p = p_ref (rho - 1),
// 1 / rho^2) in FP32 for the acceleration pass (the quotient once per particle: it was one
// of three divisions per pair there); rho_out[input index] when requested
template <int DIM, bool ONE>
__global__ void __launch_bounds__(kSphThreads)
k_sph_density(const float4* __restrict__ xs, const int* __restrict__ start, const int* __restrict__ perm,
              const int* __restrict__ cell, long long np, SphGeom g, double m_sigma, double p_ref,
              float4* __restrict__ rp, double* __restrict__ rho_out, SphKept kept) {
  pdl_begin();
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = (int)(gt % kSphLanes);
  const bool live = gt / kSphLanes < np;  // every lane stays for the shuffles
  Ff part[1] = {};
  const long long is = live ? gt / kSphLanes : 0;
  const float4 xi = xs[is];
  const float inv_h = g.inv_h;
  auto none = [](int) { return 0; };
  auto pair = [&](int, float, float, float, float r2, int) {
    part[0] = ff_add(part[0], quintic_w(sqrtf(r2) * inv_h));
  };
  if constexpr (ONE) {
    for_all_pairs<DIM>(live, xi, g, start, xs, lane, none, pair);
  } else {
    __shared__ SphLists lists;
    for_neighbours<DIM>(live, xi, slot_cell<DIM>(is, perm, cell, g.nc), g, start, xs, lane, lists, none, pair,
                        [&](int k, int j, int code) {
                          if (!kept.nb) return;
                          if (j < 0)
                            kept.n[gt] = k;
                          else if (k < kept.cap)
                            kept.nb[k * kept.stride + gt] = (unsigned)j | (unsigned)code << kSphCodeShift;
                        });
  }
  __shared__ SphSums<1> m;
  block_sums<1>(part, m);
  const long long i = (long long)blockIdx.x * kSphGroup + threadIdx.x;
  if (threadIdx.x >= kSphGroup || i >= np) return;
  const double acc = m.half[0][threadIdx.x] + m.half[1][threadIdx.x];
  const double rho = m_sigma * acc;
  const float rf = (float)rho;
  rp[i] = make_float4(rf, (float)(p_ref * (rho - 1.0)), 1.f / (rf * rf), 0.f);
  if (rho_out) rho_out[perm[i]] = rho;
}

enum SphMode { kSphRelaxAcc = 0, kSphRelaxVel = 1, kSphForces = 2 };

struct SphAccelArgs {
  const float4* xs;
  const int* start;
  const int* perm;
  const int* cell;      // per particle, input order
  const double* xw;     // wrapped (predicted) positions, input order
  const float4* rp;     // (rho, p, 1 / rho^2, -) per slot
  const float4* us;     // velocities per slot (forces only)
  long long np;
  float mass, grad_scale, p_ref, eps;  // grad_scale = sigma / h
  // relaxation velocity (combined.py:132-142)
  const double* r0;
  double kick;  // (relax_dt_factor * dt)^2
  double dt;
  double* out0;  // acc | u_out | acc_p
  double* out1;  // r_out (may be null) | acc_visc
  double* out2;  // acc_tvf
};

// Per pair (Adami 2012 eqs. 8, 10, 13 with constant mass, as relax.py:88-105/139-159):
//   pref = m (1/rho_i^2 + 1/rho_j^2), p_ij = (rho_j p_i + rho_i p_j) / (rho_i + rho_j)
//   grad = dW/dr * r_ij / (r + eps)
//   acc_p = -pref p_ij grad, acc_tvf = -pref p_ref grad, acc_visc = pref u_ij dW/dr / (r + eps)
// Relaxation acceleration = acc_p + acc_tvf / 2.
// HOW: the pairs come from a search, from the density pass's lists, or (one cell) are all.
constexpr int kPairsSearch = 0, kPairsKept = 1, kPairsAll = 2;
template <int DIM, int MODE, int HOW>
__global__ void __launch_bounds__(kSphThreads) k_sph_accel(SphAccelArgs a, SphGeom g, SphKept kept) {
  pdl_begin();
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = (int)(gt % kSphLanes);
  const bool live = gt / kSphLanes < a.np;  // every lane stays for the shuffles
  const long long is = live ? gt / kSphLanes : 0;
  const float4 xi = a.xs[is];
  const float4 rpi = a.rp[is];
  const float4 ui = MODE == kSphForces ? a.us[is] : make_float4(0.f, 0.f, 0.f, 0.f);
  constexpr int F = MODE == kSphForces ? 3 * DIM : DIM;  // values per particle
  Ff sum[F] = {};  // acc_p (relaxation: acc), forces: acc_visc, acc_tvf behind it
  auto fetch = [&](int jj) { return a.rp[jj]; };
  auto pair = [&](int jj, float dx, float dy, float dz, float r2, const float4 rpj) {
    const float r = sqrtf(r2);
    const float dw = a.grad_scale * quintic_dw(r * g.inv_h);
    const float pref = a.mass * (rpi.z + rpj.z);
    const float pij = (rpj.x * rpi.y + rpi.x * rpj.y) / (rpi.x + rpj.x);
    const float s = dw / (r + a.eps);
    if (MODE == kSphForces) {
      const float cp = -pref * pij * s, ct = -pref * a.p_ref * s;
      const float4 uj = a.us[jj];
      const float cv = pref * s;
      const float e[3] = {dx, dy, dz}, w[3] = {ui.x - uj.x, ui.y - uj.y, ui.z - uj.z};
#pragma unroll
      for (int d = 0; d < DIM; ++d) {
        sum[d] = ff_add(sum[d], cp * e[d]);
        sum[DIM + d] = ff_add(sum[DIM + d], cv * w[d]);
        sum[2 * DIM + d] = ff_add(sum[2 * DIM + d], ct * e[d]);
      }
    } else {
      const float cp = -pref * (pij + 0.5f * a.p_ref) * s;
      const float e[3] = {dx, dy, dz};
#pragma unroll
      for (int d = 0; d < DIM; ++d) sum[d] = ff_add(sum[d], cp * e[d]);
    }
  };
  if constexpr (HOW == kPairsAll) {
    for_all_pairs<DIM>(live, xi, g, a.start, a.xs, lane, fetch, pair);
  } else if constexpr (HOW == kPairsKept) {
    const int n = live ? kept.n[gt] : 0;
    if (n <= kept.cap)
      for_kept<DIM>(xi, g, a.xs, kept.nb + gt, kept.stride, n, fetch, pair);
    else
      for_neighbours_direct<DIM>(xi, slot_cell<DIM>(is, a.perm, a.cell, g.nc), g, a.start, a.xs, lane, fetch, pair);
  } else {
    __shared__ SphLists lists;
    for_neighbours<DIM>(live, xi, slot_cell<DIM>(is, a.perm, a.cell, g.nc), g, a.start, a.xs, lane, lists, fetch,
                        pair, [](int, int, int) {});
  }
  __shared__ SphSums<F> m;
  block_sums<F>(sum, m);
  // one thread per particle and value
  for (int v = threadIdx.x; v < kSphGroup * F; v += kSphThreads) {
    const long long i = (long long)blockIdx.x * kSphGroup + v / F;
    if (i >= a.np) continue;
    const int f = v % F, d = f % DIM;
    const long long j = a.perm[i];
    const double ap = m.half[0][v] + m.half[1][v];
    if (MODE == kSphRelaxAcc) {
      a.out0[j * DIM + d] = ap;
    } else if (MODE == kSphRelaxVel) {
      // r_temp <- shift(r_temp, kick * acc); u = displacement(r_temp, r0) / dt, with the
      // periodic displacement mod(d + L/2, L) - L/2; optionally r_out = shift(r0, dt u)
      const double x = wrap_period(a.xw[j * DIM + d] + a.kick * ap, g.L);
      const double dd = wrap_period(x - a.r0[j * DIM + d] + 0.5 * g.L, g.L);
      const double uv = (dd - 0.5 * g.L) / a.dt;
      a.out0[j * DIM + d] = uv;
      if (a.out1) a.out1[j * DIM + d] = wrap_period(a.r0[j * DIM + d] + a.dt * uv, g.L);
    } else {
      (f < DIM ? a.out0 : f < 2 * DIM ? a.out1 : a.out2)[j * DIM + d] = ap;
    }
  }
}

}  // namespace l3es

using namespace l3es;

struct l3es_sph_plan {
  int dim = 3, n = 0;
  long long np_max = 0;
  int ncell = 0;
  SphGeom g{};
  double dx = 0.0, mass = 0.0, sigma = 0.0;
  double* xw = nullptr;    // [np_max * dim] wrapped / predicted positions
  int* cell = nullptr;     // [np_max]
  int* count = nullptr;    // [ncell]
  int* start = nullptr;    // [ncell + 1]
  int* cursor = nullptr;   // [ncell]
  int* perm0 = nullptr;    // [np_max] unordered slots
  int* perm = nullptr;     // [np_max] slot -> input index
  float4* xs = nullptr;    // [np_max] cell-local coordinates per slot
  float4* us = nullptr;    // [np_max] velocity per slot (forces)
  float4* rp = nullptr;    // [np_max] (rho, p, 1 / rho^2, -) per slot
  SphKept kept{};          // neighbour lists of np_max particles (null: searched twice)
  void* mem = nullptr;     // the one allocation behind all of them
};

// cell list of r (+ dt u_pred when given); leaves xw, perm, xs (and us when u != null)
static int sph_build(l3es_sph_plan* p, const double* r, const double* u_pred, double dt, const double* u,
                     long long np, cudaStream_t s) {
  int rc = cuda_check(cudaMemsetAsync(p->count, 0, sizeof(int) * p->ncell, s), "l3es_sph memset");
  if (rc != L3ES_OK) return rc;
  const unsigned pb = (unsigned)((np + kSphThreads - 1) / kSphThreads);
  if (p->dim == 3) {
    pdl_launch(k_sph_bin<3>, pb, kSphThreads, 0, s, r, u_pred, dt, np, p->g, p->xw, p->cell, p->count);
  } else {
    pdl_launch(k_sph_bin<2>, pb, kSphThreads, 0, s, r, u_pred, dt, np, p->g, p->xw, p->cell, p->count);
  }
  pdl_launch(k_sph_scan, 1, 1024, 0, s, p->count, p->ncell, p->start, p->cursor);
  pdl_launch(k_sph_scatter, pb, kSphThreads, 0, s, p->cell, np, p->cursor, p->perm0);
  if (p->dim == 3)
    pdl_launch(k_sph_order<3>, pb, kSphThreads, 0, s, p->perm0, p->cell, p->start, p->xw, u, np, p->g, p->perm, p->xs,
                                               u ? p->us : nullptr);
  else
    pdl_launch(k_sph_order<2>, pb, kSphThreads, 0, s, p->perm0, p->cell, p->start, p->xw, u, np, p->g, p->perm, p->xs,
                                               u ? p->us : nullptr);
  return cuda_check(cudaGetLastError(), "l3es_sph cell list");
}

// keep: an acceleration pass over the same particles follows
static void sph_density(l3es_sph_plan* p, long long np, double p_ref, double* rho_out, bool keep, cudaStream_t s) {
  const unsigned pb = (unsigned)((np * kSphLanes + kSphThreads - 1) / kSphThreads);
  const bool one = p->g.nc < 3;
  auto kernel = p->dim == 3 ? (one ? k_sph_density<3, true> : k_sph_density<3, false>)
                            : (one ? k_sph_density<2, true> : k_sph_density<2, false>);
  pdl_launch(kernel, pb, kSphThreads, 0, s, p->xs, p->start, p->perm, p->cell, np, p->g, p->mass * p->sigma, p_ref,
             p->rp, rho_out, keep ? p->kept : SphKept{});
}

template <int DIM, int MODE>
static void sph_accel_dim(l3es_sph_plan* p, SphAccelArgs& a, cudaStream_t s) {
  const unsigned pb = (unsigned)((a.np * kSphLanes + kSphThreads - 1) / kSphThreads);
  auto kernel = p->g.nc < 3 ? k_sph_accel<DIM, MODE, kPairsAll>
                : p->kept.nb ? k_sph_accel<DIM, MODE, kPairsKept> : k_sph_accel<DIM, MODE, kPairsSearch>;
  pdl_launch(kernel, pb, kSphThreads, 0, s, a, p->g, p->kept);
}

template <int MODE>
static void sph_accel(l3es_sph_plan* p, SphAccelArgs& a, cudaStream_t s) {
  if (p->dim == 3)
    sph_accel_dim<3, MODE>(p, a, s);
  else
    sph_accel_dim<2, MODE>(p, a, s);
}

static SphAccelArgs sph_args(l3es_sph_plan* p, long long np, double u_ref) {
  SphAccelArgs a{};
  a.xs = p->xs;
  a.start = p->start;
  a.perm = p->perm;
  a.cell = p->cell;
  a.xw = p->xw;
  a.rp = p->rp;
  a.us = p->us;
  a.np = np;
  a.mass = (float)p->mass;
  a.grad_scale = (float)(p->sigma / p->dx);
  a.p_ref = (float)(100.0 * u_ref * u_ref);
  a.eps = 2.220446049250313e-16f;
  return a;
}

// plan and particle count; with np == 0 the arrays may be null (the call does nothing)
static int sph_check(l3es_sph_plan* p, const void* r, long long np, const char* who) {
  if (!p) return fail(L3ES_EINVAL, std::string(who) + ": null plan");
  if (np < 0 || np > p->np_max) return fail(L3ES_EINVAL, std::string(who) + ": np outside [0, np_max]");
  if (np > 0 && !r) return fail(L3ES_EINVAL, std::string(who) + ": null positions");
  return L3ES_OK;
}

extern "C" {

int l3es_sph_plan_create(int32_t dim, int32_t n, double box, int64_t np_max, l3es_sph_plan** out) {
  if (!out) return fail(L3ES_EINVAL, "l3es_sph_plan_create: null out");
  *out = nullptr;
  if (dim != 2 && dim != 3) return fail(L3ES_EINVAL, "l3es_sph_plan_create: dim must be 2 or 3");
  if (n < 1 || n > 1024) return fail(L3ES_EINVAL, "l3es_sph_plan_create: n must be in [1, 1024]");
  if (!(box > 0.0) || !std::isfinite(box)) return fail(L3ES_EINVAL, "l3es_sph_plan_create: box must be > 0");
  if (np_max < 1 || np_max > (1LL << 30)) return fail(L3ES_EINVAL, "l3es_sph_plan_create: np_max out of range");
  auto* p = new l3es_sph_plan();
  p->dim = dim;
  p->n = n;
  p->np_max = np_max;
  p->dx = box / n;
  p->mass = std::pow(p->dx, dim);
  // quintic normalisation (Morris 1997): 7 / (478 pi h^2) in 2D, 3 / (359 pi h^3) in 3D
  p->sigma = dim == 3 ? 3.0 / (359.0 * M_PI * p->dx * p->dx * p->dx) : 7.0 / (478.0 * M_PI * p->dx * p->dx);
  int nc = n / 3;  // cell side L / nc >= cutoff 3 dx
  if (nc < 3) nc = 1;
  p->g.L = box;
  p->g.nc = nc;
  p->g.inv_cs = nc / box;
  p->g.cs_d = box / nc;
  p->g.cs = (float)(box / nc);
  p->g.Lf = (float)box;
  p->g.inv_h = (float)(1.0 / p->dx);
  p->g.cut2 = (float)(9.0 * p->dx * p->dx);
  p->ncell = dim == 3 ? nc * nc * nc : nc * nc;
  // one allocation holds every array: a plan is made inside the first call of a relaxation
  // function, and with one per array that call took 235 us for 80^2 particles (now 171), 355 for
  // 32^3 (258)
  const size_t npm = (size_t)np_max;
  const size_t lanes = (npm * kSphLanes + kSphThreads - 1) / kSphThreads * kSphThreads;  // whole blocks
  const int cap = dim == 3 ? kSphKept3d : kSphKept2d;
  const size_t words = lanes * (cap + 1);
  // neighbour lists, where they and the slot numbers fit
  const bool keep = nc >= 3 && np_max <= (1LL << kSphCodeShift) && words * sizeof(unsigned) <= kSphKeptBytes;
  size_t bytes = 0;
  auto place = [&](auto*& ptr, size_t count) {
    using T = std::remove_reference_t<decltype(*ptr)>;
    if (p->mem) ptr = reinterpret_cast<T*>(static_cast<char*>(p->mem) + bytes);
    bytes += (count * sizeof(T) + 255) / 256 * 256;
  };
  auto arrays = [&] {
    bytes = 0;
    place(p->xw, npm * dim);
    place(p->cell, npm);
    place(p->perm0, npm);
    place(p->perm, npm);
    place(p->xs, npm);
    place(p->us, npm);
    place(p->rp, npm);
    place(p->count, p->ncell);
    place(p->cursor, p->ncell);
    place(p->start, p->ncell + 1);
  };
  arrays();
  const size_t own = bytes;
  cudaError_t e = keep ? cudaMalloc(&p->mem, own + words * sizeof(unsigned)) : cudaErrorMemoryAllocation;
  const bool kept = e == cudaSuccess;
  if (!kept) {  // without the lists the calls search twice
    cudaGetLastError();
    e = cudaMalloc(&p->mem, own);
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    delete p;
    return fail(L3ES_ENOMEM, std::string("cudaMalloc(particle arrays, ") + std::to_string(own) +
                                 " B): " + cudaGetErrorString(e));
  }
  arrays();
  if (kept) {
    unsigned* nb = reinterpret_cast<unsigned*>(static_cast<char*>(p->mem) + own);
    p->kept = SphKept{nb, reinterpret_cast<int*>(nb + lanes * cap), (long long)lanes, cap};
  }
  *out = p;
  return L3ES_OK;
}

int l3es_sph_plan_destroy(l3es_sph_plan* p) {
  if (!p) return L3ES_OK;
  cudaFree(p->mem);
  delete p;
  return L3ES_OK;
}

int l3es_sph_density(l3es_sph_plan* p, const double* r, int64_t np, double* rho, void* stream) {
  int rc = sph_check(p, r, np, "l3es_sph_density");
  if (rc != L3ES_OK) return rc;
  if (np == 0) return L3ES_OK;
  if (!rho) return fail(L3ES_EINVAL, "l3es_sph_density: null rho");
  cudaStream_t s = (cudaStream_t)stream;
  rc = sph_build(p, r, nullptr, 0.0, nullptr, np, s);
  if (rc != L3ES_OK) return rc;
  sph_density(p, np, 0.0, rho, false, s);
  return cuda_check(cudaGetLastError(), "l3es_sph_density launch");
}

int l3es_sph_relax_acceleration(l3es_sph_plan* p, const double* r, int64_t np, double u_ref, double* acc,
                                void* stream) {
  int rc = sph_check(p, r, np, "l3es_sph_relax_acceleration");
  if (rc != L3ES_OK) return rc;
  if (np == 0) return L3ES_OK;
  if (!acc) return fail(L3ES_EINVAL, "l3es_sph_relax_acceleration: null acc");
  cudaStream_t s = (cudaStream_t)stream;
  rc = sph_build(p, r, nullptr, 0.0, nullptr, np, s);
  if (rc != L3ES_OK) return rc;
  const double p_ref = 100.0 * u_ref * u_ref;
  sph_density(p, np, p_ref, nullptr, true, s);
  SphAccelArgs a = sph_args(p, np, u_ref);
  a.out0 = acc;
  sph_accel<kSphRelaxAcc>(p, a, s);
  return cuda_check(cudaGetLastError(), "l3es_sph_relax_acceleration launch");
}

int l3es_sph_forces(l3es_sph_plan* p, const double* r, const double* u, int64_t np, double u_ref, double* acc_p,
                    double* acc_visc, double* acc_tvf, void* stream) {
  int rc = sph_check(p, r, np, "l3es_sph_forces");
  if (rc != L3ES_OK) return rc;
  if (np == 0) return L3ES_OK;
  if (!u || !acc_p || !acc_visc || !acc_tvf) return fail(L3ES_EINVAL, "l3es_sph_forces: null argument");
  cudaStream_t s = (cudaStream_t)stream;
  rc = sph_build(p, r, nullptr, 0.0, u, np, s);
  if (rc != L3ES_OK) return rc;
  const double p_ref = 100.0 * u_ref * u_ref;
  sph_density(p, np, p_ref, nullptr, true, s);
  SphAccelArgs a = sph_args(p, np, u_ref);
  a.out0 = acc_p;
  a.out1 = acc_visc;
  a.out2 = acc_tvf;
  sph_accel<kSphForces>(p, a, s);
  return cuda_check(cudaGetLastError(), "l3es_sph_forces launch");
}

int l3es_sph_relax_velocity(l3es_sph_plan* p, const double* r0, const double* u_r, int64_t np, double dt,
                            double relax_dt_factor, double u_ref, double* u_out, double* r_out, void* stream) {
  int rc = sph_check(p, r0, np, "l3es_sph_relax_velocity");
  if (rc != L3ES_OK) return rc;
  if (!(dt != 0.0) || !std::isfinite(dt)) return fail(L3ES_EINVAL, "l3es_sph_relax_velocity: dt must be nonzero");
  if (np == 0) return L3ES_OK;
  if (!u_r || !u_out) return fail(L3ES_EINVAL, "l3es_sph_relax_velocity: null argument");
  if (u_out == u_r || u_out == r0 || (r_out && (r_out == r0 || r_out == u_r || r_out == u_out)))
    return fail(L3ES_EINVAL, "l3es_sph_relax_velocity: outputs must not alias the inputs");
  cudaStream_t s = (cudaStream_t)stream;
  rc = sph_build(p, r0, u_r, dt, nullptr, np, s);
  if (rc != L3ES_OK) return rc;
  const double p_ref = 100.0 * u_ref * u_ref;
  sph_density(p, np, p_ref, nullptr, true, s);
  SphAccelArgs a = sph_args(p, np, u_ref);
  a.r0 = r0;
  a.kick = (relax_dt_factor * dt) * (relax_dt_factor * dt);
  a.dt = dt;
  a.out0 = u_out;
  a.out1 = r_out;
  sph_accel<kSphRelaxVel>(p, a, s);
  return cuda_check(cudaGetLastError(), "l3es_sph_relax_velocity launch");
}

}  // extern "C"
