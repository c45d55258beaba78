// Coarsening and exact spectral interpolation kernels shared by the particle
// entry points (templates, so every translation unit may instantiate them).
#pragma once

#include <cuda_runtime.h>

#include "fft_core.cuh"
#include "pdl.cuh"

namespace l3es {

// ------------------------------------------------------------------------------
// Coarse spectrum of spectral_filtering: Hh(f) = 0.5 (C(f) + conj C(p)), with
// C(f) = U_fine(f) / (N/c)^dim on the crop set f in [-c/2, c/2-1]^dim and p the
// crop-set representative of -f mod c. The half-average is fftn(real(ifftn(crop)))
// (utils.py:126-127): it only changes modes with a component at -c/2.
// Output: rfftn layout of the coarse grid, half axis index iz in [0, c/2].
// ------------------------------------------------------------------------------
__device__ __forceinline__ int crop_freq(int i, int c) { return i < c / 2 ? i : i - c; }  // [-c/2, c/2)
__device__ __forceinline__ int crop_wrap(int f, int c) {  // -> [-c/2, c/2)
  f %= c;
  if (f < -c / 2) f += c;
  if (f >= c / 2) f -= c;
  return f;
}

template <int DIM>
__device__ __forceinline__ float2 fine_full(const float2* __restrict__ uh, int N, int fx, int fy, int fz) {
  // full-spectrum value of the rfftn half spectrum at signed frequencies (3D: fx, fy,
  // fz with fz on the half axis; 2D: fx, fy with fy on the half axis)
  const int H = N / 2 + 1;
  if (DIM == 3) {
    if (fz >= 0) return __ldg(uh + ((long long)((fx + N) % N) * N + (fy + N) % N) * H + fz);
    const float2 v = __ldg(uh + ((long long)((-fx + N) % N) * N + (-fy + N) % N) * H + (-fz));
    return make_float2(v.x, -v.y);
  } else {
    if (fy >= 0) return __ldg(uh + (long long)((fx + N) % N) * H + fy);
    const float2 v = __ldg(uh + (long long)((-fx + N) % N) * H + (-fy));
    return make_float2(v.x, -v.y);
  }
}

template <int DIM>
__global__ void __launch_bounds__(256)
k_crop(const float2* __restrict__ uh, long long cs, int N, float2* __restrict__ hh, long long hcs, int c,
       float scale) {
  pdl_begin();
  const int hc = c / 2 + 1;
  const long long per = DIM == 3 ? (long long)c * c * hc : (long long)c * hc;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int comp = blockIdx.y;
  if (i >= per) return;
  int ix, iy, iz;
  if (DIM == 3) {
    iz = (int)(i % hc);
    iy = (int)((i / hc) % c);
    ix = (int)(i / ((long long)hc * c));
  } else {
    iz = 0;
    iy = (int)(i % hc);
    ix = (int)(i / hc);
  }
  const float2* u = uh + comp * cs;
  float2 a, b;
  if (DIM == 3) {
    const int fx = crop_freq(ix, c), fy = crop_freq(iy, c), fz = iz < c / 2 ? iz : -c / 2;
    a = fine_full<3>(u, N, fx, fy, fz);
    b = fine_full<3>(u, N, crop_wrap(-fx, c), crop_wrap(-fy, c), crop_wrap(-fz, c));
  } else {
    const int fx = crop_freq(ix, c), fy = iy < c / 2 ? iy : -c / 2;
    a = fine_full<2>(u, N, fx, fy, 0);
    b = fine_full<2>(u, N, crop_wrap(-fx, c), crop_wrap(-fy, c), 0);
  }
  hh[comp * hcs + i] = make_float2(0.5f * scale * (a.x + b.x), 0.5f * scale * (a.y - b.y));
}

// ------------------------------------------------------------------------------
// Exact spectral interpolation (interp_backend="dft", integrator.py:62-91):
// u_r[j] = Re sum_{k in [-c/2, c/2-1]^dim} Hhat(k) exp(i k.x_j) / c^dim.
// Separable: per (kx[, ky]) an inner FP32 sum over the last axis, in 3D an FP32 sum of
// those over ky, an FP64 sum over kx; phase tables in shared memory (exp(i k x) per
// particle and axis by an FP64 recurrence, stored FP32).
//
// A block takes 32 particles. Each half warp owns a slice of the kx range and holds two
// particles per lane, so one mode (a broadcast 16-byte read of its staged copy
// (x, x, y, y)) feeds 4 paired FP32 FMAs per lane, and RB rows times DIM components share
// a particle's phase read; the half warps' FP64 partial sums are added in kx order. The
// FP32 sums run in the order of the plain loops, whatever the split, so a particle's
// velocity does not depend on it beyond FP64 rounding. Bound by FP32 FMAs (4 per mode,
// component and particle). With one thread per particle, one component after the other
// and the mode index arithmetic in the inner loop, 10007 particles on 32^3 modes took
// 14.2 ms (79 blocks of 4 warps); now 0.31 ms, a third of the FP32 FMA rate, 32768
// particles 0.67 ms, half of it.
// ------------------------------------------------------------------------------
constexpr int kDftTile = 32;                                 // particles per block
inline int dft_threads(int c) { return c >= 16 ? 256 : c > 2 ? 16 * c : 32; }
inline int dft_rows(int c) { return c <= 32 ? 2 : 1; }       // RB: staged rows per half warp
// shared memory of k_dft_interp: phase tables, then the warps' staged rows (which the
// FP64 partial sums reuse: 16 bytes a mode and two halves of RB c DIM modes per warp
// hold 2 x 32 x DIM doubles as long as RB c >= 32)
inline size_t dft_smem(int dim, int c) {
  const size_t table = sizeof(float2) * dim * c * kDftTile;
  const size_t rows = (size_t)(dft_threads(c) / 32) * 2 * dft_rows(c) * c * dim * sizeof(float4);
  const size_t sums = (size_t)(dft_threads(c) / 16) * kDftTile * dim * sizeof(double);
  return table + (rows > sums ? rows : sums);
}

// (a.x, a.y) <- (a.x + s.x b.x, a.y + s.y b.y) in one paired FP32 FMA
__device__ __forceinline__ float2 fma2(float2 s, float2 b, float2 a) { return __ffma2_rn(s, b, a); }

// Two blocks per SM up to c = 32 (128 registers: 306 against 334 us at 160 registers and
// one block, 10007 particles on 32^3 modes); at c = 64 shared memory holds one block.
template <int DIM, int RB>
__global__ void __launch_bounds__(256, RB == 2 ? 2 : 1)
k_dft_interp(const float2* __restrict__ hh, long long hcs, int c, const double* __restrict__ r, long long np,
             double* __restrict__ u_r, double dt, double* __restrict__ r_out) {
  pdl_begin();
  extern __shared__ __align__(16) unsigned char s_dft[];
  float2* ph = reinterpret_cast<float2*>(s_dft);  // [DIM][c][kDftTile]
  float4* rows = reinterpret_cast<float4*>(s_dft + sizeof(float2) * DIM * c * kDftTile);
  double* sums = reinterpret_cast<double*>(rows);  // [half warp][kDftTile][DIM], after the transform
  const int tid = threadIdx.x, lane = tid & 31, hl = lane & 15, half = lane >> 4;
  const int hw = tid >> 4, nhw = blockDim.x >> 4;
  const int msk = c - 1, hc = c / 2 + 1, lc = 31 - __clz(c);  // c is a power of two
  const int stage = RB * c * DIM;                    // modes staged per half warp: [row][kz][comp]
  float4* my = rows + (long long)(tid >> 5) * 2 * stage + half * stage;
  float4* warp_rows = rows + (long long)(tid >> 5) * 2 * stage;
  const int per = (c + nhw - 1) / nhw;               // kx slice of a half warp
  const long long tiles = (np + kDftTile - 1) / kDftTile;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const long long j0 = tile * kDftTile;
    for (int i = tid; i < kDftTile * DIM; i += blockDim.x) {
      // exp(i k x) for k = -c/2 .. c/2-1: two FP64 sincos, then p_{k+1} = p_k exp(i x)
      // in FP64 (the recurrence adds ~c ulp; FP64 transcendentals are slow on this GPU)
      const int q = i % kDftTile, d = i / kDftTile;
      const long long j = j0 + q < np ? j0 + q : np - 1;
      const double x = r[j * DIM + d];
      double sn, co, pi, pr;
      sincos(x, &sn, &co);
      sincos(-(double)(c / 2) * x, &pi, &pr);
      for (int k = 0; k < c; ++k) {
        ph[(d * c + k) * kDftTile + q] = make_float2((float)pr, (float)pi);
        const double tr = pr * co - pi * sn;
        pi = fma(pr, sn, pi * co);
        pr = tr;
      }
    }
    __syncthreads();
    const float2* pz = ph + (DIM - 1) * c * kDftTile + hl;  // this lane's particles: hl, hl + 16
    const float2* py = ph + c * kDftTile + hl;              // (3D)
    double tot[2][DIM];
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int d = 0; d < DIM; ++d) tot[q][d] = 0.0;
    // 3D: rows are ky at one kx; 2D: rows are kx
    const int blocks = DIM == 3 ? per * (c / RB) : (per + RB - 1) / RB;
    float2 sx[2][DIM];
    const int yb = DIM == 3 ? c / RB : 1;                   // 3D: row blocks per kx
    // Row block b of both half warps: modes (kx, ky, kz), kz = -c/2 .. c/2-1 (Hermitian
    // below 0), one (row, kz) per lane and turn. It is loaded into registers while the
    // block before it is summed (up to 64 modes per half warp, else at once).
    constexpr int TURNS = 2;  // RB c <= 64
    float2 nx[TURNS][2][DIM];
    auto fetch = [&](int b) {
      const int xo = DIM == 3 ? b / yb : b * RB, yo = DIM == 3 ? (b - b / yb * yb) * RB : 0;
#pragma unroll
      for (int n = 0; n < TURNS; ++n) {
        const int i = lane + 32 * n;
        const int row = i >> lc, kz = (i & msk) - c / 2, sg = kz >= 0 ? 1 : -1;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int xb = ((tid >> 5) * 2 + h) * per + xo + (DIM == 3 ? 0 : row);
          const int kx = xb - c / 2, ky = DIM == 3 ? yo + row - c / 2 : 0;
          const bool in = i < RB * c && xb < c;
          const long long o = DIM == 3 ? ((long long)((sg * kx) & msk) * c + ((sg * ky) & msk)) * hc + sg * kz
                                       : (long long)((sg * kx) & msk) * hc + sg * kz;
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            nx[n][h][d] = in ? __ldg(hh + d * hcs + o) : make_float2(0.f, 0.f);
            if (kz < 0) nx[n][h][d].y = -nx[n][h][d].y;
          }
        }
      }
    };
    fetch(0);
    for (int b = 0; b < blocks; ++b) {
      const int kxi = hw * per + (DIM == 3 ? b / yb : b * RB);  // table index of the (first) kx
      const int y0 = DIM == 3 ? (b - b / yb * yb) * RB : 0;
      __syncwarp();
#pragma unroll
      for (int n = 0; n < TURNS; ++n) {
        const int i = lane + 32 * n;
        if (i < RB * c) {
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
              const float2 v = nx[n][h][d];
              warp_rows[h * stage + i * DIM + d] = make_float4(v.x, v.x, v.y, v.y);
            }
        }
      }
      __syncwarp();
      if (b + 1 < blocks) fetch(b + 1);
      if (DIM == 3 && y0 == 0) {
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int d = 0; d < DIM; ++d) sx[q][d] = make_float2(0.f, 0.f);
      }
      float2 sy[RB][2][DIM];
#pragma unroll
      for (int w = 0; w < RB; ++w)
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int d = 0; d < DIM; ++d) sy[w][q][d] = make_float2(0.f, 0.f);
#pragma unroll 4
      for (int kz = 0; kz < c; ++kz) {
        const float2 e0 = pz[kz * kDftTile], e1 = pz[kz * kDftTile + 16];
        const float2 i0 = make_float2(-e0.y, e0.x), i1 = make_float2(-e1.y, e1.x);
#pragma unroll
        for (int w = 0; w < RB; ++w)
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            const float4 v = my[(w * c + kz) * DIM + d];
            const float2 vx = make_float2(v.x, v.y), vy = make_float2(v.z, v.w);
            sy[w][0][d] = fma2(vy, i0, fma2(vx, e0, sy[w][0][d]));
            sy[w][1][d] = fma2(vy, i1, fma2(vx, e1, sy[w][1][d]));
          }
      }
#pragma unroll
      for (int w = 0; w < RB; ++w) {
        const int xi = DIM == 3 ? kxi : kxi + w;
        if (DIM == 2 && (xi >= (hw + 1) * per || xi >= c)) continue;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (DIM == 3) {
            const float2 ey = py[(y0 + w) * kDftTile + 16 * q];
#pragma unroll
            for (int d = 0; d < DIM; ++d) {
              const float2 t = sy[w][q][d];
              sx[q][d] = make_float2(fmaf(-t.y, ey.y, fmaf(t.x, ey.x, sx[q][d].x)),
                                     fmaf(t.y, ey.x, fmaf(t.x, ey.y, sx[q][d].y)));
            }
          } else {
            const float2 ex = ph[xi * kDftTile + hl + 16 * q];
#pragma unroll
            for (int d = 0; d < DIM; ++d)
              tot[q][d] += (double)sy[w][q][d].x * ex.x - (double)sy[w][q][d].y * ex.y;
          }
        }
      }
      if (DIM == 3 && y0 + RB == c && kxi < c) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const float2 ex = ph[kxi * kDftTile + hl + 16 * q];
#pragma unroll
          for (int d = 0; d < DIM; ++d) tot[q][d] += (double)sx[q][d].x * ex.x - (double)sx[q][d].y * ex.y;
        }
      }
    }
    __syncthreads();  // the staged rows are read
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int d = 0; d < DIM; ++d) sums[(hw * kDftTile + hl + 16 * q) * DIM + d] = tot[q][d];
    __syncthreads();
    for (int i = tid; i < kDftTile * DIM; i += blockDim.x) {
      const long long j = j0 + i / DIM;
      if (j >= np) continue;
      double t = 0.0;
      for (int h = 0; h < nhw; ++h) t += sums[h * kDftTile * DIM + i];
      const double ur = t / (DIM == 3 ? (double)c * c * c : (double)c * c);
      u_r[j * DIM + i % DIM] = ur;
      if (r_out) {
        const double two_pi = 2.0 * 3.14159265358979323846;
        double x = r[j * DIM + i % DIM] + dt * ur;
        x = x - two_pi * floor(x / two_pi);
        if (x >= two_pi) x -= two_pi;
        r_out[j * DIM + i % DIM] = x;
      }
    }
    __syncthreads();  // before the next tile's tables
  }
}

// Launches k_dft_interp<dim> over np particles. Grids that a one-thread-per-particle block
// of 128 could not serve (phase tables above 227 KB: c = 128, or c = 64 with more axes than
// fit) are refused by the caller's check of dft_supported.
inline bool dft_supported(int dim, int c) { return sizeof(float2) * dim * c * 128 <= 227 * 1024; }

inline cudaError_t dft_launch(int dim, const float2* hh, long long hcs, int c, const double* r, long long np,
                              double* u_r, double dt, double* r_out, cudaStream_t s) {
  const long long tiles = (np + kDftTile - 1) / kDftTile;
  const unsigned grid = (unsigned)(tiles < (1LL << 30) ? tiles : (1LL << 30));
  const size_t smem = dft_smem(dim, c);
  auto go = [&](auto kernel) {
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    pdl_launch(kernel, grid, dft_threads(c), smem, s, hh, hcs, c, r, np, u_r, dt, r_out);
    return cudaGetLastError();
  };
  if (dim == 3) return dft_rows(c) == 2 ? go(k_dft_interp<3, 2>) : go(k_dft_interp<3, 1>);
  return dft_rows(c) == 2 ? go(k_dft_interp<2, 2>) : go(k_dft_interp<2, 1>);
}

}  // namespace l3es
