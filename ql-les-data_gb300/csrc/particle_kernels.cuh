// Coarsening and exact spectral interpolation kernels shared by the particle
// entry points (templates, so every translation unit may instantiate them).
#pragma once

#include <cuda_runtime.h>

#include "fft_core.cuh"
#include "pdl.cuh"

namespace l3es {

// x in [0, L) by whole periods (the periodic shift of integrator.py:21-23; Python's % never
// returns the modulus itself). For x in [+0, L) the quotient's floor is 0 (x / L never rounds
// up to 1) and x stays as it is; that is told from the bits, since an FP64 division is some
// twenty instructions on a pipe of two a clock and SM.
__device__ __forceinline__ double wrap_period(double x, double L) {
  const unsigned long long xb = (unsigned long long)__double_as_longlong(x);
  const unsigned long long lb = (unsigned long long)__double_as_longlong(L);
  if (lb < 0x7ff0000000000000ull && xb < lb) return x;  // (L positive and finite)
  x = x - L * floor(x / L);
  return x >= L ? x - L : x;
}

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
// A block takes 8 P particles. Each part of a warp (8 lanes) owns a slice of the kx range
// and holds P particles per lane. Two rows are staged side by side as (x0, x1, y0, y1), so
// one broadcast 16-byte read feeds 4 P paired FP32 FMAs per lane; the read returns 512 bytes
// to a warp, 4 cycles of the SM's shared memory, which is why a lane holds several particles
// and the modes are not stored doubled. The parts' FP64 partial sums are added in kx order.
// The FP32 sums run in the order of the plain loops, whatever the split, so a particle's
// velocity does not depend on it beyond FP64 rounding. Bound by FP32 FMAs (4 per mode,
// component and particle). With one thread per particle, one component after the other and
// the mode index arithmetic in the inner loop, 10007 particles on 32^3 modes took 14.2 ms
// (79 blocks of 4 warps); with 2 particles per lane, parts of 16 lanes and each mode stored
// as (x, x, y, y), 306 us; now 244 (32768 particles: 529 us, 77 % of the FMA rate).
// ------------------------------------------------------------------------------
template <int DIM, int P>
struct DftCfg {
  static constexpr int LN = 8;          // lanes per part
  static constexpr int TILE = P * LN;   // particles per block
  // 3D: a kx per part up to c = 32, four at c = 64 (two blocks per SM); 2D: row pairs of kx
  static int threads(int c) {
    const int t = DIM == 3 ? (c <= 32 ? c * LN : 128) : (c / 2) * LN;
    return t >= 256 ? 256 : t > 32 ? t : 32;
  }
  // row pairs staged per part, [kz][component], and one to spread the parts over the banks
  static __host__ __device__ int stage(int c) { return c * DIM + 1; }
  // shared memory: phase tables, FP64 partial sums, staged rows
  static size_t smem(int c) {
    const size_t parts = threads(c) / LN;
    return sizeof(float2) * DIM * c * TILE + parts * (TILE * DIM * sizeof(double) + stage(c) * sizeof(float4));
  }
};

// (a.x, a.y) <- (a.x + s.x b.x, a.y + s.y b.y) in one paired FP32 FMA
__device__ __forceinline__ float2 fma2(float2 s, float2 b, float2 a) { return __ffma2_rn(s, b, a); }

template <int DIM, int P>
__global__ void __launch_bounds__(256, 2)
k_dft_interp(const float2* __restrict__ hh, long long hcs, int c, const double* __restrict__ r, long long np,
             double* __restrict__ u_r, double dt, double* __restrict__ r_out) {
  pdl_begin();
  using K = DftCfg<DIM, P>;
  constexpr int LN = K::LN, kDftTile = K::TILE, PARTS = 32 / LN;  // parts of a warp
  extern __shared__ __align__(16) unsigned char s_dft[];
  const int tid = threadIdx.x, lane = tid & 31, hl = lane % LN;
  const int hw = tid / LN, nhw = blockDim.x / LN;
  const int msk = c - 1, hc = c / 2 + 1, lc = 31 - __clz(c);  // c is a power of two
  const int stage = K::stage(c);
  float2* ph = reinterpret_cast<float2*>(s_dft);              // [DIM][c][kDftTile]
  double* sums = reinterpret_cast<double*>(ph + DIM * c * kDftTile);  // [part][DIM][kDftTile]
  float4* rows = reinterpret_cast<float4*>(sums + nhw * DIM * kDftTile);
  const float4* my = rows + hw * stage;
  double* mine = sums + hw * DIM * kDftTile + hl;  // this lane's particles: hl + LN q
  const int per = (c + nhw - 1) / nhw;               // kx slice of a part
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
    const float2* pz = ph + (DIM - 1) * c * kDftTile + hl;
    const float2* py = ph + c * kDftTile + hl;              // (3D)
#pragma unroll
    for (int i = 0; i < P * DIM; ++i) mine[LN * i] = 0.0;
    // row pairs: 3D two ky of one kx; 2D two kx
    const int yb = DIM == 3 ? c / 2 : 1;                    // 3D: row pairs per kx
    const int blocks = DIM == 3 ? per * yb : (per + 1) / 2;
    float2 sx[P][DIM];
    for (int b = 0; b < blocks; ++b) {
      const int xo = DIM == 3 ? b / yb : 2 * b, y0 = DIM == 3 ? (b - xo * yb) * 2 : 0;
      const int kxi = hw * per + xo;  // table index of the (first) kx
      // Stage the pair's modes (kx, ky, kz), kz = -c/2 .. c/2-1 (Hermitian below 0), one
      // (row, kz) per lane and turn; the other warps cover the loads.
      __syncwarp();
      for (int i = lane; i < 2 * c; i += 32) {
        const int row = i >> lc, kz = (i & msk) - c / 2, sg = kz >= 0 ? 1 : -1;
        float2 v[PARTS][DIM];
#pragma unroll
        for (int h = 0; h < PARTS; ++h) {
          const int xb = ((tid >> 5) * PARTS + h) * per + xo + (DIM == 3 ? 0 : row);
          const int kx = xb - c / 2, ky = DIM == 3 ? y0 + row - c / 2 : 0;
          const long long o = DIM == 3 ? ((long long)((sg * kx) & msk) * c + ((sg * ky) & msk)) * hc + sg * kz
                                       : (long long)((sg * kx) & msk) * hc + sg * kz;
#pragma unroll
          for (int d = 0; d < DIM; ++d) v[h][d] = xb < c ? __ldg(hh + d * hcs + o) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int h = 0; h < PARTS; ++h)
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            float* w = reinterpret_cast<float*>(rows + ((tid >> 5) * PARTS + h) * stage + (i & msk) * DIM + d);
            w[row] = v[h][d].x;
            w[2 + row] = kz < 0 ? -v[h][d].y : v[h][d].y;
          }
      }
      __syncwarp();
      if (DIM == 3 && y0 == 0) {
#pragma unroll
        for (int q = 0; q < P; ++q)
#pragma unroll
          for (int d = 0; d < DIM; ++d) sx[q][d] = make_float2(0.f, 0.f);
      }
      float2 re[P][DIM], im[P][DIM];  // (row 0, row 1)
#pragma unroll
      for (int q = 0; q < P; ++q)
#pragma unroll
        for (int d = 0; d < DIM; ++d) re[q][d] = im[q][d] = make_float2(0.f, 0.f);
#pragma unroll 2
      for (int kz = 0; kz < c; ++kz) {
        float4 v[DIM];
#pragma unroll
        for (int d = 0; d < DIM; ++d) v[d] = my[kz * DIM + d];
#pragma unroll
        for (int q = 0; q < P; ++q) {
          const float2 e = pz[kz * kDftTile + LN * q];
          const float2 ex = make_float2(e.x, e.x), ey = make_float2(e.y, e.y), en = make_float2(-e.y, -e.y);
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            const float2 x = make_float2(v[d].x, v[d].y), y = make_float2(v[d].z, v[d].w);
            re[q][d] = fma2(y, en, fma2(x, ex, re[q][d]));
            im[q][d] = fma2(y, ex, fma2(x, ey, im[q][d]));
          }
        }
      }
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        const int xi = kxi + w;
        if (DIM == 2 && (xi >= (hw + 1) * per || xi >= c)) continue;
#pragma unroll
        for (int q = 0; q < P; ++q) {
          const float2 e = DIM == 3 ? py[(y0 + w) * kDftTile + LN * q] : ph[xi * kDftTile + hl + LN * q];
#pragma unroll
          for (int d = 0; d < DIM; ++d) {
            const float tx = w ? re[q][d].y : re[q][d].x, ty = w ? im[q][d].y : im[q][d].x;
            if (DIM == 3)
              sx[q][d] = make_float2(fmaf(-ty, e.y, fmaf(tx, e.x, sx[q][d].x)),
                                     fmaf(ty, e.x, fmaf(tx, e.y, sx[q][d].y)));
            else
              mine[d * kDftTile + LN * q] += (double)tx * e.x - (double)ty * e.y;
          }
        }
      }
      if (DIM == 3 && y0 + 2 == c && kxi < c) {
#pragma unroll
        for (int q = 0; q < P; ++q) {
          const float2 ex = ph[kxi * kDftTile + hl + LN * q];
#pragma unroll
          for (int d = 0; d < DIM; ++d)
            mine[d * kDftTile + LN * q] += (double)sx[q][d].x * ex.x - (double)sx[q][d].y * ex.y;
        }
      }
    }
    __syncthreads();
    for (int i = tid; i < kDftTile * DIM; i += blockDim.x) {
      const long long j = j0 + i / DIM;
      if (j >= np) continue;
      double t = 0.0;
      for (int h = 0; h < nhw; ++h) t += sums[(h * DIM + i % DIM) * kDftTile + i / DIM];
      const double ur = t * __longlong_as_double((1023LL - DIM * lc) << 52);  // / c^DIM
      u_r[j * DIM + i % DIM] = ur;
      if (r_out) {
        r_out[j * DIM + i % DIM] = wrap_period(r[j * DIM + i % DIM] + dt * ur, 2.0 * 3.14159265358979323846);
      }
    }
    __syncthreads();  // before the next tile's tables
  }
}

// Grids that a one-thread-per-particle block of 128 could not serve (phase tables above
// 227 KB) stay refused by the callers.
inline bool dft_supported(int dim, int c) { return sizeof(float2) * dim * c * 128 <= 227 * 1024; }
constexpr int kDftMaxC = 64;  // the largest of them, 2D and 3D

// Launches k_dft_interp over np particles: two per lane while one round of two blocks per
// SM takes them all (32^3 modes: 300 particles 74 against 103 us with four), four above, where
// the shared memory reads bound (9000: 205 two per lane, 177 four; 32768: 653, 529).
inline cudaError_t dft_launch(int dim, const float2* hh, long long hcs, int c, const double* r, long long np,
                              double* u_r, double dt, double* r_out, cudaStream_t s) {
  auto go = [&](auto cfg, auto kernel) {
    using K = decltype(cfg);
    const long long tiles = (np + K::TILE - 1) / K::TILE;
    const unsigned grid = (unsigned)(tiles < (1LL << 30) ? tiles : (1LL << 30));
    const size_t smem = K::smem(c);
    // the limit of the largest c, whatever this one's: another thread may set it between this
    // call and the launch
    const cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)K::smem(kDftMaxC));
    if (e != cudaSuccess) return e;
    pdl_launch(kernel, grid, K::threads(c), smem, s, hh, hcs, c, r, np, u_r, dt, r_out);
    return cudaGetLastError();
  };
  const bool small = np <= 2LL * sm_count() * DftCfg<3, 2>::TILE;
  if (dim == 3) return small ? go(DftCfg<3, 2>{}, k_dft_interp<3, 2>) : go(DftCfg<3, 4>{}, k_dft_interp<3, 4>);
  return small ? go(DftCfg<2, 2>{}, k_dft_interp<2, 2>) : go(DftCfg<2, 4>{}, k_dft_interp<2, 4>);
}

}  // namespace l3es
