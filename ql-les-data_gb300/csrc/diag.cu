// Diagnostics of the drivers (l3es/spectral_solver.py:123-127, :318-320;
// l3es/utils.py:35-97, :300-315) with FP64 partial sums. Each point's or mode's
// contribution is formed in FP32 and accumulated in float-float (Ff, ~48 bits: energy and
// dissipation) or in F3 (at least FP64's bits: statistics and spectrum); FP64 arithmetic is
// scarce on this GPU and only combines the threads' sums.
//   l3es_field_stats      max |u_c| per component and 0.5 mean sum u^2 of a physical field
//   l3es_dissipation      nu <|curl u|^2> by Parseval on the half spectrum
//   l3es_energy_spectrum  shell sums E(k), shells int(|k| + 0.5)
#include <cuda_runtime.h>

#include <cmath>

#include "l3es_internal.h"

namespace l3es {

// Sum of non-negative FP32 terms that loses less than an FP64 one: every addition's rounding
// error goes to b and that addition's to c (TwoSum), so only c rounds, at 2^-72 of the sum.
// Thirteen FP32 instructions a term; FP64 runs at two a clock and SM. An infinite or overflowing
// sum has NaN error terms: where a is not finite the caller adds in FP64.
struct F3 {
  float a, b, c;
  // (c is zero unless the terms' sizes differ by 2^24, and converting it costs as much as the
  // others)
  __device__ __forceinline__ double value() const {
    double lo = (double)b;
    if (c != 0.f) lo += (double)c;
    return lo + (double)a;
  }
};
__device__ __forceinline__ float two_sum(float x, float y, float& err) {
  const float s = x + y, q = s - x;
  err = (x - (s - q)) + (y - q);
  return s;
}
__device__ __forceinline__ F3 f3_add(F3 s, F3 t) {
  float e0, e1, e2;
  s.a = two_sum(s.a, t.a, e0);
  s.b = two_sum(two_sum(s.b, t.b, e1), e0, e2);
  s.c += t.c + (e1 + e2);
  return s;
}
// the sum of M terms over pairs, pairs of pairs, ...
template <int M>
__device__ __forceinline__ F3 f3_tree(const float* e) {
  if constexpr (M == 2) {
    F3 s{0.f, 0.f, 0.f};
    s.a = two_sum(e[0], e[1], s.b);
    return s;
  } else {
    return f3_add(f3_tree<M / 2>(e), f3_tree<M / 2>(e + M / 2));
  }
}

// Eight floats from p + i on (VEC: two 16-byte loads), zeros from n on.
template <bool VEC>
__device__ __forceinline__ void load8(const float* __restrict__ p, unsigned i, unsigned n, float (&v)[8]) {
  if (VEC && i + 8 <= n) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p + i)), b = __ldg(reinterpret_cast<const float4*>(p + i) + 1);
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
  } else {
#pragma unroll
    for (int q = 0; q < 8; ++q) v[q] = i + q < n ? __ldg(p + i + q) : 0.f;
  }
}

// per block: max |u_c| for c = 0..2 and sum_c u_c^2, over ps values per component; eight
// neighbouring points per thread and turn, the sum in F3 (where that is not finite, again in
// FP64). VEC: u is 16-byte aligned and ps a multiple of 4. Bound by the reads: both launches
// take 35.8 us on a 256^3 field, 201 MB (35.3 with the sum in float-float, which keeps 48 bits;
// 68 with one point in flight and an FP64 addition per point).
template <bool VEC>
__global__ void __launch_bounds__(256)
k_field_stats(const float* __restrict__ u, long long ps, int nblk, double* __restrict__ partial) {
  pdl_begin();
  const int batch = blockIdx.y;
  const float* ub = u + (long long)batch * 3 * ps;
  float mx[3] = {0.f, 0.f, 0.f};
  F3 acc{0.f, 0.f, 0.f};
  const unsigned n = (unsigned)ps, step = 8u * (unsigned)nblk * blockDim.x;  // ps <= 512^3
  const unsigned first = 8u * (blockIdx.x * blockDim.x + threadIdx.x);
  auto energy = [](float x, float y, float z) { return fmaf(z, z, fmaf(y, y, x * x)); };
  for (unsigned i = first; i < n; i += step) {
    float v[3][8], e[8];
#pragma unroll
    for (int c = 0; c < 3; ++c) load8<VEC>(ub + c * ps, i, n, v[c]);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
#pragma unroll
      for (int c = 0; c < 3; ++c) mx[c] = fmaxf(mx[c], fabsf(v[c][q]));
      e[q] = energy(v[0][q], v[1][q], v[2][q]);
    }
    acc = f3_add(acc, f3_tree<8>(e));
  }
  double s = acc.value();
  if (!isfinite(acc.a)) {
    s = 0.0;
    for (unsigned i = first; i < n; i += step)
      for (unsigned j = i; j < i + 8 && j < n; ++j) s += (double)energy(ub[j], ub[ps + j], ub[2 * ps + j]);
  }
  __shared__ float smx[3][32];
  __shared__ double ss[32];
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
#pragma unroll
    for (int c = 0; c < 3; ++c) mx[c] = fmaxf(mx[c], __shfl_xor_sync(0xffffffffu, mx[c], o));
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    ss[wid] = s;
    for (int c = 0; c < 3; ++c) smx[c][wid] = mx[c];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    float m[3] = {0.f, 0.f, 0.f};
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      t += ss[w];
      for (int c = 0; c < 3; ++c) m[c] = fmaxf(m[c], smx[c][w]);
    }
    double* o = partial + ((long long)batch * nblk + blockIdx.x) * 4;
    o[0] = m[0];
    o[1] = m[1];
    o[2] = m[2];
    o[3] = t;
  }
}

// out[batch*4 + {0,1,2}] = max |u_c|, out[batch*4 + 3] = 0.5 mean sum u^2; one block per
// trajectory (a single thread walking 608 partials took 163 us)
__global__ void __launch_bounds__(256)
k_field_stats_final(const double* __restrict__ partial, int nblk, double inv_ps, double* __restrict__ out) {
  pdl_begin();
  const int batch = blockIdx.x;
  double m[3] = {0.0, 0.0, 0.0}, s = 0.0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) {
    const double* p = partial + ((long long)batch * nblk + b) * 4;
    for (int c = 0; c < 3; ++c) m[c] = fmax(m[c], p[c]);
    s += p[3];
  }
  __shared__ double red[8][4];
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    for (int c = 0; c < 3; ++c) m[c] = fmax(m[c], __shfl_xor_sync(0xffffffffu, m[c], o));
  }
  if ((threadIdx.x & 31) == 0) {
    double* o = red[threadIdx.x >> 5];
    o[0] = m[0];
    o[1] = m[1];
    o[2] = m[2];
    o[3] = s;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = red[0][threadIdx.x];
    for (int w = 1; w < 8; ++w) t = threadIdx.x < 3 ? fmax(t, red[w][threadIdx.x]) : t + red[w][threadIdx.x];
    out[batch * 4 + threadIdx.x] = threadIdx.x < 3 ? t : 0.5 * t * inv_ps;
  }
}

// dissipation partials: Parseval sum of w |C|^2 over the half spectrum, C = k x u_hat
// with the reference kkk. irfftn keeps only the Hermitian part of the kh = 0 and
// kh = N/2 planes, and i C is not Hermitian there (kz = +N/2 for both partners), so
// those planes use |(C(k) - conj C(-k)) / 2|^2 with weight 1 (utils.py:312-315).
template <int DIM>
__device__ __forceinline__ void curl_of(const float2* v, int n, int kxi, int mid, int kh, float* re, float* im) {
  float k0, k1, k2;
  kvec<DIM>(kfull(kxi, n), DIM == 3 ? kfull(mid, n) : 0, kh, k0, k1, k2);
  const float2 a = v[0], b = v[1], c = v[2];
  // (k x u)_x = k1 c - k2 b, (k x u)_y = k2 a - k0 c, (k x u)_z = k0 b - k1 a
  re[0] = k1 * c.x - k2 * b.x;
  im[0] = k1 * c.y - k2 * b.y;
  re[1] = k2 * a.x - k0 * c.x;
  im[1] = k2 * a.y - k0 * c.y;
  re[2] = k0 * b.x - k1 * a.x;
  im[2] = k0 * b.y - k1 * a.y;
}

// Four neighbouring modes per thread and turn over the flat half spectrum (a warp per
// 129-mode row left every fifth turn to one lane). VEC: uh is 16-byte aligned (cs is even).
template <int DIM, bool VEC>
__global__ void __launch_bounds__(256)
k_diss_partial(const float2* __restrict__ uh, long long cs, int n, int nblk, double* __restrict__ partial) {
  pdl_begin();
  const int batch = blockIdx.y;
  const float2* ub = uh + (long long)batch * 3 * cs;
  const unsigned h = (unsigned)(n / 2 + 1), nmid = DIM == 3 ? (unsigned)n : 1u, ucs = (unsigned)cs;  // cs < 2^31
  const unsigned step = 4u * (unsigned)nblk * blockDim.x;
  Ff s{0.f, 0.f};
  for (unsigned i0 = 4u * (blockIdx.x * blockDim.x + threadIdx.x); i0 < ucs; i0 += step) {
    float v[3][8];
#pragma unroll
    for (int c = 0; c < 3; ++c) load8<VEC>(reinterpret_cast<const float*>(ub + c * cs), 2u * i0, 2u * ucs, v[c]);
    unsigned row = i0 / h;
    int kh = (int)(i0 - row * h);
#pragma unroll
    for (int q = 0; q < 4; ++q, ++kh) {
      if (i0 + q >= ucs) break;
      if (kh == (int)h) {
        kh = 0;
        ++row;
      }
      const int mid = (int)(row % nmid), kxi = (int)(row / nmid);
      const float2 a[3] = {make_float2(v[0][2 * q], v[0][2 * q + 1]), make_float2(v[1][2 * q], v[1][2 * q + 1]),
                           make_float2(v[2][2 * q], v[2][2 * q + 1])};
      float re[3], im[3];
      curl_of<DIM>(a, n, kxi, mid, kh, re, im);
      float e = 0.f;
      if (kh == 0 || kh == n / 2) {
        const int mx = (n - kxi) % n, mm = DIM == 3 ? (n - mid) % n : 0;
        const long long o = ((long long)mx * nmid + mm) * h + kh;
        const float2 w[3] = {ub[o], ub[cs + o], ub[2 * cs + o]};
        float re2[3], im2[3];
        curl_of<DIM>(w, n, mx, mm, kh, re2, im2);
        // Hermitian part of i C is i (C(k) - conj C(-k)) / 2
        for (int c = 0; c < 3; ++c) {
          const float hr = 0.5f * (re[c] - re2[c]), hi = 0.5f * (im[c] + im2[c]);
          e = fmaf(hr, hr, fmaf(hi, hi, e));
        }
      } else {
        for (int c = 0; c < 3; ++c) e = fmaf(re[c], re[c], fmaf(im[c], im[c], e));
        e *= 2.f;
      }
      s = ff_add(s, e);
    }
  }
  block_sum_store_ff(s, partial, batch * nblk + blockIdx.x);
}

constexpr int kSpecThreads = 128;

// Energy spectrum over shells int(|k| + 0.5) < n: per-warp shared-memory histograms of
// the mode count and of weight * |u_hat|^2, merged with FP64 atomics into
// acc[batch][2][n]. The shell depends on the magnitudes of the wavenumbers only, so a warp
// takes all rows (+-a, +-b) and (+-b, +-a) of one pair a >= b (2D: +-a) at once, sums a
// mode's energies over them in F3 (up to 8 rows, 24 loads in flight per lane) and
// makes one shared FP64 addition for the lot: those atomics are a compare-and-swap loop,
// and two per mode into one histogram per block took 289 us on a 256^3 spectrum (76 us with
// one addition per 8 modes, 57 us with a histogram per warp, 52 us with the count's addition
// before the energies, while the loads are in flight). shell int(|k| + 0.5): |k|^2 is an
// integer below 3 (n/2)^2, whose square root is never within 1/(8|k|) of a half integer,
// far more than the FP32 rounding.
template <int DIM>
__global__ void __launch_bounds__(kSpecThreads)
k_spectrum(const float2* __restrict__ uh, long long cs, int n, int nblk, double scale, double* __restrict__ acc) {
  pdl_begin();
  extern __shared__ double s_hist[];  // [warp][n] energies, then [warp][n] counts (32-bit)
  const int batch = blockIdx.y;
  const int wpb = blockDim.x >> 5;
  unsigned* s_cnt = reinterpret_cast<unsigned*>(s_hist + wpb * n);
  for (int i = threadIdx.x; i < wpb * n; i += blockDim.x) {
    s_hist[i] = 0.0;
    s_cnt[i] = 0u;
  }
  __syncthreads();
  double* hist = s_hist + (threadIdx.x >> 5) * n;
  unsigned* cnt = s_cnt + (threadIdx.x >> 5) * n;
  const float2* ub = uh + (long long)batch * 3 * cs;
  const int h = n / 2 + 1, m = n / 2;
  const int lane = threadIdx.x & 31;
  const int tasks = DIM == 3 ? (m + 1) * (m + 2) / 2 : m + 1;
  for (int t = blockIdx.x * wpb + (threadIdx.x >> 5); t < tasks; t += nblk * wpb) {
    int a = t, b = 0;
    if (DIM == 3) {  // t = a (a + 1) / 2 + b, 0 <= b <= a
      a = (int)((sqrtf(8.f * (float)t + 1.f) - 1.f) * 0.5f);
      while (a * (a + 1) / 2 > t) --a;
      while ((a + 1) * (a + 2) / 2 <= t) ++a;
      b = t - a * (a + 1) / 2;
    }
    // storage indices of +-a, +-b: 0 and n/2 stand once
    const int na = a == 0 || a == m ? 1 : 2, nb = DIM == 2 ? 1 : b == 0 || b == m ? 1 : 2;
    const int rows = na * nb * (DIM == 3 && a != b ? 2 : 1);
    constexpr int R = DIM == 3 ? 8 : 2;
    unsigned off[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int sw = r / (na * nb), rr = r - sw * (na * nb);
      const int ia = rr % na == 0 ? a : n - a, ib = rr / na == 0 ? b : n - b;
      const int x = sw ? ib : ia, y = sw ? ia : ib;
      off[r] = r < rows ? (DIM == 3 ? (unsigned)(x * n + y) : (unsigned)x) * (unsigned)h : 0u;
    }
    for (int kh = lane; kh < h; kh += 32) {
      float2 v[R][3];
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) v[r][c] = r < rows ? __ldg(ub + c * cs + off[r] + kh) : make_float2(0.f, 0.f);
      const int k2 = a * a + b * b + kh * kh;
      const int shell = (int)(sqrtf((float)k2) + 0.5f), w = (kh == 0 || kh == n / 2) ? 1 : 2;
      if (shell < n) atomicAdd(cnt + shell, (unsigned)(w * rows));  // while the loads are in flight
      float e[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        e[r] = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) e[r] = fmaf(v[r][c].x, v[r][c].x, fmaf(v[r][c].y, v[r][c].y, e[r]));
      }
      if (shell < n) {
        const F3 f = f3_tree<R>(e);
        double s = f.value();
        if (!isfinite(f.a)) {
          s = 0.0;
          for (int r = 0; r < R; ++r) s += (double)e[r];
        }
        atomicAdd(hist + shell, (w * scale) * s);
      }
    }
  }
  __syncthreads();
  double* ab = acc + (long long)batch * 2 * n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    unsigned k = 0;
    double e = 0.0;
    for (int w = 0; w < wpb; ++w) {
      k += s_cnt[w * n + i];
      e += s_hist[w * n + i];
    }
    if (k) {
      atomicAdd(&ab[i], (double)k);
      atomicAdd(&ab[n + i], e);
    }
  }
}

// sum of n partials per trajectory times scale
__global__ void __launch_bounds__(256)
k_diag_sum(const double* __restrict__ partial, int n, double scale, double* __restrict__ out) {
  pdl_begin();
  __shared__ double red[32];
  const int batch = blockIdx.x;
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += partial[(long long)batch * n + i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < (int)(blockDim.x >> 5); ++i) t += red[i];
    out[batch] = t * scale;
  }
}

__global__ void k_spectrum_final(const double* __restrict__ acc, int n, double eps, double* __restrict__ ek) {
  pdl_begin();
  const int batch = blockIdx.y;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const double* a = acc + (long long)batch * 2 * n;
  const double pi = 3.14159265358979323846;
  ek[(long long)batch * n + k] = a[n + k] * 4.0 * pi * (double)k * k / (a[k] + eps);
}

}  // namespace l3es

using namespace l3es;

extern "C" {

int l3es_field_stats(l3es_plan* plan, const float* u, double* out_dev, void* stream) {
  if (!plan || !u || !out_dev) return fail(L3ES_EINVAL, "l3es_field_stats: null argument");
  const Ctx& c = plan_ctx(plan);
  cudaStream_t s = (cudaStream_t)stream;
  const int nblk = (int)std::min<long long>(608, (c.ps + 2047) / 2048);
  const bool vec = !misaligned16(u) && c.ps % 4 == 0;
  L3ES_LAUNCH(c, KK_REDUCE, 4.0 * 3.0 * c.ps * c.batch, s,
              pdl_launch(vec ? k_field_stats<true> : k_field_stats<false>, dim3(nblk, c.batch), 256, 0, s, u, c.ps,
                         nblk,
                         c.partial));
  L3ES_LAUNCH(c, KK_REDUCE, 0.0, s,
              pdl_launch(k_field_stats_final, c.batch, 256, 0, s, c.partial, nblk, 1.0 / (double)c.ps, out_dev));
  return cuda_check(cudaGetLastError(), "l3es_field_stats launch");
}

int l3es_dissipation(l3es_plan* plan, const void* u_hat, double nu, double* out_dev, void* stream) {
  if (!plan || !u_hat || !out_dev) return fail(L3ES_EINVAL, "l3es_dissipation: null argument");
  const Ctx& c = plan_ctx(plan);
  cudaStream_t s = (cudaStream_t)stream;
  const int nblk = (int)std::min<long long>(608, (c.cs + 1023) / 1024);
  const double scale = nu / std::pow((double)c.n, 2 * c.dim);
  const bool vec = !misaligned16(u_hat);
  auto kernel = c.dim == 3 ? (vec ? k_diss_partial<3, true> : k_diss_partial<3, false>)
                           : (vec ? k_diss_partial<2, true> : k_diss_partial<2, false>);
  L3ES_LAUNCH(c, KK_REDUCE, 8.0 * 3.0 * c.cs * c.batch, s,
              pdl_launch(kernel, dim3(nblk, c.batch), 256, 0, s, (const float2*)u_hat, c.cs, c.n, nblk, c.partial));
  L3ES_LAUNCH(c, KK_REDUCE, 0.0, s, pdl_launch(k_diag_sum, c.batch, 256, 0, s, c.partial, nblk, scale, out_dev));
  return cuda_check(cudaGetLastError(), "l3es_dissipation launch");
}

int l3es_energy_spectrum(l3es_plan* plan, const void* u_hat, double mul_fac, double* ek_dev, void* stream) {
  if (!plan || !u_hat || !ek_dev) return fail(L3ES_EINVAL, "l3es_energy_spectrum: null argument");
  const Ctx& c = plan_ctx(plan);
  cudaStream_t s = (cudaStream_t)stream;
  const int n = c.n;
  int rc = cuda_check(cudaMemsetAsync(c.partial, 0, sizeof(double) * 2 * n * c.batch, s), "l3es_energy_spectrum");
  if (rc != L3ES_OK) return rc;
  // one warp per pair of wavenumber magnitudes; few of them per warp, so that the last ones
  // do not run alone (256^3, 8385 pairs: 608 blocks of 4 warps 63 us, 1216 57 us)
  const long long tasks = c.dim == 3 ? (long long)c.h * (c.h + 1) / 2 : c.h;
  const int nblk = (int)std::min<long long>(1216, (tasks + kSpecThreads / 32 - 1) / (kSpecThreads / 32));
  // |u_hat / n^dim|^2 * mul_fac (utils.py:82-86)
  const double scale = mul_fac / std::pow((double)n, 2 * c.dim);
  const size_t smem = (sizeof(double) + sizeof(unsigned)) * n * (kSpecThreads / 32);
  if (c.dim == 3)
    L3ES_LAUNCH(c, KK_REDUCE, 8.0 * 3.0 * c.cs * c.batch, s,
                pdl_launch(k_spectrum<3>, dim3(nblk, c.batch), kSpecThreads, smem, s, (const float2*)u_hat, c.cs, n,
                           nblk, scale,
                                                                    c.partial));
  else
    L3ES_LAUNCH(c, KK_REDUCE, 8.0 * 3.0 * c.cs * c.batch, s,
                pdl_launch(k_spectrum<2>, dim3(nblk, c.batch), kSpecThreads, smem, s, (const float2*)u_hat, c.cs, n,
                           nblk, scale,
                                                                    c.partial));
  L3ES_LAUNCH(c, KK_REDUCE, 0.0, s,
              pdl_launch(k_spectrum_final, dim3((n + 127) / 128, c.batch), 128, 0, s, c.partial, n,
                         2.220446049250313e-16,
                                                                              ek_dev));
  return cuda_check(cudaGetLastError(), "l3es_energy_spectrum launch");
}

}  // extern "C"
