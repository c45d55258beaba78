// Pseudo-spectral Navier-Stokes kernels (2D and 3D periodic box) for sm_103a.
//
// Spectral arrays use the reference layout (l3es/spectral_solver.py:206):
//   3D  u_hat[c][kx][ky][kz], kz in [0, N/2]  (rfftn over axes 1,2,3)
//   2D  u_hat[c][kx][ky],     ky in [0, N/2]  (rfftn over axes 1,2, squeezed)
// i.e. a half axis of H = N/2+1 complex64 values, preceded by a "middle" axis
// (3D: N values, 2D: none) and the full x axis.
//
// One right-hand side evaluation + RK stage (l3es/spectral_solver.py:50-60, :74-80)
// is six passes:
//   kx_inv       x-axis inverse c2c of u_hat and of i k x u_hat (curl prologue)
//   ky_pass      y-axis inverse c2c (3D only), 6 fields in place
//   line_cross   half-axis c2r of the 6 fields, u x curl, r2c of the 3 products,
//                stored only for the kept (dealiased) half-axis modes
//   ky_pass      y-axis forward c2c (3D only), stored only for kept ky rows
//   kx_fwd_band  x-axis forward c2c on the kept band, dealias mask, Leray projection
//                (and the constant-power band coefficient of the stage field)
//   k_rk_update  elementwise viscosity, extension terms and RK4 stage combination
// The default explicit step has no elementwise pass: in 2D and on small 3D grids
// kx_stage (stage_kernels.cuh) takes the places of kx_fwd_band, k_rk_update and the next
// stage's kx_inv; on larger 3D grids kx_fwd_band combines the stages on the band in place,
// and the next stage's kx_inv scales every other mode by the closed form of its linear
// decay (XLin, BandRk).
// Intermediate fields never exist in physical space in HBM.
#pragma once

#include "fft_core.cuh"
#include "pdl.cuh"
#include "tma.cuh"

namespace l3es {

constexpr int TW = 8;  // pencils (columns) per CTA in the strided x / y passes

// Bits of a plan's device error word (reported and cleared by l3es_plan_check).
constexpr int kErrTimeout = 1;    // a bounded wait on a bulk copy ran out
constexpr int kErrNonFinite = 2;  // the RK update produced a NaN or infinity

// Half-axis line passes: one line (an M = N/2 point complex FFT) per T = M/8
// threads, all in one warp, so the FFT exchanges use __syncwarp only and warps run
// independently. 4 warps per CTA.
template <int N>
struct LineCfg {
  static constexpr int M = N / 2;                          // half-length complex FFT
  // radix 8: at 16 values per thread the 3 cross-product accumulators spill (measured
  // 224 us vs 193 us per 256^3 launch), so the line passes keep two exchanges
  static constexpr int E = Fft<M>::E;
  static constexpr int T = M / E;                          // threads per line
  static_assert(T <= 32, "line passes need the line inside one warp (N <= 512)");
  static constexpr int LPW = 32 / T;                       // lines per warp
  static constexpr int THREADS = 128;
  static constexpr int LPC = LPW * (THREADS / 32);         // lines per CTA
  static constexpr int XS = xpad_len<1>(M);                // exchange slots per line
  // parked 3-field physical line: stride 3M + T float2, so the 16 / T lines that share a
  // half warp start T slots apart mod 16 and their 8-byte accesses cover all banks
  static constexpr int PS = 3 * M + T;
};

// y-axis pass tiling, two schedules (the plan's autotuner picks one per grid):
//   V = 0: radix 16 from N = 128 (one exchange at N = 256), radix 8 below;
//   V = 1: radix 8 throughout (two exchanges at N = 256, twice the threads per tile).
// 16-column tiles where the shared-memory tile fits the static limit, else 8.
template <int N, int V = 0>
struct KyCfg {
  static constexpr int E = (V == 0 && N >= 128) ? 16 : Fft<N>::E;
  static constexpr int TWY = (N >= 128 && N <= 256) ? 16 : 8;
  static constexpr int T = N / E;
  static constexpr int THREADS = TWY * T;
};

// wavenumber vector (reference kkk, spectral_solver.py:32-39): 3D (kx, kmid, khalf),
// 2D (kx, khalf, 0); the half-axis Nyquist entry is +N/2.
template <int DIM>
__device__ __forceinline__ void kvec(int kx, int km, int kh, float& k0, float& k1, float& k2) {
  k0 = (float)kx;
  if (DIM == 3) {
    k1 = (float)km;
    k2 = (float)kh;
  } else {
    k1 = (float)kh;
    k2 = 0.f;
  }
}

// Closed-form RK4 of a mode whose right-hand side is exactly -(nu k^2 + drag) u (no
// nonlinear or forcing term), z = (nu k^2 + drag) dt: the field that stage rk writes is
// a polynomial in z times the step's initial state u0,
//   rk 0: 1 - z/2               rk 1: 1 - z/2 + z^2/4
//   rk 2: 1 - z + z^2/2 - z^3/4 rk 3: 1 - z + z^2/2 - z^3/6 + z^4/24 (the new state)
__device__ __forceinline__ float lin_stage_factor(int rk, float z) {
  if (rk == 0) return fmaf(-0.5f, z, 1.f);
  if (rk == 1) return fmaf(z, fmaf(0.25f, z, -0.5f), 1.f);
  if (rk == 2) return fmaf(z, fmaf(z, fmaf(-0.25f, z, 0.5f), -1.f), 1.f);
  return fmaf(z, fmaf(z, fmaf(z, fmaf(z, 1.f / 24.f, -1.f / 6.f), 0.5f), -1.f), 1.f);
}

// RK4 step with the stage combination fused into the band pass (kx_fwd_band FUSED):
// the band B = {|kx| <= kd, |kmid| <= kd (3D), khalf < kt} holds the nonlinear and
// forcing terms, and its stage fields are written in place into the state S; every
// other mode keeps the step's initial value u0 in S during the step. The x inverse of
// stage rk (> 0) reads S and scales a mode outside B by lin_stage_factor(rk - 1, z) on
// the fly, so that mode is neither read nor written by an elementwise update; the last
// stage's x inverse also writes its new state lin_stage_factor(3, z) u0 back to S.
struct XLin {
  float2* S;                 // the state (the x pass's input), [batch][3][cs]
  long long cs;
  const float* nu_b;         // per-trajectory viscosity
  float drag, dt;
  int kd, kt, rk;            // rk 0 passes u0 through unscaled
  int band_kf;               // > 0: block 0 of each trajectory computes the constant-power
  double inv_n2d, eps_inj;   //   coefficient of the stage field into band_scale
  double* band_scale;
};

template <int DIM, int THREADS>
__device__ __forceinline__ void band_coefficient(const float2* __restrict__ ub, long long cs, int N, int kf,
                                                 double inv_n2d, double eps_inj, double tiny, double* out);

// Scale the outside-B modes of one x-pass column tile (a[c][e]: x row t + T e of column
// m = mid * H + kh) to stage rk's field; the last stage stores their new state to S.
template <int N>
__device__ __forceinline__ void xlin_scale(float2 (&a)[3][Fft<N>::E], int t, int m, const XLin& xl, int batch,
                                           int* __restrict__ err) {
  constexpr int E = Fft<N>::E, T = Fft<N>::T, H = N / 2 + 1;
  constexpr int MC = N * H;
  const int mid = m / H;
  const int kh = m - mid * H;
  const int km = kfull(mid, N);
  const unsigned ukd = 2u * (unsigned)xl.kd;
  const bool colband = (unsigned)(km + xl.kd) <= ukd && kh < xl.kt;
  const float nu = xl.nu_b[batch];
  const int k2c = km * km + kh * kh;
  bool bad = false;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int kx = kfull(t + T * e, N);
    if (colband && (unsigned)(kx + xl.kd) <= ukd) continue;
    const float z = (nu * (float)(kx * kx + k2c) + xl.drag) * xl.dt;
    if (xl.rk == 3) {
      const float g = lin_stage_factor(3, z);
      float2* dst = xl.S + (long long)batch * 3 * xl.cs + (long long)(t + T * e) * MC + m;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float2 nv = make_float2(g * a[c][e].x, g * a[c][e].y);
        dst[c * xl.cs] = nv;
        bad |= !isfinite(nv.x + nv.y);
      }
    }
    const float f = lin_stage_factor(xl.rk - 1, z);
#pragma unroll
    for (int c = 0; c < 3; ++c) a[c][e] = make_float2(f * a[c][e].x, f * a[c][e].y);
  }
  if (bad) atomicOr(err, kErrNonFinite);
}

// ------------------------------------------------------------------------------
// x-axis inverse pass. Columns m in [0, NMID*H) of each x-plane; CURL adds the
// three components of i k x u_hat (np.cross(kkk, u_hat) * 1j) as fields 3..5.
// ------------------------------------------------------------------------------
// The six fields of one tile of TW columns m = mid * H + kh (a[c][e]: component c at
// x row t + T e of column m): x-axis inverse FFT of u and of i k x u, stored to w.
// SKIPWX (3D RHS): field 3 (curl_x) is neither transformed nor stored, and fields 1, 2
// (u_y, u_z) go to the side buffer wx + wxofs (two fields) instead; the y pass
// (ky_inv_rhs) forms curl_x from them and writes all six fields.
template <int N, int DIM, bool CURL, bool SKIPWX = false, int XW = TW>
__device__ __forceinline__ void kx_inv_fields(float2 (&a)[3][Fft<N>::E], int t, int m, bool ok, float2* sm,
                                              float2* __restrict__ w, long long wofs, long long fs,
                                              const float2* __restrict__ tw, float2* __restrict__ wx = nullptr,
                                              long long wxofs = 0) {
  constexpr int E = Fft<N>::E, T = Fft<N>::T, H = N / 2 + 1;
  constexpr int NMID = DIM == 3 ? N : 1;
  constexpr int MC = NMID * H;
  constexpr int NF = CURL ? 6 : 3;
  const int kh = m % H;
  const int km = DIM == 3 ? kfull(m / H, N) : 0;
#pragma unroll
  for (int f = 0; f < NF; ++f) {
    if (SKIPWX && f == 3) continue;
    float2 v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (f < 3) {
        v[e] = a[f][e];
      } else {
        float k0, k1, k2;
        kvec<DIM>(kfull(t + T * e, N), km, kh, k0, k1, k2);
        float2 cr;
        if (f == 3) {
          cr = make_float2(k1 * a[2][e].x - k2 * a[1][e].x, k1 * a[2][e].y - k2 * a[1][e].y);
        } else if (f == 4) {
          cr = make_float2(k2 * a[0][e].x - k0 * a[2][e].x, k2 * a[0][e].y - k0 * a[2][e].y);
        } else {
          cr = make_float2(k0 * a[1][e].x - k1 * a[0][e].x, k0 * a[1][e].y - k1 * a[0][e].y);
        }
        v[e] = mul_i<kInv>(cr);  // times 1j
      }
    }
    // single adds from 256: paired, the 512^3 pass took 1235 us instead of 1222, the 256^3
    // pass 116 and 115; a 128^3 step and its physical field 338 us instead of 330 so
    block_fft<N, E, kInv, XW, kSyncCta, false, N <= 128>(v, sm, t, tw, 1);
    if (ok) {
      float2* dst = (SKIPWX && (f == 1 || f == 2)) ? wx + wxofs + (f - 1) * fs : w + wofs + f * fs;
#pragma unroll
      for (int e = 0; e < E; ++e) dst[(long long)(t + T * e) * MC + m] = v[e];
    }
    __syncthreads();
  }
}

// LINF: the x inverse of a band-fused RK stage (XLin). XW: columns per CTA (2D grids
// take narrow tiles: one 256^2 field has only 129 columns).
template <int N, int DIM, bool CURL, bool SKIPWX = false, bool LINF = false, int XW = TW>
__global__ void __launch_bounds__(XW * Fft<N>::T)
kx_inv(const float2* __restrict__ uh, long long cs, float2* __restrict__ w, long long fs,
       const float2* __restrict__ tw, float2* __restrict__ wx = nullptr, XLin xl = XLin{},
       int* __restrict__ err = nullptr) {
  pdl_begin();
  constexpr int E = Fft<N>::E, T = Fft<N>::T, H = N / 2 + 1;
  constexpr int NMID = DIM == 3 ? N : 1;
  constexpr int MC = NMID * H;
  constexpr int NF = CURL ? 6 : 3;
  __shared__ float2 sm[xpad_len<XW>(N) * XW];
  const int p = threadIdx.x % XW, t = threadIdx.x / XW;
  const int m = blockIdx.x * XW + p;
  const bool ok = m < MC;
  const long long bofs = (long long)blockIdx.y * 3 * cs;  // batch of trajectories
  if constexpr (LINF) {
    if (xl.band_kf > 0 && blockIdx.x == 0)
      band_coefficient<DIM, XW * T>(uh + bofs, cs, N, xl.band_kf, xl.inv_n2d, xl.eps_inj, 1e-30,
                                    xl.band_scale + blockIdx.y);
  }
  float2 a[3][E];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int e = 0; e < E; ++e)
      a[c][e] = ok ? uh[bofs + c * cs + (long long)(t + T * e) * MC + m] : make_float2(0.f, 0.f);
  if constexpr (LINF) {
    if (ok && xl.rk > 0) xlin_scale<N>(a, t, m, xl, (int)blockIdx.y, err);
  }
  kx_inv_fields<N, DIM, CURL, SKIPWX, XW>(a, t, m, ok, sm + p, w, (long long)blockIdx.y * NF * fs, fs, tw, wx,
                                          (long long)blockIdx.y * 2 * fs);
}

// Persistent 3D variant: each CTA walks the tiles blockIdx.x, + gridDim.x, ...; the
// next tile's 3 x N x TW input block (all three components) is fetched by one bulk
// tensor load into shared memory while the current tile is transformed. The staging
// block is refilled only after every thread has copied its elements to registers.
// umap: u_hat as a 3D tensor (MC columns, N rows, 3 * batch components), box
// (TW, min(N, 256), 3). A wait that times out sets *err and ends the CTA's loop.
template <int N>
struct KxTma {
  static constexpr int NY = N > 256 ? 256 : N;   // rows per bulk load (box limit 256)
  static constexpr int LOADS = N / NY;
  static constexpr int STAGE = 3 * N * TW;       // float2 per tile
  static constexpr int SMEM = (STAGE + xpad_len<TW>(N) * TW) * (int)sizeof(float2);
  static constexpr unsigned BYTES = (unsigned)STAGE * sizeof(float2);
};

template <int N, bool CURL, bool SKIPWX = false>
__global__ void __launch_bounds__(TW * Fft<N>::T, TW * Fft<N>::T >= 512 ? 1 : 2)
kx_inv_tma(const __grid_constant__ CUtensorMap umap, float2* __restrict__ w, long long fs,
           const float2* __restrict__ tw, int ntiles, int* __restrict__ err, float2* __restrict__ wx) {
  pdl_begin();
  using K = KxTma<N>;
  constexpr int E = Fft<N>::E, T = Fft<N>::T;
  constexpr int NF = CURL ? 6 : 3;
  extern __shared__ __align__(128) float2 s_dyn[];
  float2* stage = s_dyn;            // [load][c][NY rows][TW columns]
  float2* sm = s_dyn + K::STAGE;    // FFT exchange
  __shared__ uint64_t bar;
  const int p = threadIdx.x % TW, t = threadIdx.x / TW;
  const int batch = blockIdx.y;
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  auto issue = [&](int tile) {
    mbar_arrive_expect_tx(&bar, K::BYTES);
#pragma unroll
    for (int l = 0; l < K::LOADS; ++l)
      tma_load_3d(stage + l * 3 * K::NY * TW, &umap, &bar, tile * TW, l * K::NY, 3 * batch);
  };
  int tile = blockIdx.x;
  if (threadIdx.x == 0 && tile < ntiles) issue(tile);
  unsigned parity = 0;
  for (; tile < ntiles; tile += gridDim.x) {
    // warp 0 polls the barrier; the other threads check it once after the CTA barrier
    // (the phase is complete then), which orders the bulk copy's writes before their reads
    const bool got = threadIdx.x < 32 ? mbar_wait(&bar, parity) : true;
    if (__syncthreads_or(!got)) {  // every thread leaves together
      if (threadIdx.x == 0) atomicOr(err, kErrTimeout);
      // the load in flight (if any) must land before the CTA's shared memory is released
      mbar_wait(&bar, parity);
      return;
    }
    if (threadIdx.x >= 32) mbar_wait(&bar, parity);
    parity ^= 1u;
    float2 a[3][E];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int row = t + T * e;
        a[c][e] = stage[(((row / K::NY) * 3 + c) * K::NY + row % K::NY) * TW + p];
      }
    __syncthreads();  // the staging block is free
    const int next = tile + gridDim.x;
    if (threadIdx.x == 0 && next < ntiles) {
      fence_proxy_async_smem();
      issue(next);
    }
    kx_inv_fields<N, 3, CURL, SKIPWX>(a, t, tile * TW + p, true, sm + p, w, (long long)batch * NF * fs, fs, tw,
                                      wx, (long long)batch * 2 * fs);
  }
}

// ------------------------------------------------------------------------------
// y-axis pass (3D only), in place on fields [blockIdx.z]: rows of `row` complex,
// columns [0, ncols). Only rows whose signed wavenumber satisfies |ky| <= kd_store
// are written (forward pass truncated to the dealiased band; kd_store = N/2 keeps all).
// ------------------------------------------------------------------------------
template <int N, int DIR, int V = 0>
__global__ void __launch_bounds__(KyCfg<N, V>::THREADS)
ky_pass(float2* __restrict__ w, long long fs, int row, int ncols, int kd_store,
        const float2* __restrict__ tw) {
  pdl_begin();
  using C = KyCfg<N, V>;
  constexpr int E = C::E, T = C::T, TWY = C::TWY;
  __shared__ float2 sm[xpad_len<TWY>(N) * TWY];
  const int p = threadIdx.x % TWY, t = threadIdx.x / TWY;
  const int col = blockIdx.x * TWY + p;
  const bool ok = col < ncols;
  float2* base = w + blockIdx.z * fs + (long long)blockIdx.y * N * row + col;
  float2 v[E];
#pragma unroll
  for (int e = 0; e < E; ++e) v[e] = ok ? base[(long long)(t + T * e) * row] : make_float2(0.f, 0.f);
  block_fft<N, E, DIR, TWY>(v, sm + p, t, tw, 1);
  if (ok) {
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int ky = t + T * e;
      const int k = kfull(ky, N);
      if ((unsigned)(k + kd_store) <= 2u * (unsigned)kd_store) base[(long long)ky * row] = v[e];  // |k| <= kd_store
    }
  }
}

// 3D y inverse pass of the RHS: six one-FFT jobs per (column tile, kx plane blockIdx.y,
// trajectory blockIdx.z), the job index varying fastest (blockIdx.x = 6 tile + job) so
// the jobs that share an input run side by side and its second read is served by L2:
//   jobs 0..2: u_x, curl_y, curl_z (fields 0, 4, 5) in place;
//   job 3: curl_x = FFT_y(i (ky W_z - kz W_y)) -> field 3; after the x pass curl_x is
//          that pointwise combination (ky, kz are constant along an x pencil), so the x
//          pass does not store it;
//   jobs 4, 5: u_y, u_z from the side buffer wx (x-transformed W_y, W_z) -> fields 1, 2.
// No job writes what another job reads.
template <int N, int V = 0>
__global__ void __launch_bounds__(KyCfg<N, V>::THREADS)
ky_inv_rhs(float2* __restrict__ w, const float2* __restrict__ wx, long long fs, const float2* __restrict__ tw) {
  pdl_begin();
  using C = KyCfg<N, V>;
  constexpr int E = C::E, T = C::T, TWY = C::TWY, H = N / 2 + 1;
  __shared__ float2 sm[xpad_len<TWY>(N) * TWY];
  const int p = threadIdx.x % TWY, t = threadIdx.x / TWY;
  const int job = blockIdx.x % 6, col = (blockIdx.x / 6) * TWY + p;
  const bool ok = col < H;
  const long long plane = (long long)blockIdx.y * N * H + col;
  float2* wb = w + (long long)blockIdx.z * 6 * fs + plane;
  const float2* xb = wx + (long long)blockIdx.z * 2 * fs + plane;
  float2 v[E];
  if (job == 3) {
    const float kz = (float)col;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const long long o = (long long)(t + T * e) * H;
      const float2 wy = ok ? xb[o] : make_float2(0.f, 0.f);
      const float2 wz = ok ? xb[fs + o] : make_float2(0.f, 0.f);
      const float ky = (float)kfull(t + T * e, N);
      v[e] = mul_i<kInv>(make_float2(ky * wz.x - kz * wy.x, ky * wz.y - kz * wy.y));
    }
  } else {
    const float2* src = job < 3 ? wb + (job == 0 ? 0 : (job + 3) * fs) : xb + (job - 4) * fs;
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = ok ? src[(long long)(t + T * e) * H] : make_float2(0.f, 0.f);
  }
  // single adds at 512: paired, the registers pass the limit of three CTAs per SM (1416 us
  // instead of 1291; held to that limit 1314)
  block_fft<N, E, kInv, TWY, kSyncCta, false, kPaired<E> && N <= 256>(v, sm + p, t, tw, 1);
  if (ok) {
    const int f = job == 0 ? 0 : job < 3 ? job + 3 : job == 3 ? 3 : job - 3;
    float2* dst = wb + f * fs;
#pragma unroll
    for (int e = 0; e < E; ++e) dst[(long long)(t + T * e) * H] = v[e];
  }
}

// Hermitian half-spectrum X[0..M] -> packed z (z[n] = x[2n] + i x[2n+1]) input of an
// M-point inverse FFT (numpy irfft semantics: Im X[0] and Im X[M] are ignored):
//   Z[k] = (X[k] + conj X[M-k]) + i exp(+2 pi i k/N) (X[k] - conj X[M-k]).
__device__ __forceinline__ float2 c2r_pack_pair(float2 a, float2 b, int k, const float2* __restrict__ twN,
                                                float scale) {
  if (k == 0) {
    a.y = 0.f;
    b.y = 0.f;
  }
  const float2 s = make_float2(a.x + b.x, a.y - b.y);  // a + conj(b)
  const float2 d = make_float2(a.x - b.x, a.y + b.y);  // a - conj(b)
  const float2 wk = conjf2(__ldg(twN + k));             // exp(+2 pi i k / N)
  const float2 id = mul_i<kInv>(cmul(wk, d));
  return make_float2(scale * (s.x + id.x), scale * (s.y + id.y));
}

// Packs one half-spectrum line for an M-point c2r by T = M/E threads of one warp
// (thread t holds xk[e] = X[t + T e]; xm = X[M] is used by t = 0 only). Each X[k] is
// read once: the partner X[M-k] lives in thread (T - t) mod T, slot E-1-e (slot
// (E-e) mod E for t = 0, plus X[M] for k = 0), and arrives by warp shuffle.
template <int M, int E>
__device__ __forceinline__ void c2r_pack(const float2 (&xk)[E], float2 xm, int t, float2 (&v)[E],
                                         const float2* __restrict__ twN, float scale) {
  constexpr int T = M / E;
  const int lane = threadIdx.x & 31;
  const int src = lane - t + (t == 0 ? 0 : T - t);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const float2 give = (t == 0) ? xk[(E - e) % E] : xk[E - 1 - e];
    float2 b;
    b.x = __shfl_sync(0xffffffffu, give.x, src);
    b.y = __shfl_sync(0xffffffffu, give.y, src);
    if (t == 0 && e == 0) b = xm;
    v[e] = c2r_pack_pair(xk[e], b, t + T * e, twN, scale);
  }
}

// c2r_pack of a line read from global memory
template <int M, int E>
__device__ __forceinline__ void c2r_load_pack(const float2* __restrict__ X, int t, float2 (&v)[E],
                                              const float2* __restrict__ twN, float scale) {
  constexpr int T = M / E;
  float2 xk[E];
#pragma unroll
  for (int e = 0; e < E; ++e) xk[e] = __ldg(X + t + T * e);
  const float2 xm = __ldg(X + M);  // Nyquist, used by t = 0
  c2r_pack<M, E>(xk, xm, t, v, twN, scale);
}

// M-point forward FFT output Z (exchange buffer, padded index) -> r2c value X[k],
// k in [0, M] (Z is M-periodic; W^M = -1 gives X[M] = Re Z0 - Im Z0).
template <int E>
__device__ __forceinline__ float2 r2c_unpack(const float2* Z, int k, int M,
                                             const float2* __restrict__ twN) {
  const float2 zk = Z[xpad<1, E>(k < M ? k : 0)];
  const float2 zm = Z[xpad<1, E>(k == 0 ? 0 : M - k)];
  const float2 s = make_float2(zk.x + zm.x, zk.y - zm.y);
  const float2 d = make_float2(zk.x - zm.x, zk.y + zm.y);
  const float2 id = mul_i<kFwd>(cmul(__ldg(twN + k), d));  // -i W^k d
  return make_float2(0.5f * (s.x + id.x), 0.5f * (s.y + id.y));
}

// r2c outputs X[k], k = t + T e, from an M-point forward FFT held in registers
// (v[e] = Z[t + T e]); the partner Z[M - k] comes from lane (T - t) mod T by shuffle
// (slot E-1-e, or (E-e) mod E for t = 0, whose e = 0 partner is Z[M] = Z[0]).
template <int M, int E>
__device__ __forceinline__ void r2c_unpack_regs(const float2 (&v)[E], int t, const float2* __restrict__ twN,
                                                float2 (&X)[E]) {
  constexpr int T = M / E;
  const int lane = threadIdx.x & 31;
  const int src = lane - t + (t == 0 ? 0 : T - t);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const float2 give = (t == 0) ? v[(E - e) % E] : v[E - 1 - e];
    float2 zm;
    zm.x = __shfl_sync(0xffffffffu, give.x, src);
    zm.y = __shfl_sync(0xffffffffu, give.y, src);
    const float2 zk = v[e];
    const int k = t + T * e;
    const float2 s = make_float2(zk.x + zm.x, zk.y - zm.y);
    const float2 d = make_float2(zk.x - zm.x, zk.y + zm.y);
    const float2 id = mul_i<kFwd>(cmul(__ldg(twN + k), d));  // -i W^k d
    X[e] = make_float2(0.5f * (s.x + id.x), 0.5f * (s.y + id.y));
  }
}

// ------------------------------------------------------------------------------
// Half-axis line pass of the RHS: 6 half-spectrum lines (u, curl u) -> c2r -> u x
// curl u -> r2c of the 3 products, written for k <= kd (zeros up to kt). scale
// normalises each inverse transform (1/N^dim). Lines are contiguous rows of H.
// Physical u is parked in shared memory (same thread writes and reads it), the
// cross product accumulates in registers while the curl lines are transformed.
// ------------------------------------------------------------------------------
// 4 CTAs (16 warps) per SM up to N = 256: 128 registers, no spills (measured at 256^3:
// 160.6 vs 166.5 us per launch at 3 CTAs / 168 registers; 5 CTAs spill and take 176 us).
// N = 512 (256-point lines, one more exchange stage) would spill at 128 and keeps 3.
template <int N>
__global__ void __launch_bounds__(LineCfg<N>::THREADS, N <= 256 ? 4 : 3)
line_cross(const float2* __restrict__ w, long long fs, float2* __restrict__ du, long long ds,
           int kt, int kd, float scale, const float2* __restrict__ twN, int nlines) {
  pdl_begin();
  using C = LineCfg<N>;
  constexpr int M = C::M, H = N / 2 + 1, E = C::E, T = C::T, LPC = C::LPC;
  __shared__ float2 s_x[LPC * C::XS];
  __shared__ float2 s_u[LPC * C::PS];
  const int batch = blockIdx.y;
  const int q = threadIdx.x / T, t = threadIdx.x % T;
  // lines from the last to the first: the y pass before this one ends with the upper
  // planes of the last fields (still in L2), and the forward y pass after it starts
  // with the lower planes, which this pass writes last (measured: -6 us per stage over
  // the three passes at 256^3)
  const long long idx = (long long)blockIdx.x * LPC + q;
  const bool valid = idx < nlines;
  const long long line = valid ? nlines - 1 - idx : 0;  // idle lines mirror a valid one
  const float2* src = w + (long long)batch * 6 * fs + line * H;
  float2* xs = s_x + q * C::XS;
  float2* su = s_u + q * C::PS;
  float2 cr[3][E];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int e = 0; e < E; ++e) cr[c][e] = make_float2(0.f, 0.f);
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    float2 v[E];
    c2r_load_pack<M, E>(src + f * fs, t, v, twN, scale);
    warp_fft<M, E, kInv>(v, xs, t, twN + N);
    // v[e] packs the physical values at 2n and 2n+1, n = t + T*e
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int n = t + T * e;
      const float2 o = v[e];
      if (f < 3) {
        su[f * M + n] = o;
      } else if (f == 3) {  // curl_x: c_y += u_z w_x, c_z -= u_y w_x
        const float2 uz = su[2 * M + n], uy = su[M + n];
        cr[1][e].x = fmaf(uz.x, o.x, cr[1][e].x);
        cr[1][e].y = fmaf(uz.y, o.y, cr[1][e].y);
        cr[2][e].x = fmaf(-uy.x, o.x, cr[2][e].x);
        cr[2][e].y = fmaf(-uy.y, o.y, cr[2][e].y);
      } else if (f == 4) {  // curl_y: c_x -= u_z w_y, c_z += u_x w_y
        const float2 uz = su[2 * M + n], ux = su[n];
        cr[0][e].x = fmaf(-uz.x, o.x, cr[0][e].x);
        cr[0][e].y = fmaf(-uz.y, o.y, cr[0][e].y);
        cr[2][e].x = fmaf(ux.x, o.x, cr[2][e].x);
        cr[2][e].y = fmaf(ux.y, o.y, cr[2][e].y);
      } else {  // curl_z: c_x += u_y w_z, c_y -= u_x w_z
        const float2 uy = su[M + n], ux = su[n];
        cr[0][e].x = fmaf(uy.x, o.x, cr[0][e].x);
        cr[0][e].y = fmaf(uy.y, o.y, cr[0][e].y);
        cr[1][e].x = fmaf(-ux.x, o.x, cr[1][e].x);
        cr[1][e].y = fmaf(-ux.y, o.y, cr[1][e].y);
      }
    }
    __syncwarp();
  }
  float2* db = du + (long long)batch * 3 * ds + line * kt;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    warp_fft<M, E, kFwd>(cr[c], xs, t, twN + N);
    float2 X[E];
    r2c_unpack_regs<M, E>(cr[c], t, twN, X);
    if (valid) {
      float2* dst = db + c * ds;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int k = t + T * e;
        if (k < kt) dst[k] = k <= kd ? X[e] : make_float2(0.f, 0.f);
      }
      for (int k = M + t; k < kt; k += T) dst[k] = make_float2(0.f, 0.f);  // kt > M only for tiny N
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------
// Half-axis line pass of the RHS, two real lines per complex FFT (N = 64 .. 256).
//
// Two real lines x, y of length N have spectra X, Y (half axis, H = N/2 + 1 values);
// one N-point complex inverse FFT of Z = X_ext + i Y_ext (Hermitian extensions) gives
// x + i y, and one forward FFT of x + i y gives Z with X[k] = (Z[k] + conj Z[N-k]) / 2,
// Y[k] = (Z[k] - conj Z[N-k]) / (2 i). A line's six fields pair up as (u_x, u_y),
// (u_z, curl_x), (curl_y, curl_z): after three inverse FFTs every lane holds all six
// physical values at its own N/T positions, so u x curl u is formed in registers (no
// parking in shared memory). Its x, y components pair in one forward FFT; the z
// component waits for the z component of the next line, and the two share one. A line
// takes T = N/8 lanes (N = 256: a whole warp); a line slot does two lines (A then B),
// lines counted from the last (as in line_cross). Per pair of lines: 9 N-point FFTs
// against 18 N/2-point FFTs with pack / unpack passes and parked velocities.
// ct: compact twiddle table of the N-point FFT (Sched<N, 8>, at line2_ct_offset<N>()
// in the plan's table).
// ------------------------------------------------------------------------------
template <int N>
__host__ __device__ constexpr int line2_ct_offset() {
  return N + Sched<N / 2, Fft<N / 2>::E>::ctlen();
}

// Z[n] = X_ext[n] + i Y_ext[n] for n = t + T e (lane t, slot e) from two half-spectrum
// lines (numpy irfft semantics: the imaginary parts of X[0] and X[N/2] are ignored).
template <int N>
__device__ __forceinline__ void c2r_pair_load(const float2* __restrict__ X, const float2* __restrict__ Y, int t,
                                              float2 (&z)[8]) {
  constexpr int T = N / 8;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int n = t + T * e;
    const bool lo = e < 4;  // n < N/2 (e = 4 starts at the Nyquist entry N/2 + 0)
    const int idx = lo ? n : N - n;
    float2 x = __ldg(X + idx), y = __ldg(Y + idx);
    if ((e == 0 || e == 4) && t == 0) {  // n = 0 and n = N/2: real parts only
      x.y = 0.f;
      y.y = 0.f;
    }
    z[e] = lo ? make_float2(x.x - y.y, x.y + y.x)   // X + i Y
              : make_float2(x.x + y.y, y.x - x.y);  // conj X + i conj Y (mirror N - n)
  }
}

// From Z = FFT(x + i y) in registers (lane t, slot e holds Z[t + T e]): X[k] and Y[k] for
// k = t + T e, e < 4, scaled by s (s includes the 1/2).
template <int N>
__device__ __forceinline__ void r2c_pair_unpack(const float2 (&z)[8], int t, float s, float2 (&X)[4],
                                                float2 (&Y)[4]) {
  constexpr int T = N / 8;
  const int lane = threadIdx.x & 31;
  const int src = lane - t + (t == 0 ? 0 : T - t);  // lane holding Z[N - k]
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    // the partner Z[N - k] is slot 7 - e of lane T - t, or slot (8 - e) mod 8 of lane 0
    const float2 give = (t == 0) ? z[(8 - e) & 7] : z[7 - e];
    float2 zm;
    zm.x = __shfl_sync(0xffffffffu, give.x, src);
    zm.y = __shfl_sync(0xffffffffu, give.y, src);
    const float2 zk = z[e];
    X[e] = make_float2(s * (zk.x + zm.x), s * (zk.y - zm.y));
    Y[e] = make_float2(s * (zk.y + zm.y), s * (zm.x - zk.x));
  }
}

// stores X[k], k = t + T e < kt, of one DU line (zeros for kd < k < kt)
template <int N>
__device__ __forceinline__ void store_du_line(float2* __restrict__ dst, const float2 (&X)[4], int t, int kt, int kd) {
  constexpr int T = N / 8;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int k = t + T * e;
    if (k < kt) dst[k] = k <= kd ? X[e] : make_float2(0.f, 0.f);
  }
}

template <int N>
struct Line2Cfg {
  static constexpr int T = N / 8;             // lanes per line
  static constexpr int THREADS = 128;
  static constexpr int SLOTS = THREADS / T;   // line slots per CTA
  static constexpr int LPC = 2 * SLOTS;       // lines per CTA (two per slot)
  static constexpr int XS = xpad_len<1>(N);   // exchange slots per line slot
};

// L1 prefetch of the six field lines of one line (H float2 each, fs apart): 9 prefetches
// of 128 bytes cover a 1032-byte line at any 8-byte offset; lanes share the 54.
template <int N>
__device__ __forceinline__ void prefetch_line6(const float2* src, long long fs, int t) {
  constexpr int T = N / 8, H = N / 2 + 1, CH = (H * 8 + 127) / 128 + ((H * 8) % 128 ? 1 : 0);
  for (int k = t; k < 6 * CH; k += T) {
    const int f = k / CH, q = k % CH;
    const float2* a = src + f * fs + (q * 16 < H ? q * 16 : H - 1);
    asm volatile("prefetch.global.L1 [%0];" ::"l"(a));
  }
}

// One line pair (A, B) per line slot, lines counted from the last; line B's six input
// lines are prefetched into L1 while line A is transformed, so B's loads hit L1 instead
// of waiting on L2 / DRAM (the kernel's registers leave no room for a register prefetch).
// Measured alternatives, kept out: persistent slots walking many pairs with a prefetch of
// each next line (144.7 vs 141.5 us at 256^3: the drifting warps miss the instruction
// cache), the same with rolled loops and work counters (161 us: 22% more instructions).
template <int N>
__global__ void __launch_bounds__(Line2Cfg<N>::THREADS, 4)
line_cross2(const float2* __restrict__ w, long long fs, float2* __restrict__ du, long long ds, int kt, int kd,
            float s2, const float2* __restrict__ ct, int nlines) {
  pdl_begin();
  static_assert(N >= 64 && N <= 256, "two-for-one line pass: N in [64, 256]");
  using C = Line2Cfg<N>;
  constexpr int T = C::T, H = N / 2 + 1;
  __shared__ float2 s_x[C::SLOTS * C::XS];
  const int slot = threadIdx.x / T, t = threadIdx.x % T;
  float2* xs = s_x + slot * C::XS;
  const float2* wb = w + (long long)blockIdx.y * 6 * fs;
  float2* db = du + (long long)blockIdx.y * 3 * ds;
  const long long ia = 2 * ((long long)blockIdx.x * C::SLOTS + slot);  // line A; B = A + 1
  if (ia + 1 < nlines) prefetch_line6<N>(wb + (nlines - 2 - ia) * H, fs, t);
  float pa[8], pb[8];  // z component of u x curl u of lines A and B
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const long long idx = ia + half;
    const bool valid = idx < nlines;
    const long long line = valid ? nlines - 1 - idx : nlines - 1;  // idle slots mirror a valid line
    const float2* src = wb + line * H;
    float2 h1[8], h2[8], z[8];
    c2r_pair_load<N>(src, src + fs, t, z);  // u_x + i u_y
    warp_fft<N, 8, kInv>(z, xs, t, ct);
#pragma unroll
    for (int e = 0; e < 8; ++e) h1[e] = z[e];
    __syncwarp();
    c2r_pair_load<N>(src + 2 * fs, src + 3 * fs, t, z);  // u_z + i curl_x
    warp_fft<N, 8, kInv>(z, xs, t, ct);
#pragma unroll
    for (int e = 0; e < 8; ++e) h2[e] = z[e];
    __syncwarp();
    c2r_pair_load<N>(src + 4 * fs, src + 5 * fs, t, z);  // curl_y + i curl_z
    warp_fft<N, 8, kInv>(z, xs, t, ct);
    __syncwarp();
    // u x curl u at this lane's positions (unnormalised: the scale enters in s2)
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float ux = h1[e].x, uy = h1[e].y, uz = h2[e].x, wx = h2[e].y, wy = z[e].x, wz = z[e].y;
      const float pz = fmaf(ux, wy, -uy * wx);
      if (half == 0)
        pa[e] = pz;
      else
        pb[e] = pz;
      z[e] = make_float2(fmaf(uy, wz, -uz * wy), fmaf(uz, wx, -ux * wz));
    }
    warp_fft<N, 8, kFwd>(z, xs, t, ct);
    float2 X[4], Y[4];
    r2c_pair_unpack<N>(z, t, s2, X, Y);
    if (valid) {
      float2* dst = db + line * kt;
      store_du_line<N>(dst, X, t, kt, kd);
      store_du_line<N>(dst + ds, Y, t, kt, kd);
    }
    __syncwarp();
  }
  // z components of lines A and B in one forward FFT
  float2 z[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) z[e] = make_float2(pa[e], pb[e]);
  warp_fft<N, 8, kFwd>(z, xs, t, ct);
  float2 X[4], Y[4];
  r2c_pair_unpack<N>(z, t, s2, X, Y);
  if (ia < nlines) store_du_line<N>(db + 2 * ds + (nlines - 1 - ia) * kt, X, t, kt, kd);
  if (ia + 1 < nlines) store_du_line<N>(db + 2 * ds + (nlines - 2 - ia) * kt, Y, t, kt, kd);
}

// ------------------------------------------------------------------------------
// Half-axis line pass of the RHS with radix-16 line FFTs (N = 256): 16 lanes per line,
// two lines per warp side by side (lanes 0-15 line A, 16-31 line B), each lane holding
// 16 values, so a 256-point FFT is two in-register radix-16 stages around ONE shared-
// memory exchange (the 32-lane radix-8 schedule of line_cross2 needs two). Per line:
// three inverse two-for-one FFTs ((u_x, u_y), (u_z, curl_x), (curl_y, curl_z)), u x curl u
// in registers, one forward FFT of (p_x, p_y); the z products of lines A and B meet in
// one 32-lane FFT (radix 8, line_cross2's schedule) after one exchange between the half
// warps. Each input mode is loaded once: the mirrored half of the Hermitian extension
// arrives by shuffle from lane 16 - t of the same half warp.
// ct16: compact table of the radix-16 schedule (at line3_ct16_offset<N>()), ct8: that of
// the radix-8 schedule (line2_ct_offset<N>()).
// ------------------------------------------------------------------------------
template <int N>
__host__ __device__ constexpr int line3_ct16_offset() {
  return line2_ct_offset<N>() + Sched<N, 8>::ctlen();
}

template <int N>
struct Line3Cfg {
  static constexpr int T = 16;                 // lanes per line
  static constexpr int E = N / T;              // values per lane
  static constexpr int THREADS = 128;
  static constexpr int LPC = THREADS / T;      // lines per CTA (two per warp)
  static constexpr int XS = xpad_len<1>(N);    // exchange slots per line
  // bulk-copy staged form (dynamic shared memory): per warp two stages of two fields x
  // the warp's two (adjacent) rows, then the two exchange buffers; barriers in front
  static constexpr int ROW2 = 2 * (N / 2 + 1);              // float2 of two rows of one field
  static constexpr int WARP_F2 = 2 * 2 * ROW2 + 2 * XS;     // float2 per warp
  static constexpr int BAR_BYTES = 128;
  static constexpr int SMEM_STAGED = BAR_BYTES + (THREADS / 32) * WARP_F2 * 8;
};

// Z[n] = X_ext[n] + i Y_ext[n], n = t + 16 e (16-lane layout), from two half-spectrum
// lines; lanes load X[k], Y[k] for k < N/2 and the Nyquist entry, and take the mirrored
// values X[N - n] (n > N/2) from lane (16 - t) mod 16 of their half warp. numpy irfft
// semantics: Im X[0] and Im X[N/2] are ignored.
template <int N>
__device__ __forceinline__ void c2r_pair_load16(const float2* __restrict__ X, const float2* __restrict__ Y, int t,
                                                float2 (&z)[N / 16]) {
  constexpr int E = N / 16, H2 = E / 2;  // H2 slots cover k < N/2
  const int lane = threadIdx.x & 31;
  const int src = (lane & 16) | ((16 - t) & 15);
  float2 xa[H2], ya[H2];
#pragma unroll
  for (int e = 0; e < H2; ++e) {
    xa[e] = __ldg(X + t + 16 * e);
    ya[e] = __ldg(Y + t + 16 * e);
  }
  const float2 xn = __ldg(X + N / 2), yn = __ldg(Y + N / 2);
#pragma unroll
  for (int e = H2; e < E; ++e) {
    // partner of n = t + 16 e is N - n: slot E - 1 - e of lane 16 - t, or slot E - e of
    // lane 0 (t = 0; E - e = H2 is the Nyquist entry, loaded directly)
    const float2 gx = (t == 0 && e > H2) ? xa[(E - e) % H2] : xa[E - 1 - e];
    const float2 gy = (t == 0 && e > H2) ? ya[(E - e) % H2] : ya[E - 1 - e];
    float2 mx, my;
    mx.x = __shfl_sync(0xffffffffu, gx.x, src);
    mx.y = __shfl_sync(0xffffffffu, gx.y, src);
    my.x = __shfl_sync(0xffffffffu, gy.x, src);
    my.y = __shfl_sync(0xffffffffu, gy.y, src);
    if (e == H2 && t == 0) {  // n = N/2: real parts only
      mx = make_float2(xn.x, 0.f);
      my = make_float2(yn.x, 0.f);
    }
    z[e] = make_float2(mx.x + my.y, my.x - mx.y);  // conj X + i conj Y
  }
#pragma unroll
  for (int e = 0; e < H2; ++e) {
    float2 x = xa[e], y = ya[e];
    if (e == 0 && t == 0) {  // n = 0: real parts only
      x.y = 0.f;
      y.y = 0.f;
    }
    z[e] = make_float2(x.x - y.y, x.y + y.x);  // X + i Y
  }
}

// From Z = FFT(x + i y) in the 16-lane layout: X[k], Y[k] for k = t + 16 e, e < NE,
// scaled by s (s includes the 1/2); the partner Z[N - k] comes from lane (16 - t) mod 16.
template <int N, int NE>
__device__ __forceinline__ void r2c_pair_unpack16(const float2 (&z)[N / 16], int t, float s, float2 (&X)[NE],
                                                  float2 (&Y)[NE]) {
  constexpr int E = N / 16;
  const int lane = threadIdx.x & 31;
  const int src = (lane & 16) | ((16 - t) & 15);
#pragma unroll
  for (int e = 0; e < NE; ++e) {
    const float2 give = (t == 0) ? z[(E - e) % E] : z[E - 1 - e];
    float2 zm;
    zm.x = __shfl_sync(0xffffffffu, give.x, src);
    zm.y = __shfl_sync(0xffffffffu, give.y, src);
    const float2 zk = z[e];
    X[e] = make_float2(s * (zk.x + zm.x), s * (zk.y - zm.y));
    Y[e] = make_float2(s * (zk.y + zm.y), s * (zm.x - zk.x));
  }
}

// Z[n] = X_ext[n] + i Y_ext[n], n = t + 16 e, from two half-spectrum rows staged in
// shared memory (both halves of the Hermitian extension read directly).
template <int N>
__device__ __forceinline__ void c2r_pair_smem16(const float2* X, const float2* Y, int t, float2 (&z)[N / 16]) {
  constexpr int E = N / 16, H2 = E / 2;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int n = t + 16 * e;
    const int m = e < H2 ? n : N - n;  // N - n in [1, N/2] for n > N/2 ... and N/2 itself
    float2 x = X[m], y = Y[m];
    if ((e == 0 || e == H2) && t == 0) {  // n = 0 and n = N/2: real parts only
      x.y = 0.f;
      y.y = 0.f;
    }
    z[e] = e < H2 ? make_float2(x.x - y.y, x.y + y.x)   // X + i Y
                  : make_float2(x.x + y.y, y.x - x.y);  // conj X + i conj Y
  }
}

// 168 registers at 3 CTAs per SM. Measured at 256^3 (per launch): 133.7 us against
// line_cross2's 139.7; parking u_x + i u_y in shared memory to fit 4 CTAs per SM at 128
// registers (44 bytes of spills) took 135.4.
//
// STAGED (127.2 us): each warp's input rows come into shared memory by 1D bulk copies
// (the TMA engine, completion on an mbarrier), one field pair ahead of the FFTs: the
// loads leave the warps' critical path and take no registers. The warp's two lines are
// adjacent rows (2m, 2m + 1), so one 16-byte aligned copy of 2 (N/2 + 1) float2 moves
// both rows of a field. Needs nlines % 8 == 0 and SMEM_STAGED bytes of dynamic shared
// memory. Every wait is bounded: on timeout the warp sets kErrTimeout in *err, waits
// (bounded) for its copies in flight and returns. Measured and kept out: two line pairs
// per warp with the copies running on across them (131.0 us: spills), Blackwell's paired
// FP32 adds in the FFT butterflies (130.9 us: register pairs, spills).
//
// FEW (STAGED only): a launch of at most one CTA per SM, where latency counts and not
// occupancy: paired adds with the registers they need (212; ten 256^2 steps 492 -> 481 us).
template <int N, bool STAGED, bool FEW = false>
__global__ void __launch_bounds__(Line3Cfg<N>::THREADS, FEW ? 1 : 3)
line_cross3(const float2* __restrict__ w, long long fs, float2* __restrict__ du, long long ds, int kt, int kd,
            float s2, const float2* __restrict__ ct8, const float2* __restrict__ ct16, int nlines, int* err) {
  pdl_begin();
  static_assert(N == 256, "radix-16 line pass: N = 256");
  using C = Line3Cfg<N>;
  constexpr int E = C::E, H = N / 2 + 1;
  constexpr int NE = (N / 3 + 10 + 15) / 16;  // slots e with 16 e < kt (kt <= N/3 + 10)
  const int lane = threadIdx.x & 31, t = lane & 15, half = lane >> 4, warp = threadIdx.x >> 5;
  const float2* wb = w + (long long)blockIdx.y * 6 * fs;
  float2* db = du + (long long)blockIdx.y * 3 * ds;
  // lines from the last to the first (as in line_cross); idle lanes mirror a valid line
  const long long idx = (long long)blockIdx.x * C::LPC + 2 * warp + half;
  const bool valid = idx < nlines;
  const long long line = valid ? nlines - 1 - idx : nlines - 1;
  float2 h1[E], h2[E], z[E];
  float2* s_x;  // exchange buffers: two per warp
  if constexpr (STAGED) {
    extern __shared__ __align__(128) unsigned char l3_dyn[];
    uint64_t* bar = reinterpret_cast<uint64_t*>(l3_dyn) + 2 * warp;
    float2* wsm = reinterpret_cast<float2*>(l3_dyn + C::BAR_BYTES) + warp * C::WARP_F2;
    float2* stg0 = wsm;
    float2* stg1 = wsm + 2 * C::ROW2;
    s_x = wsm + 4 * C::ROW2 - 2 * warp * C::XS;  // so that s_x + 2 warp XS is this warp's pair
    // rows (2m, 2m + 1) of the warp: line B (half 1) = 2m, line A (half 0) = 2m + 1
    const long long row0 = nlines - 2 - ((long long)blockIdx.x * C::LPC + 2 * warp);
    const float2* rows = wb + row0 * H;
    constexpr unsigned kPairBytes = 2u * C::ROW2 * sizeof(float2);
    if (lane == 0) {
      mbar_init(&bar[0], 1);
      mbar_init(&bar[1], 1);
      mbar_init_fence();
    }
    __syncwarp();
    if (lane == 0) {
      mbar_arrive_expect_tx(&bar[0], kPairBytes);
      bulk_load(stg0, rows, kPairBytes / 2, &bar[0]);
      bulk_load(stg0 + C::ROW2, rows + fs, kPairBytes / 2, &bar[0]);
      mbar_arrive_expect_tx(&bar[1], kPairBytes);
      bulk_load(stg1, rows + 2 * fs, kPairBytes / 2, &bar[1]);
      bulk_load(stg1 + C::ROW2, rows + 3 * fs, kPairBytes / 2, &bar[1]);
    }
    const int rsel = half ? 0 : H;  // this half's row inside a staged pair of rows
    float2* xs = s_x + (2 * warp + half) * C::XS;
    // bounded waits; on a timeout every copy this warp issued must land before it leaves
    auto give_up = [&](int pending0, int pending1) {
      if (lane == 0) atomicOr(err, kErrTimeout);
      if (pending0 >= 0) mbar_wait(&bar[0], (unsigned)pending0);
      if (pending1 >= 0) mbar_wait(&bar[1], (unsigned)pending1);
    };
    if (__any_sync(0xffffffffu, !mbar_wait(&bar[0], 0))) {
      give_up(0, 0);
      return;
    }
    c2r_pair_smem16<N>(stg0 + rsel, stg0 + C::ROW2 + rsel, t, z);  // u_x + i u_y
    __syncwarp();  // stage 0 read by every lane
    if (lane == 0) {
      fence_proxy_async_smem();
      mbar_arrive_expect_tx(&bar[0], kPairBytes);
      bulk_load(stg0, rows + 4 * fs, kPairBytes / 2, &bar[0]);
      bulk_load(stg0 + C::ROW2, rows + 5 * fs, kPairBytes / 2, &bar[0]);
    }
    block_fft<N, E, kInv, 1, kSyncWarp, true, FEW>(z, xs, t, ct16, 0);
#pragma unroll
    for (int e = 0; e < E; ++e) h1[e] = z[e];
    __syncwarp();
    if (__any_sync(0xffffffffu, !mbar_wait(&bar[1], 0))) {
      give_up(1, 0);
      return;
    }
    c2r_pair_smem16<N>(stg1 + rsel, stg1 + C::ROW2 + rsel, t, z);  // u_z + i curl_x
    block_fft<N, E, kInv, 1, kSyncWarp, true, FEW>(z, xs, t, ct16, 0);
#pragma unroll
    for (int e = 0; e < E; ++e) h2[e] = z[e];
    __syncwarp();
    if (__any_sync(0xffffffffu, !mbar_wait(&bar[0], 1))) {
      give_up(1, -1);
      return;
    }
    c2r_pair_smem16<N>(stg0 + rsel, stg0 + C::ROW2 + rsel, t, z);  // curl_y + i curl_z
    block_fft<N, E, kInv, 1, kSyncWarp, true, FEW>(z, xs, t, ct16, 0);
    __syncwarp();
  } else {
    __shared__ float2 s_xs[C::LPC * C::XS];
    s_x = s_xs;
    float2* xs = s_x + (2 * warp + half) * C::XS;
    const float2* src = wb + line * H;
    c2r_pair_load16<N>(src, src + fs, t, z);  // u_x + i u_y
    block_fft<N, E, kInv, 1, kSyncWarp, true, FEW>(z, xs, t, ct16, 0);
#pragma unroll
    for (int e = 0; e < E; ++e) h1[e] = z[e];
    __syncwarp();
    c2r_pair_load16<N>(src + 2 * fs, src + 3 * fs, t, z);  // u_z + i curl_x
    block_fft<N, E, kInv, 1, kSyncWarp, true, FEW>(z, xs, t, ct16, 0);
#pragma unroll
    for (int e = 0; e < E; ++e) h2[e] = z[e];
    __syncwarp();
    c2r_pair_load16<N>(src + 4 * fs, src + 5 * fs, t, z);  // curl_y + i curl_z
    block_fft<N, E, kInv, 1, kSyncWarp, true, FEW>(z, xs, t, ct16, 0);
    __syncwarp();
  }
  float2* xs = s_x + (2 * warp + half) * C::XS;
  // u x curl u at this lane's positions (unnormalised: the scale enters in s2)
  float pz[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const float ux = h1[e].x, uy = h1[e].y, uz = h2[e].x, wx = h2[e].y, wy = z[e].x, wz = z[e].y;
    pz[e] = fmaf(ux, wy, -uy * wx);
    z[e] = make_float2(fmaf(uy, wz, -uz * wy), fmaf(uz, wx, -ux * wz));
  }
  block_fft<N, E, kFwd, 1, kSyncWarp, true, FEW>(z, xs, t, ct16, 0);
  {
    float2 X[NE], Y[NE];
    r2c_pair_unpack16<N, NE>(z, t, s2, X, Y);
    if (valid) {
      float2* dst = db + line * kt;
#pragma unroll
      for (int e = 0; e < NE; ++e) {
        const int k = t + 16 * e;
        if (k < kt) {
          dst[k] = k <= kd ? X[e] : make_float2(0.f, 0.f);
          dst[ds + k] = k <= kd ? Y[e] : make_float2(0.f, 0.f);
        }
      }
    }
  }
  __syncwarp();
  // z products of lines A (lanes 0-15) and B (16-31) as one 32-lane FFT of pz_A + i pz_B:
  // lane L = t + 16 h' holds n = L + 32 e' (e = 2 e' + h' in the 16-lane layout); half A
  // keeps pz_A of even e and receives pz_B of even e, half B the odd ones
  float2 y[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const float give = half ? pz[2 * q] : pz[2 * q + 1];
    const float got = __shfl_xor_sync(0xffffffffu, give, 16);
    y[q] = half ? make_float2(got, pz[2 * q + 1]) : make_float2(pz[2 * q], got);
  }
  float2* xw = s_x + 2 * warp * C::XS;  // the warp's first exchange buffer
  warp_fft<N, 8, kFwd>(y, xw, lane, ct8);
  float2 X[4], Y[4];
  r2c_pair_unpack<N>(y, lane, s2, X, Y);
  // line A = nlines - 1 - idx_A, line B = line A - 1 (idx_B = idx_A + 1)
  const long long idx_a = (long long)blockIdx.x * C::LPC + 2 * warp;
  if (idx_a < nlines) store_du_line<N>(db + 2 * ds + (nlines - 1 - idx_a) * kt, X, lane, kt, kd);
  if (idx_a + 1 < nlines) store_du_line<N>(db + 2 * ds + (nlines - 2 - idx_a) * kt, Y, lane, kt, kd);
}

// ------------------------------------------------------------------------------
// Half-axis c2r of 3 fields to physical space (irfftn's last axis): out[c][line][0..N).
// ------------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(LineCfg<N>::THREADS)
line_c2r(const float2* __restrict__ w, long long fs, float* __restrict__ out, long long os,
         float scale, const float2* __restrict__ twN, int nlines) {
  pdl_begin();
  using C = LineCfg<N>;
  constexpr int M = C::M, H = N / 2 + 1, E = C::E, T = C::T, LPC = C::LPC;
  __shared__ float2 s_x[LPC * C::XS];
  const int batch = blockIdx.y;
  const int q = threadIdx.x / T, t = threadIdx.x % T;
  const long long line_raw = (long long)blockIdx.x * LPC + q;
  const bool valid = line_raw < nlines;
  const long long line = valid ? line_raw : nlines - 1;
  float2* xs = s_x + q * C::XS;
#pragma unroll 1
  for (int f = 0; f < 3; ++f) {
    const float2* src = w + (long long)batch * 3 * fs + f * fs + line * H;
    float2 v[E];
    c2r_load_pack<M, E>(src, t, v, twN, scale);
    warp_fft<M, E, kInv>(v, xs, t, twN + N);
    if (valid) {
      float2* dst = reinterpret_cast<float2*>(out + (long long)batch * 3 * os + f * os + line * N);
#pragma unroll
      for (int e = 0; e < E; ++e) dst[t + T * e] = v[e];
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------
// Half-axis r2c of 3 physical fields: in[c][line][0..N) -> w[c][line][0..H).
// ------------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(LineCfg<N>::THREADS)
line_r2c(const float* __restrict__ in, long long is, float2* __restrict__ w, long long fs,
         const float2* __restrict__ twN, int nlines) {
  pdl_begin();
  using C = LineCfg<N>;
  constexpr int M = C::M, H = N / 2 + 1, E = C::E, T = C::T, LPC = C::LPC;
  __shared__ float2 s_x[LPC * C::XS];
  const int batch = blockIdx.y;
  const int q = threadIdx.x / T, t = threadIdx.x % T;
  const long long line_raw = (long long)blockIdx.x * LPC + q;
  const bool valid = line_raw < nlines;
  const long long line = valid ? line_raw : nlines - 1;
  float2* xs = s_x + q * C::XS;
#pragma unroll 1
  for (int f = 0; f < 3; ++f) {
    const float2* src = reinterpret_cast<const float2*>(in + (long long)batch * 3 * is + f * is + line * N);
    float2 v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = __ldg(src + t + T * e);
    warp_fft<M, E, kFwd>(v, xs, t, twN + N);
    float2 X[E];
    r2c_unpack_regs<M, E>(v, t, twN, X);
    if (valid) {
      float2* dst = w + (long long)batch * 3 * fs + f * fs + line * H;
#pragma unroll
      for (int e = 0; e < E; ++e) dst[t + T * e] = X[e];
      if (t == 0) dst[M] = make_float2(v[0].x - v[0].y, 0.f);  // X[M] = Re Z0 - Im Z0
    }
    __syncwarp();
  }
}

// ------------------------------------------------------------------------------
// x-axis forward pass without epilogue: w[c][x][mid][kh] -> uh[c][kx][mid][kh].
// ------------------------------------------------------------------------------
template <int N, int DIM>
__global__ void __launch_bounds__(TW * Fft<N>::T)
kx_fwd_plain(const float2* __restrict__ w, long long fs, float2* __restrict__ uh, long long cs,
             const float2* __restrict__ tw) {
  pdl_begin();
  constexpr int E = Fft<N>::E, T = Fft<N>::T, H = N / 2 + 1;
  constexpr int NMID = DIM == 3 ? N : 1;
  constexpr int MC = NMID * H;
  __shared__ float2 sm[xpad_len<TW>(N) * TW];
  const int p = threadIdx.x % TW, t = threadIdx.x / TW;
  const int m = blockIdx.x * TW + p;
  const bool ok = m < MC;
  const long long bw = (long long)blockIdx.y * 3 * fs, bu = (long long)blockIdx.y * 3 * cs;
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
    float2 v[E];
#pragma unroll
    for (int e = 0; e < E; ++e)
      v[e] = ok ? w[bw + c * fs + (long long)(t + T * e) * MC + m] : make_float2(0.f, 0.f);
    block_fft<N, E, kFwd, TW>(v, sm + p, t, tw, 1);
    if (ok) {
#pragma unroll
      for (int e = 0; e < E; ++e) uh[bu + c * cs + (long long)(t + T * e) * MC + m] = v[e];
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------
// Low-wavenumber band helpers (few hundred modes; one CTA per trajectory).
// band: 0 < |k|^2 <= kf^2 (init_fields.py:167-188). weights: half-axis multiplicity.
// ------------------------------------------------------------------------------
template <int DIM>
__device__ __forceinline__ bool band_mode(int i, int N, int kf, long long& idx, int& wgt) {
  // enumerate kx in [-kf, kf], (3D) km in [-kf, kf], kh in [0, kf]
  const int n1 = 2 * kf + 1, nh = kf + 1;
  const int kh = i % nh;
  const int r = i / nh;
  const int km = DIM == 3 ? (r % n1) - kf : 0;
  const int kx = DIM == 3 ? (r / n1) - kf : r - kf;
  const int k2 = kx * kx + km * km + kh * kh;
  if (k2 == 0 || k2 > kf * kf) return false;
  const int H = N / 2 + 1;
  const int xi = kx < 0 ? kx + N : kx;
  const int mi = km < 0 ? km + N : km;
  idx = DIM == 3 ? ((long long)xi * N + mi) * H + kh : (long long)xi * H + kh;
  wgt = (kh == 0 || kh == N / 2) ? 1 : 2;
  return true;
}

template <int DIM>
__device__ __forceinline__ int band_count(int kf) {
  return DIM == 3 ? (2 * kf + 1) * (2 * kf + 1) * (kf + 1) : (2 * kf + 1) * (kf + 1);
}

// Sum of v over the lanes of a warp, in every lane. A block smaller than a warp (its THREADS
// a power of two) has no other lanes: neither named in the mask nor read.
template <int THREADS>
__device__ __forceinline__ double lanes_sum(double v) {
  constexpr int L = THREADS < 32 ? THREADS : 32;
  static_assert((L & (L - 1)) == 0 && THREADS % L == 0, "whole warps, or a power of two below one");
  constexpr unsigned mask = L == 32 ? 0xffffffffu : (1u << L % 32) - 1u;
#pragma unroll
  for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}

// Constant-power band forcing coefficient eps / (2 E_f + tiny) of a stage field
// (extension), computed by all THREADS threads of one block; thread 0 stores it.
template <int DIM, int THREADS>
__device__ __forceinline__ void band_coefficient(const float2* __restrict__ ub, long long cs, int N, int kf,
                                                 double inv_n2d, double eps_inj, double tiny, double* out) {
  __shared__ double red_band[32];
  double lo = 0.0;
  const int nb = band_count<DIM>(kf);
  for (int i = threadIdx.x; i < nb; i += blockDim.x) {
    long long idx;
    int wg;
    if (!band_mode<DIM>(i, N, kf, idx, wg)) continue;
    for (int c = 0; c < 3; ++c) {
      const float2 v = ub[c * cs + idx];
      lo += wg * ((double)v.x * v.x + (double)v.y * v.y);
    }
  }
  lo = lanes_sum<THREADS>(lo);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red_band[wid] = lo;
  __syncthreads();
  if (threadIdx.x == 0) {
    double L = 0.0;
    for (int i = 0; i < (THREADS + 31) / 32; ++i) L += red_band[i];
    *out = eps_inj / (2.0 * (0.5 * L * inv_n2d) + tiny);
  }
}

// a0 / b0 of the classical RK4 tableau (1/6 over 1/2): stage 1 rebuilds the stage-0
// accumulator term a0 dt k1 from its input us = u0 + b0 dt k1, so stage 0 stores no
// accumulator and stage 1 reads none (2 spectra less traffic per step; the rebuilt
// term carries one FP32 rounding of u0, as storing it did).
constexpr float kAccFromStage0 = 1.0f / 3.0f;

// RK4 stage combination and extension terms for the elementwise update.
struct EpiParams {
  float a_dt;        // a_rk4[rk] * dt
  float b_dt;        // b_rk4[rk] * dt (rk < 3)
  float nu;
  float drag;        // linear drag coefficient (extension, 0 = off)
  float kolm_amp;    // Kolmogorov forcing: du_x(kx=0, khalf=kolm_k) += -i amp N^2 / 2
  int kolm_k;        //   (2D extension, kolm_k = 0 = off)
  int band_kf2;      // constant-power band forcing 0 < |k|^2 <= band_kf2 (0 = off)
  int rk;            // 0..3, or -1: write the right-hand side du itself to `out`
  float if_h;        // > 0: integrating-factor RK4 with step if_h (viscous term exact)
  float dt = 0.f;    // the step (used with lin)
  int lin = 0;       // explicit RK4 step whose forcing lies inside the stage region: modes
                     // outside it take the closed form of their linear decay (k_rk_update)
  int band_rk = 0;   // explicit RK4 step combined inside the band pass (XLin, BandRk)
};

// Float-float (hi + lo) accumulator: error-free FP32 additions (Knuth's TwoSum, then
// Dekker's fast renormalisation) carry ~48 significant bits without FP64 arithmetic,
// which is scarce on this GPU. Values are non-negative energies here.
struct Ff {
  float hi, lo;
};
__device__ __forceinline__ Ff ff_add(Ff a, float b) {
  const float s = a.hi + b;
  const float bb = s - a.hi;
  const float e = (a.hi - (s - bb)) + (b - bb);
  const float lo = a.lo + e;
  const float h = s + lo;
  return Ff{h, lo - (h - s)};
}
__device__ __forceinline__ Ff ff_add(Ff a, Ff b) {
  const float s = a.hi + b.hi;
  const float bb = s - a.hi;
  const float e = (a.hi - (s - bb)) + (b.hi - bb) + (a.lo + b.lo);
  const float h = s + e;
  return Ff{h, e - (h - s)};
}

// FP64 block reduction into partial[block]; all threads must call.
__device__ __forceinline__ void block_sum_store(double v, double* partial, int block) {
  __shared__ double red[32];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  if (wid == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    v = lane < nw ? red[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) partial[block] = v;
  }
}

// Block reduction of float-float partials into partial[block] (FP64): warps combine in
// float-float by shuffles, the per-warp sums in FP64; all threads must call.
__device__ __forceinline__ void block_sum_store_ff(Ff v, double* partial, int block) {
  __shared__ double red_ff[32];
  for (int o = 16; o > 0; o >>= 1) {
    Ff w;
    w.hi = __shfl_xor_sync(0xffffffffu, v.hi, o);
    w.lo = __shfl_xor_sync(0xffffffffu, v.lo, o);
    v = ff_add(v, w);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red_ff[wid] = (double)v.hi + (double)v.lo;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < (int)((blockDim.x + 31) >> 5); ++i) t += red_ff[i];
    partial[block] = t;
  }
}

// rk_core_r: the right-hand side of one mode from its projected nonlinear term r (zero
// outside the kept band) and the stage combination (ik2 = |k|^2 as an integer).
template <int N, int DIM, bool VIF = false>
__device__ __forceinline__ float2 rk_core_r(int kxi, int mid, int kh, int ik2, int c, float2 r, float2 sv, float2 a0,
                                            float2 z0, const EpiParams& prm, float fscale, float2& nv) {
  const float kk2 = (float)ik2;
  const float nu = prm.nu;
  const bool vif = VIF && prm.rk >= 0;
  if (!vif) {
    r.x -= nu * kk2 * sv.x;
    r.y -= nu * kk2 * sv.y;
  }
  if (prm.drag != 0.f) {
    r.x -= prm.drag * sv.x;
    r.y -= prm.drag * sv.y;
  }
  if (c == 0 && prm.kolm_k > 0 && kxi == 0 && mid == 0 && kh == prm.kolm_k) r.y += -0.5f * prm.kolm_amp * (float)N * (float)N;
  if (prm.band_kf2 > 0 && ik2 > 0 && ik2 <= prm.band_kf2) {
    r.x += fscale * sv.x;
    r.y += fscale * sv.y;
  }
  if (prm.rk < 0) {
    nv = r;
    return r;
  }
  if (vif) {
    // Integrating-factor RK4 (Lawson) with eh = exp(-nu k^2 h / 2), e1 = eh^2 and r the
    // right-hand side without viscosity:
    //   rk 0: out = eh (u0 + h/2 r)                         (us = u0; no accumulator)
    //   rk 1: out = eh u0 + h/2 r,  acc = 2/3 e1 u0 + eh/3 us + h/3 eh r
    //         (h/6 e1 k1 rebuilt from us = eh (u0 + h/2 k1), as in the explicit form)
    //   rk 2: out = e1 u0 + h eh r, acc += h/3 eh r
    //   rk 3: fin = acc + h/6 r
    const float eh = expf(-0.5f * prm.if_h * nu * kk2);
    const float e1 = eh * eh;
    if (prm.rk == 0) {
      nv = make_float2(eh * fmaf(prm.b_dt, r.x, sv.x), eh * fmaf(prm.b_dt, r.y, sv.y));
      return r;
    }
    if (prm.rk == 1) {
      nv = make_float2(fmaf(eh, z0.x, prm.b_dt * r.x), fmaf(eh, z0.y, prm.b_dt * r.y));
      const float c0 = (2.0f / 3.0f) * e1, c1 = eh * (1.0f / 3.0f), c2 = prm.a_dt * eh;
      return make_float2(fmaf(c2, r.x, fmaf(c1, sv.x, c0 * z0.x)), fmaf(c2, r.y, fmaf(c1, sv.y, c0 * z0.y)));
    }
    if (prm.rk == 2) {
      const float bh = prm.b_dt * eh, ah = prm.a_dt * eh;
      nv = make_float2(fmaf(bh, r.x, e1 * z0.x), fmaf(bh, r.y, e1 * z0.y));
      return make_float2(fmaf(ah, r.x, a0.x), fmaf(ah, r.y, a0.y));
    }
    nv = make_float2(fmaf(prm.a_dt, r.x, a0.x), fmaf(prm.a_dt, r.y, a0.y));
    return nv;
  }
  if (prm.rk == 0) {  // the accumulator is not stored: stage 1 rebuilds it from us and u0
    nv = make_float2(fmaf(prm.b_dt, r.x, sv.x), fmaf(prm.b_dt, r.y, sv.y));
    return r;
  }
  if (prm.rk == 1) {
    // acc = u0 + a0 dt k1 + a1 dt k2 with a0 dt k1 = (a0 / b0) (us - u0), us = u0 + b0 dt k1
    nv = make_float2(fmaf(prm.b_dt, r.x, z0.x), fmaf(prm.b_dt, r.y, z0.y));
    return make_float2(fmaf(prm.a_dt, r.x, fmaf(sv.x - z0.x, kAccFromStage0, z0.x)),
                       fmaf(prm.a_dt, r.y, fmaf(sv.y - z0.y, kAccFromStage0, z0.y)));
  }
  if (prm.rk < 3) {
    nv = make_float2(fmaf(prm.b_dt, r.x, z0.x), fmaf(prm.b_dt, r.y, z0.y));
    return make_float2(fmaf(prm.a_dt, r.x, a0.x), fmaf(prm.a_dt, r.y, a0.y));
  }
  nv = make_float2(fmaf(prm.a_dt, r.x, a0.x), fmaf(prm.a_dt, r.y, a0.y));
  return nv;
}

// Band-fused RK step (XLin): the band pass combines the stages itself. P holds the
// step's initial state on the band (written at rk 0) and acc the accumulator, both in
// P's compact layout; S is updated in place on the band.
struct BandRk {
  float2* S;
  float2* acc;
  long long cs;
  EpiParams prm;
  const double* band_scale;
  const float* nu_b;
  int* err;
};

// ------------------------------------------------------------------------------
// x-axis forward pass of the nonlinear term on the dealiased band only
// (spectral_solver.py:55-58: du *= dealias; du -= (sum du.k/k^2) k). CTA = (half-axis
// tile inside kt, middle-axis row inside the band). Output P keeps only the kept
// modes: P[c][kx + kd][kmid + kd][kh] (3D), P[c][kx + kd][kh] (2D), kh < kt, with
// zeros for kh > kd.
// ------------------------------------------------------------------------------
// One tile of kx_fwd_band: d[c][e] = DU component c at x row t + T e of column kh of
// middle row kmb (band index); x forward FFT, dealias mask, Leray projection into P.
// PK: paired adds (the bulk-load variant; with direct loads the 128^3 pass took 14.0 us, not 13.5).
template <int N, int DIM, bool FUSED = false, int XW = TW, bool PK = false>
__device__ __forceinline__ void kx_fwd_band_tile(float2 (&d)[3][Fft<N>::E], int t, int kh, int kmb, int kd, int kt,
                                                 float2* sm, float2* __restrict__ P, long long pcs, long long bp,
                                                 const float2* __restrict__ tw, const BandRk* br = nullptr,
                                                 int batch = 0) {
  constexpr int E = Fft<N>::E, T = Fft<N>::T, H = N / 2 + 1;
  constexpr int NMID = DIM == 3 ? N : 1;
  const int nb = 2 * kd + 1;
  const int km = DIM == 3 ? kmb - kd : 0;
  const int mid = km < 0 ? km + N : km;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    block_fft<N, E, kFwd, XW, kSyncCta, false, PK>(d[c], sm, t, tw, 1);
    __syncthreads();
  }
  // (kt can exceed the half axis only at N = 8: those columns hold no mode of S)
  const bool live = !FUSED || kh < H;
  bool inb[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int kx = kfull(t + T * e, N);
    inb[e] = live && (unsigned)(kx + kd) <= 2u * (unsigned)kd;  // |kx| <= kd
    if (!inb[e]) continue;
    float k0, k1, k2;
    kvec<DIM>(kx, km, kh, k0, k1, k2);
    const bool keep = kh <= kd;
    const int ik2 = kx * kx + km * km + kh * kh;
    const float inv = 1.0f / (ik2 == 0 ? 1.0f : (float)ik2);
    const float2 v0 = keep ? d[0][e] : make_float2(0.f, 0.f);
    const float2 v1 = keep ? d[1][e] : make_float2(0.f, 0.f);
    const float2 v2 = keep ? d[2][e] : make_float2(0.f, 0.f);
    const float pr = (v0.x * k0 + v1.x * k1 + v2.x * k2) * inv;
    const float pi_ = (v0.y * k0 + v1.y * k1 + v2.y * k2) * inv;
    d[0][e] = make_float2(v0.x - pr * k0, v0.y - pi_ * k0);
    d[1][e] = make_float2(v1.x - pr * k1, v1.y - pi_ * k1);
    d[2][e] = make_float2(v2.x - pr * k2, v2.y - pi_ * k2);
    if constexpr (!FUSED) {
      const long long o = bp + ((long long)(kx + kd) * (DIM == 3 ? nb : 1) + kmb) * kt + kh;
#pragma unroll
      for (int c = 0; c < 3; ++c) P[o + c * pcs] = d[c][e];
    }
  }
  if constexpr (FUSED) {
    // the stage combination of rk_core on the band modes, in place in S; P holds the
    // step's initial band values (written at rk 0), br->acc the accumulator. Software
    // pipelined by one mode: the next mode's operands are loaded before this mode's
    // results are stored (a load may not pass an earlier store to the same arrays, so
    // load/store pairs in program order would each wait on memory).
    EpiParams prm = br->prm;
    prm.nu = br->nu_b[batch];
    const float fscale = prm.band_kf2 > 0 ? (float)br->band_scale[batch] : 0.f;
    float2* sb = br->S + (long long)batch * 3 * br->cs + (long long)mid * H + kh;
    auto sofs = [&](int e) { return (long long)(t + T * e) * NMID * H; };
    auto pofs = [&](int e) {
      return bp + ((long long)(kfull(t + T * e, N) + kd) * (DIM == 3 ? nb : 1) + kmb) * kt + kh;
    };
    float2 sv[3], z0[3], a0[3], sv1[3], z01[3], a01[3];
    auto load = [&](int e, float2(&s_)[3], float2(&z_)[3], float2(&a_)[3]) {
      const long long so = sofs(e), o = pofs(e);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        s_[c] = sb[so + c * br->cs];
        z_[c] = (prm.rk == 1 || prm.rk == 2) ? P[o + c * pcs] : make_float2(0.f, 0.f);
        a_[c] = prm.rk >= 2 ? br->acc[o + c * pcs] : make_float2(0.f, 0.f);
      }
    };
    if (inb[0]) load(0, sv, z0, a0);
    bool bad = false;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (e + 1 < E && inb[e + 1]) load(e + 1, sv1, z01, a01);
      if (inb[e]) {
        const int row = t + T * e;
        const int kx = kfull(row, N);
        const long long so = sofs(e), o = pofs(e);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          float2 nv;
          const float2 ra = rk_core_r<N, DIM, false>(row, mid, kh, kx * kx + km * km + kh * kh, c, d[c][e], sv[c],
                                                     a0[c], z0[c], prm, fscale, nv);
          if (prm.rk == 0) P[o + c * pcs] = sv[c];
          if (prm.rk == 1 || prm.rk == 2) br->acc[o + c * pcs] = ra;
          sb[so + c * br->cs] = nv;
          if (prm.rk == 3) bad |= !isfinite(nv.x + nv.y);
        }
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        sv[c] = sv1[c];
        z0[c] = z01[c];
        a0[c] = a01[c];
      }
    }
    if (bad) atomicOr(br->err, kErrNonFinite);
  }
}

// FUSED: the band-fused RK step (BandRk; the constant-power coefficient then comes from
// the stage's x inverse, band_kf = 0 here).
template <int N, int DIM, bool FUSED = false, int XW = TW>
__global__ void __launch_bounds__(XW * Fft<N>::T)
kx_fwd_band(const float2* __restrict__ du, long long dcs, int kt, int kd, float2* __restrict__ P, long long pcs,
            const float2* __restrict__ tw, const float2* __restrict__ us, long long cs, int band_kf,
            double inv_n2d, double eps_inj, double* __restrict__ band_scale, const BandRk br = BandRk{}) {
  pdl_begin();
  constexpr int E = Fft<N>::E, T = Fft<N>::T;
  constexpr int NMID = DIM == 3 ? N : 1;
  __shared__ float2 sm[xpad_len<XW>(N) * XW];
  const int p = threadIdx.x % XW, t = threadIdx.x / XW;
  const int kmb = DIM == 3 ? (int)blockIdx.y : 0;
  const int km = DIM == 3 ? kmb - kd : 0;
  const int mid = km < 0 ? km + N : km;
  const int kh = blockIdx.x * XW + p;  // < kt (kt is a multiple of TW, hence of XW)
  const int batch = blockIdx.z;
  const long long bd = (long long)batch * 3 * dcs, bp = (long long)batch * 3 * pcs;
  if (band_kf > 0 && blockIdx.x == 0 && blockIdx.y == 0)
    band_coefficient<DIM, XW * T>(us + (long long)batch * 3 * cs, cs, N, band_kf, inv_n2d, eps_inj, 1e-30,
                                  band_scale + batch);
  float2 d[3][E];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int e = 0; e < E; ++e) d[c][e] = du[bd + c * dcs + ((long long)(t + T * e) * NMID + mid) * kt + kh];
  kx_fwd_band_tile<N, DIM, FUSED, XW>(d, t, kh, kmb, kd, kt, sm + p, P, pcs, bp, tw, &br, batch);
}

// Persistent 3D variant of kx_fwd_band: tiles (column tile, band row kmb) are walked
// blockIdx.x, + gridDim.x, ...; the next tile's DU block (TW columns x N x rows x 3
// components at middle row `mid`) arrives by one 4D bulk tensor load while the current
// one is transformed. dmap: DU as (kt, N mid, N x, 3 * batch), box (TW, 1, min(N, 256), 3).
template <int N, bool FUSED = false>
__global__ void __launch_bounds__(TW * Fft<N>::T, TW * Fft<N>::T >= 512 ? 1 : 2)
kx_fwd_band_tma(const __grid_constant__ CUtensorMap dmap, int kt, int kd, float2* __restrict__ P, long long pcs,
                const float2* __restrict__ tw, const float2* __restrict__ us, long long cs, int band_kf,
                double inv_n2d, double eps_inj, double* __restrict__ band_scale, int* __restrict__ err,
                const __grid_constant__ BandRk br) {
  pdl_begin();
  using K = KxTma<N>;
  constexpr int E = Fft<N>::E, T = Fft<N>::T;
  extern __shared__ __align__(128) float2 s_dyn[];
  float2* stage = s_dyn;
  float2* sm = s_dyn + K::STAGE;
  __shared__ uint64_t bar;
  const int p = threadIdx.x % TW, t = threadIdx.x / TW;
  const int batch = blockIdx.y;
  const int ntx = kt / TW, nb = 2 * kd + 1, ntiles = ntx * nb;
  if (band_kf > 0 && blockIdx.x == 0)
    band_coefficient<3, TW * T>(us + (long long)batch * 3 * cs, cs, N, band_kf, inv_n2d, eps_inj, 1e-30, band_scale + batch);
  if (threadIdx.x == 0) {
    mbar_init(&bar, 1);
    mbar_init_fence();
  }
  __syncthreads();
  auto issue = [&](int tile) {
    const int kmb = tile / ntx, x0 = (tile % ntx) * TW;
    const int km = kmb - kd, mid = km < 0 ? km + N : km;
    mbar_arrive_expect_tx(&bar, K::BYTES);
#pragma unroll
    for (int l = 0; l < K::LOADS; ++l)
      tma_load_4d(stage + l * 3 * K::NY * TW, &dmap, &bar, x0, mid, l * K::NY, 3 * batch);
  };
  int tile = blockIdx.x;
  if (threadIdx.x == 0 && tile < ntiles) issue(tile);
  unsigned parity = 0;
  for (; tile < ntiles; tile += gridDim.x) {
    const bool got = threadIdx.x < 32 ? mbar_wait(&bar, parity) : true;  // as in kx_inv_tma
    if (__syncthreads_or(!got)) {
      if (threadIdx.x == 0) atomicOr(err, kErrTimeout);
      mbar_wait(&bar, parity);
      return;
    }
    if (threadIdx.x >= 32) mbar_wait(&bar, parity);
    parity ^= 1u;
    float2 d[3][E];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int row = t + T * e;
        d[c][e] = stage[(((row / K::NY) * 3 + c) * K::NY + row % K::NY) * TW + p];
      }
    __syncthreads();
    const int next = tile + gridDim.x;
    if (threadIdx.x == 0 && next < ntiles) {
      fence_proxy_async_smem();
      issue(next);
    }
    kx_fwd_band_tile<N, 3, FUSED, TW, true>(d, t, (tile % ntx) * TW + p, tile / ntx, kd, kt, sm + p, P, pcs,
                                  (long long)batch * 3 * pcs, tw, &br, batch);
  }
}

// ------------------------------------------------------------------------------
// Elementwise linear terms + RK4 stage combination (spectral_solver.py:59, :74-80),
// two complex values (one float4) per thread over all 3 components:
//   du = P(k) (kept band, else 0) - nu k^2 us [- drag us + forcing terms]
//   rk 0   : out <- us + b dt du                               (us = u0; no acc)
//   rk 1   : acc <- u0 + (a0/b0)(us - u0) + a dt du, out <- u0 + b dt du
//   rk 2   : acc += a dt du,       out <- u0 + b dt du         (us aliases out)
//   rk 3   : fin <- acc + a dt du
//   rk -1  : out <- du (the reference's rhs_fn)
// Every thread loads all its operands before storing (us/out and acc alias).
// VIF: the integrating-factor form (a separate instantiation, so the reference's explicit
// form keeps its own code).
// ------------------------------------------------------------------------------
// rk_core: one mode given its indices (kxi, mid, kh: storage indices on the x, middle
// and half axes; kx, km: their signed wavenumbers); rk_elem: by flat index i.
template <int N, int DIM, bool VIF = false>
__device__ __forceinline__ float2 rk_core(int kxi, int mid, int kh, int kx, int km, int c, float2 sv, float2 a0,
                                          float2 z0, const float2* __restrict__ P, long long pcs, int kt, int kd,
                                          const EpiParams& prm, float fscale, float2& nv) {
  const int ik2 = kx * kx + km * km + kh * kh;
  float2 r = make_float2(0.f, 0.f);
  // band rows as unsigned offsets: in the band iff 0 <= k + kd <= 2 kd on every axis
  const unsigned nb = 2u * (unsigned)kd + 1u;
  const unsigned bx = (unsigned)(kx + kd);
  const unsigned bm = DIM == 3 ? (unsigned)(km + kd) : 0u;
  if (bx < nb && bm < nb && (unsigned)kh <= (unsigned)kd) {
    const long long row = DIM == 3 ? (long long)bx * nb + bm : (long long)bx;
    r = __ldg(P + c * pcs + row * kt + kh);
  }
  return rk_core_r<N, DIM, VIF>(kxi, mid, kh, ik2, c, r, sv, a0, z0, prm, fscale, nv);
}

template <int N, int DIM, bool VIF = false>
__device__ __forceinline__ float2 rk_elem(unsigned i, int c, float2 sv, float2 a0, float2 z0,
                                          const float2* __restrict__ P, long long pcs, int kt, int kd,
                                          const EpiParams& prm, float fscale, float2& nv) {
  // i < 3 N^2 (N/2+1) < 2^31 for N <= 512: 32-bit division by compile-time constants
  constexpr unsigned H = N / 2 + 1;
  constexpr unsigned NMID = DIM == 3 ? N : 1;
  const int kh = (int)(i % H);
  const unsigned rest = i / H;
  const int mid = (int)(rest % NMID);
  const int kxi = (int)(rest / NMID);
  return rk_core<N, DIM, VIF>(kxi, mid, kh, kfull(kxi, N), DIM == 3 ? kfull(mid, N) : 0, c, sv, a0, z0, P, pcs, kt,
                              kd, prm, fscale, nv);
}

// Stage region of the explicit step: modes whose right-hand side can carry the nonlinear
// term or a forcing term: in 3D the half-axis rows |ky| <= kd, in 2D the columns kh < kt.
// Outside it du = -(nu k^2 + drag) u exactly, so with z = (nu k^2 + drag) dt the RK4
// stages are polynomials in z times the step's initial state u0:
//   stage fields  (1 - z/2) u0,  (1 - z/2 + z^2/4) u0,  (1 - z + z^2/2 - z^3/4) u0,
//   new state     (1 - z + z^2/2 - z^3/6 + z^4/24) u0,
// and such a mode needs neither the previous stage field nor the accumulator: per step
// it is read 4 times and written 4 times instead of 8 and 6 times (1/3 of the modes at
// 256^3).
//
// Stage-region form of k_rk_update (explicit scheme, rk >= 0), over float4 pairs of
// modes like k_rk_update. A mode outside the region reads only u0 (us = u0 at rk 0) and
// writes the closed form; the accumulator is stored only inside the region. In 3D the
// region is taken in whole half-axis rows (|ky| <= kd), which keeps the streams dense:
// also cutting the rows at kh = kt moved fewer bytes but ran slower (127.8 against
// 117.6 us per 256^3 launch; the plain form with constant divisions 120.0 us).
template <int N, int DIM>
__device__ __forceinline__ bool in_stage_region(int kh, int mid, int kt, int kd) {
  if (DIM == 2) return kh < kt;
  return (unsigned)(kfull(mid, N) + kd) <= 2u * (unsigned)kd;
}

template <int N, int DIM>
__global__ void __launch_bounds__(256)
k_rk_update_lin(const float2* __restrict__ P, long long pcs, int kt, int kd, const float2* us, const float2* u0,
                float2* acc, float2* out, float2* fin, long long cs, EpiParams prm,
                const double* __restrict__ band_scale, const float* __restrict__ nu_b, int* __restrict__ err) {
  pdl_begin();
  constexpr unsigned H = N / 2 + 1, NMID = DIM == 3 ? N : 1, CS = NMID * N * H;  // CS == cs
  const int batch = blockIdx.y;
  prm.nu = nu_b[batch];  // per-trajectory viscosity
  const long long pairs = 3 * cs / 2;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= pairs) return;
  const long long bo = (long long)batch * 3 * cs;
  const float fscale = prm.band_kf2 > 0 ? (float)band_scale[batch] : 0.f;
  const float2* Pb = P + (long long)batch * 3 * pcs;
  const unsigned ug = (unsigned)(2 * q);
  int cc[2], kxi[2], mid[2], kh[2];
  bool in[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const unsigned g = ug + (unsigned)h;
    cc[h] = (int)(g / CS);
    const unsigned i = g - (unsigned)cc[h] * CS;
    kh[h] = (int)(i % H);
    const unsigned rest = i / H;
    mid[h] = (int)(rest % NMID);
    kxi[h] = (int)(rest / NMID);
    in[h] = in_stage_region<N, DIM>(kh[h], mid[h], kt, kd);
  }
  const bool any_in = in[0] || in[1];
  float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f), a4 = s4, z4 = s4;
  if (any_in) s4 = reinterpret_cast<const float4*>(us + bo)[q];
  if (any_in && prm.rk > 1) a4 = reinterpret_cast<const float4*>(acc + bo)[q];
  if ((any_in && prm.rk > 0 && prm.rk < 3) || !(in[0] && in[1])) z4 = reinterpret_cast<const float4*>(u0 + bo)[q];
  float2 nv[2], r[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float2 sv = h ? make_float2(s4.z, s4.w) : make_float2(s4.x, s4.y);
    const float2 a0 = h ? make_float2(a4.z, a4.w) : make_float2(a4.x, a4.y);
    const float2 z0 = h ? make_float2(z4.z, z4.w) : make_float2(z4.x, z4.y);
    const int kx = kfull(kxi[h], N), km = DIM == 3 ? kfull(mid[h], N) : 0;
    r[h] = make_float2(0.f, 0.f);
    if (in[h]) {
      r[h] = rk_core<N, DIM, false>(kxi[h], mid[h], kh[h], kx, km, cc[h], sv, a0, z0, Pb, pcs, kt, kd, prm, fscale,
                                    nv[h]);
    } else {
      const float z = (prm.nu * (float)(kx * kx + km * km + kh[h] * kh[h]) + prm.drag) * prm.dt;
      const float f = lin_stage_factor(prm.rk, z);
      nv[h] = make_float2(f * z0.x, f * z0.y);
    }
  }
  if (prm.rk < 3) {
    // the accumulator of a mode outside the region is never read
    if (prm.rk > 0 && any_in) reinterpret_cast<float4*>(acc + bo)[q] = make_float4(r[0].x, r[0].y, r[1].x, r[1].y);
    reinterpret_cast<float4*>(out + bo)[q] = make_float4(nv[0].x, nv[0].y, nv[1].x, nv[1].y);
  } else {
    reinterpret_cast<float4*>(fin + bo)[q] = make_float4(nv[0].x, nv[0].y, nv[1].x, nv[1].y);
    if (!isfinite((nv[0].x + nv[0].y) + (nv[1].x + nv[1].y))) atomicOr(err, kErrNonFinite);
  }
}

// The last stage (rk 3) also flags a non-finite value of the new state in *err
// (kErrNonFinite): the blow-up check of the drivers, one add and one compare per
// thread, no extra pass.
template <int N, int DIM, bool VIF = false>
__global__ void __launch_bounds__(256)
k_rk_update(const float2* __restrict__ P, long long pcs, int kt, int kd, const float2* us, const float2* u0,
            float2* acc, float2* out, float2* fin, long long cs, EpiParams prm,
            const double* __restrict__ band_scale, const float* __restrict__ nu_b, int* __restrict__ err) {
  pdl_begin();
  const int batch = blockIdx.y;
  prm.nu = nu_b[batch];  // per-trajectory viscosity
  const long long pairs = 3 * cs / 2;
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long bo = (long long)batch * 3 * cs;
  const float fscale = prm.band_kf2 > 0 ? (float)band_scale[batch] : 0.f;
  if (q < pairs) {
    const long long g = 2 * q;  // global element (component-major)
    const float4 s4 = reinterpret_cast<const float4*>(us + bo)[q];
    float4 a4 = make_float4(0.f, 0.f, 0.f, 0.f), z4 = a4;
    if (prm.rk > 1) a4 = reinterpret_cast<const float4*>(acc + bo)[q];
    if (prm.rk > 0 && prm.rk < 3) z4 = reinterpret_cast<const float4*>(u0 + bo)[q];
    const float2* Pb = P + (long long)batch * 3 * pcs;
    float2 nv0, nv1;
    constexpr unsigned ucs = (DIM == 3 ? N : 1) * N * (N / 2 + 1);  // == cs: constant divisions
    const unsigned ug = (unsigned)g;
    const int c0 = (int)(ug / ucs), c1 = (int)((ug + 1u) / ucs);
    const float2 r0 = rk_elem<N, DIM, VIF>(ug - (unsigned)c0 * ucs, c0, make_float2(s4.x, s4.y), make_float2(a4.x, a4.y),
                                      make_float2(z4.x, z4.y), Pb, pcs, kt, kd, prm, fscale, nv0);
    const float2 r1 = rk_elem<N, DIM, VIF>(ug + 1u - (unsigned)c1 * ucs, c1, make_float2(s4.z, s4.w),
                                      make_float2(a4.z, a4.w), make_float2(z4.z, z4.w), Pb, pcs, kt, kd, prm,
                                      fscale, nv1);
    if (prm.rk < 0) {
      reinterpret_cast<float4*>(out + bo)[q] = make_float4(r0.x, r0.y, r1.x, r1.y);
    } else if (prm.rk < 3) {
      if (prm.rk > 0) reinterpret_cast<float4*>(acc + bo)[q] = make_float4(r0.x, r0.y, r1.x, r1.y);
      reinterpret_cast<float4*>(out + bo)[q] = make_float4(nv0.x, nv0.y, nv1.x, nv1.y);
    } else {
      reinterpret_cast<float4*>(fin + bo)[q] = make_float4(nv0.x, nv0.y, nv1.x, nv1.y);
      // a sum of values is non-finite if one of them is (or if it overflows, which a
      // field near FLT_MAX is about to do anyway)
      if (!isfinite((nv0.x + nv0.y) + (nv1.x + nv1.y))) atomicOr(err, kErrNonFinite);
    }
  }
}

// Lamorgese et al. KE rescaling (spectral_solver.py:82-112), one CTA per trajectory.
// E_new from the per-CTA partials of the energy pass (deterministic order), E_low from the
// band, alpha = sqrt(max(0, (E0 - (E_new - E_low)) / (E_low + eps))), band *= alpha.
template <int DIM>
__global__ void __launch_bounds__(256)
k_force_ekin(float2* __restrict__ uh, long long cs, const double* __restrict__ partial,
             int npartial, const double* __restrict__ e0, double dt, int N, int kf,
             double inv_n2d, double eps, double* __restrict__ e_inj, double* __restrict__ ke_out) {
  pdl_begin();
  const int batch = blockIdx.x;
  float2* ub = uh + (long long)batch * 3 * cs;
  __shared__ double red[32];
  __shared__ double s_alpha;
  double s = 0.0;
  for (int i = threadIdx.x; i < npartial; i += blockDim.x) s += partial[(long long)batch * npartial + i];
  double lo = 0.0;
  const int nb = band_count<DIM>(kf);
  for (int i = threadIdx.x; i < nb; i += blockDim.x) {
    long long idx;
    int wg;
    if (!band_mode<DIM>(i, N, kf, idx, wg)) continue;
    for (int c = 0; c < 3; ++c) {
      const float2 v = ub[c * cs + idx];
      lo += wg * ((double)v.x * v.x + (double)v.y * v.y);
    }
  }
  // reduce (s, lo) over the CTA
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o);
    lo += __shfl_xor_sync(0xffffffffu, lo, o);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) {
    red[wid] = s;
    red[16 + wid] = lo;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double S = 0.0, L = 0.0;
    for (int i = 0; i < nw; ++i) {
      S += red[i];
      L += red[16 + i];
    }
    const double e_new = 0.5 * S * inv_n2d;
    const double e_low = 0.5 * L * inv_n2d;
    const double e_high = e_new - e_low;
    const double E0 = e0[batch];
    const double arg = (E0 - e_high) / (e_low + eps);
    s_alpha = sqrt(arg > 0.0 ? arg : 0.0);
    const double inj = (E0 - e_new) / dt;
    e_inj[batch] = inj > 0.0 ? inj : 0.0;
    if (ke_out) ke_out[batch] = e_high + s_alpha * s_alpha * e_low;
  }
  __syncthreads();
  const float alpha = (float)s_alpha;
  for (int i = threadIdx.x; i < nb; i += blockDim.x) {
    long long idx;
    int wg;
    if (!band_mode<DIM>(i, N, kf, idx, wg)) continue;
    for (int c = 0; c < 3; ++c) {
      float2 v = ub[c * cs + idx];
      ub[c * cs + idx] = make_float2(v.x * alpha, v.y * alpha);
    }
  }
}

}  // namespace l3es
