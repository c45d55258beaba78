// The x pass of the explicit RK4 step for sm_103a: one kernel closes a stage and opens
// the next one.
//
// On an x pencil (fixed middle and half-axis wavenumbers) the forward x FFT of the
// nonlinear term, the dealias mask, the Leray projection, the RK4 stage combination and
// the next stage's inverse x FFT of u and curl u all act on the same column of modes, so
// kx_stage does them in one visit: the new stage field goes from the combination into
// the inverse transform without a trip through memory, and a stage is two launches
// (kx_stage and in 2D the line pass, in 3D k_yz_plane or k_yz_half).
//
// The band B = {|kx| <= kd, |kmid| <= kd (3D), khalf < kt} holds every nonlinear and
// forcing term. Outside it du = -(nu k^2 + drag) u exactly, so a stage field there is a
// polynomial in z = (nu k^2 + drag) dt times the step's initial value (lin_stage_factor):
// those modes keep u0 in the state S until stage 2 replaces them by their new state, and
// are read and scaled on the way into each inverse transform. On the band, S keeps u0
// until stage 3 writes the new state, T holds the stage field and C the accumulator, all
// in S's layout.
#pragma once

#include "dns_kernels.cuh"

namespace l3es {

// Where the explicit step takes kx_stage: every 2D grid and 3D grids up to 64^3 (there with
// k_yz_plane between two x passes). Those are bound by latency: few CTAs, each a chain of
// dependent transforms, and the launches count. Measured per step against the separate
// passes (x inverse, y inverse, line, y forward, band pass, 2D also the update): 2D 256^2
// 98.3 -> 69.7 us, 128^2 x 8 98.4 -> 70.6 us, 512^2 122.9 -> 97.7 us; 3D, dependent launches
// on both sides, 64^3 89 -> 71 us, 64^3 x 6 222 -> 208 us, 64^3 x 12 425 -> 423 us; from
// plain launches 32^3 121 -> 35 us, 16^3 130 -> 41 us. (With dependent launches, paired adds
// and the line passes of their size those steps now take 47, 42 and 51 us.) With kx_stage 128^3 takes 38 instead
// of 32.6 us for one stage's x passes and 256^3 267 instead of 195 us: there the chip is full
// and the barriers of the three groups cost more than the saved round trip. Larger 3D grids
// keep kx_inv and the band-fused kx_fwd_band.
constexpr int kStageMax3d = 64;  // largest 3D grid with kx_stage kernels
inline bool step_by_kx_stage(int dim, int n) { return dim == 2 || n <= kStageMax3d; }

// 3D grids whose y transforms between two x passes go by halves (k_yz_half; 16^3 has too few
// rows for a warp and takes k_yz_plane)
constexpr bool yz_by_halves(int n) { return n >= 32 && n <= kStageMax3d; }

// Parameters of one stage.
struct XStage {
  long long cs;
  int kd, kt;
  EpiParams prm;             // prm.rk is the kernel's RK
  const double* band_scale;  // [batch] constant-power coefficient of the stage's input field
  const float* nu_b;         // [batch] viscosities
  int* err;
};

// XW columns per CTA and one thread group per velocity component, XW T threads each
// (thread = (component g, x row t, column p), p fastest). A group transforms its own
// component; the two contractions that mix components (projection, curl) read the other
// two from shared memory. Against one group that walks through the components, the CTA
// has three times the threads and a third of the registers per thread, and the chain of
// dependent transforms is 3 instead of 8 (3D) or 9 (2D).
template <int N, int XW, int EE>
struct XStageCfg {
  static constexpr int E = EE, T = N / E;
  static constexpr int G = XW * T;                       // threads per component
  static constexpr int THREADS = 3 * G;
  static_assert(G % 32 == 0, "a component's barriers count whole warps");
  static constexpr int XS = xpad_len<XW>(N) * XW;        // exchange slots per component
  static constexpr int US = N * XW;                      // shared column values per component
  static constexpr int SMEM = 3 * (XS + US) * (int)sizeof(float2);
};

// S: the state, T_: stage field, C: accumulator, [batch][3][cs] each.
// RK = -1: opens a step: inverse transforms of S as it is. RK = 0..3: closes stage RK
// from the y-transformed nonlinear term du; INV: also opens the next stage (RK < 3) or
// the next step (RK = 3), else only the band of S is written.
// 3D: u_x, curl_y, curl_z go to w (fields 0, 4, 5) and u_y, u_z to wx, as ky_inv_rhs
// reads them; 2D: six fields to w.
template <int N, int DIM, int XW, int EE, int RK, bool INV>
__global__ void __launch_bounds__(XStageCfg<N, XW, EE>::THREADS)
kx_stage(const float2* __restrict__ du, long long dcs, float2* __restrict__ S, float2* __restrict__ T_,
         float2* __restrict__ C, const __grid_constant__ XStage st, float2* __restrict__ w, float2* __restrict__ wx,
         long long fs, const float2* __restrict__ tw) {
  pdl_begin();
  using K = XStageCfg<N, XW, EE>;
  constexpr int E = K::E, T = K::T, H = N / 2 + 1;
  constexpr int NMID = DIM == 3 ? N : 1;
  constexpr int MC = NMID * H;
  extern __shared__ __align__(16) float2 s_stage[];
  const int g = threadIdx.x / K::G, q = threadIdx.x % K::G;
  const int p = q % XW, t = q / XW;
  float2* su = s_stage;                           // [component][row][column]
  float2* sx = s_stage + 3 * K::US + g * K::XS;   // this component's exchange buffer
  const int m = blockIdx.x * XW + p;
  const int batch = blockIdx.y;
  const bool ok = m < MC;
  const int mid = DIM == 3 ? m / H : 0;
  const int kh = m - mid * H;
  const int km = DIM == 3 ? kfull(mid, N) : 0;
  const int kd = st.kd, kt = st.kt;
  const unsigned ukd = 2u * (unsigned)kd;
  const bool colband = RK >= 0 && ok && kh < kt && (DIM == 2 || (unsigned)(km + kd) <= ukd);
  const long long so = ((long long)batch * 3 + g) * st.cs + m;  // + row * MC
  const float nu = st.nu_b[batch];
  float2 v[E];
  // operands of the combination, in flight while the nonlinear term is transformed (a
  // CTA's chain of loads and transforms is what a small grid waits for; registers are not)
  float2 u0[RK >= 0 ? E : 1], sv[RK >= 1 ? E : 1], ac[RK >= 2 ? E : 1];
  if (RK >= 0) {
    const bool tile_band = __syncthreads_or(colband);
    if (!INV && !tile_band) return;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int row = t + T * e;
      const bool band = colband && (unsigned)(kfull(row, N) + kd) <= ukd;
      const long long o = so + (long long)row * MC;
      const float2 z = make_float2(0.f, 0.f);
      u0[RK >= 0 ? e : 0] = (band ? RK < 3 : INV && ok) ? S[o] : z;
      if (RK >= 1) sv[RK >= 1 ? e : 0] = band ? T_[o] : z;
      if (RK >= 2) ac[RK >= 2 ? e : 0] = band ? C[o] : z;
    }
    if (tile_band) {
      // nonlinear term: x forward, dealias, Leray projection of this component
      constexpr bool half = DIM == 3 && yz_by_halves(N);  // du holds the halves of the y transform
      const float2* db = du + ((long long)batch * 3 + g) * dcs + (long long)(half ? mid % (N / 2) : mid) * kt + kh;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const float2* d = db + (long long)(t + T * e) * NMID * kt;
        v[e] = colband ? __ldg(d) : make_float2(0.f, 0.f);
        if (half && colband) {
          const float2 o = __ldg(d + N / 2 * kt);
          v[e] = mid < N / 2 ? cadd(v[e], o) : csub(v[e], o);
        }
      }
      block_fft<N, E, kFwd, XW, kSyncGroup>(v, sx + p, t, tw, 1);
#pragma unroll
      for (int e = 0; e < E; ++e) su[g * K::US + (t + T * e) * XW + p] = v[e];
      __syncthreads();
      const bool keep = kh <= kd;
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int row = t + T * e;
        const float2 z = make_float2(0.f, 0.f);
        const float2 v0 = keep ? su[row * XW + p] : z;
        const float2 v1 = keep ? su[K::US + row * XW + p] : z;
        const float2 v2 = keep ? su[2 * K::US + row * XW + p] : z;
        float k0, k1, k2;
        const int kx = kfull(row, N);
        kvec<DIM>(kx, km, kh, k0, k1, k2);
        const int ik2 = kx * kx + km * km + kh * kh;
        const float inv = 1.0f / (ik2 == 0 ? 1.0f : (float)ik2);
        const float pr = (v0.x * k0 + v1.x * k1 + v2.x * k2) * inv;
        const float pi_ = (v0.y * k0 + v1.y * k1 + v2.y * k2) * inv;
        const float2 own = g == 0 ? v0 : g == 1 ? v1 : v2;
        const float kg = g == 0 ? k0 : g == 1 ? k1 : k2;
        v[e] = make_float2(own.x - pr * kg, own.y - pi_ * kg);
      }
      if (INV) __syncthreads();  // the products are read; su takes the new stage field
    }
  }
  // stage combination on the band, closed form elsewhere: v becomes this component's field
  if constexpr (RK < 0) {
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = ok ? S[so + (long long)(t + T * e) * MC] : make_float2(0.f, 0.f);
  } else {
    EpiParams prm = st.prm;
    prm.rk = RK;
    prm.nu = nu;
    const float fscale = prm.band_kf2 > 0 ? (float)st.band_scale[batch] : 0.f;
    bool bad = false;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int row = t + T * e;
      const int kx = kfull(row, N);
      const long long o = so + (long long)row * MC;
      const int ik2 = kx * kx + km * km + kh * kh;
      const float2 z0 = make_float2(0.f, 0.f);
      float2 nv;
      if (colband && (unsigned)(kx + kd) <= ukd) {
        const float2 ra = rk_core_r<N, DIM, false>(row, mid, kh, ik2, g, v[e], RK == 0 ? u0[e] : sv[RK >= 1 ? e : 0],
                                                   RK >= 2 ? ac[RK >= 2 ? e : 0] : z0, u0[e], prm, fscale, nv);
        if (RK == 1 || RK == 2) C[o] = ra;
        if (RK == 3)
          S[o] = nv;
        else
          T_[o] = nv;
        if (RK == 3) bad |= !isfinite(nv.x + nv.y);
        v[e] = nv;
      } else if (RK == 3) {
        v[e] = u0[e];  // the new state, written by stage 2
      } else {
        const float z = (nu * (float)ik2 + prm.drag) * prm.dt;
        const float f = lin_stage_factor(RK, z);
        if (RK == 2 && ok) {
          const float gn = lin_stage_factor(3, z);
          nv = make_float2(gn * u0[e].x, gn * u0[e].y);
          S[o] = nv;
          bad |= !isfinite(nv.x + nv.y);
        }
        v[e] = make_float2(f * u0[e].x, f * u0[e].y);
      }
    }
    if (RK >= 2 && bad) atomicOr(st.err, kErrNonFinite);
  }
  if constexpr (INV) {
#pragma unroll
    for (int e = 0; e < E; ++e) su[g * K::US + (t + T * e) * XW + p] = v[e];
    __syncthreads();
    block_fft<N, E, kInv, XW, kSyncGroup>(v, sx + p, t, tw, 1);
    if (ok) {
      float2* dst = DIM == 3 && g > 0 ? wx + ((long long)batch * 2 + g - 1) * fs : w + ((long long)batch * 6 + g) * fs;
#pragma unroll
      for (int e = 0; e < E; ++e) dst[(long long)(t + T * e) * MC + m] = v[e];
    }
    // curl component g = i (k x u)_g; in 3D the y pass forms the x component itself
    if (DIM == 3 && g == 0) return;
    const int ga = g == 2 ? 0 : g + 1, gb = g == 0 ? 2 : g - 1;  // (k x u)_g = k_ga u_gb - k_gb u_ga
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int row = t + T * e;
      float k0, k1, k2;
      kvec<DIM>(kfull(row, N), km, kh, k0, k1, k2);
      const float ka = g == 0 ? k1 : g == 1 ? k2 : k0, kb = g == 0 ? k2 : g == 1 ? k0 : k1;
      const float2 ua = su[ga * K::US + row * XW + p], ub = su[gb * K::US + row * XW + p];
      v[e] = mul_i<kInv>(make_float2(ka * ub.x - kb * ua.x, ka * ub.y - kb * ua.y));
    }
    group_sync<K::G>();  // the exchange buffer's last reads are done
    block_fft<N, E, kInv, XW, kSyncGroup>(v, sx + p, t, tw, 1);
    if (ok) {
      float2* dst = w + ((long long)batch * 6 + 3 + g) * fs;
#pragma unroll
      for (int e = 0; e < E; ++e) dst[(long long)(t + T * e) * MC + m] = v[e];
    }
  }
}

// ------------------------------------------------------------------------------
// Half-axis line pass of 64^2 and 128^2 grids: one line per slot of T = N / 8 lanes, 32 / T
// lines per warp, and the z products of two neighbouring slots in one transform that both
// run (a slot doing two lines one after the other, as line_cross2 does, has a chain of 9
// transforms instead of 5, on half as many warps: 8.1 us for 8 fields of 128^2). lines is
// even.
// ------------------------------------------------------------------------------
template <int N>
__global__ void __launch_bounds__(128)
line_cross_slots(const float2* __restrict__ w, long long fs, float2* __restrict__ du, long long ds, int kt, int kd,
                 float s2, const float2* __restrict__ ct8, int lines) {
  pdl_begin();
  static_assert(N >= 64 && N <= 128, "two lines per warp");
  constexpr int T = N / 8, H = N / 2 + 1;
  __shared__ float2 s_x[128 / T * xpad_len<1>(N)];
  const int slot = threadIdx.x / T, t = threadIdx.x % T;
  float2* xs = s_x + slot * xpad_len<1>(N);
  const int line_raw = blockIdx.x * (128 / T) + slot;
  const bool valid = line_raw < lines;
  const int line = valid ? line_raw : lines - 2 + (slot & 1);
  const float2* src = w + (long long)blockIdx.y * 6 * fs + (long long)line * H;
  float2 h1[8], h2[8], z[8];
  c2r_pair_load<N>(src, src + fs, t, h1);               // u_x + i u_y
  c2r_pair_load<N>(src + 2 * fs, src + 3 * fs, t, h2);  // u_z + i curl_x
  c2r_pair_load<N>(src + 4 * fs, src + 5 * fs, t, z);   // curl_y + i curl_z
  warp_fft<N, 8, kInv>(h1, xs, t, ct8);
  __syncwarp();
  warp_fft<N, 8, kInv>(h2, xs, t, ct8);
  __syncwarp();
  warp_fft<N, 8, kInv>(z, xs, t, ct8);
  __syncwarp();
  float2 y[8];
  const bool odd = slot & 1;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float ux = h1[e].x, uy = h1[e].y, uz = h2[e].x, wx = h2[e].y, wy = z[e].x, wz = z[e].y;
    const float pz = fmaf(ux, wy, -uy * wx);
    const float other = __shfl_xor_sync(0xffffffffu, pz, T);
    y[e] = odd ? make_float2(other, pz) : make_float2(pz, other);
    z[e] = make_float2(fmaf(uy, wz, -uz * wy), fmaf(uz, wx, -ux * wz));
  }
  warp_fft<N, 8, kFwd>(z, xs, t, ct8);
  __syncwarp();
  warp_fft<N, 8, kFwd>(y, xs, t, ct8);
  float2 X[4], Y[4], A[4], B[4];
  r2c_pair_unpack<N>(z, t, s2, X, Y);
  r2c_pair_unpack<N>(y, t, s2, A, B);
  if (valid) {
    float2* dst = du + (long long)blockIdx.y * 3 * ds + (long long)line * kt;
    store_du_line<N>(dst, X, t, kt, kd);
    store_du_line<N>(dst + ds, Y, t, kt, kd);
    store_du_line<N>(dst + 2 * ds, odd ? B : A, t, kt, kd);
  }
}

// ------------------------------------------------------------------------------
// Everything between two x passes of a small 3D grid in one kernel, one x plane per CTA (16^3;
// 32^3 and 64^3 take k_yz_half): y inverse of the six fields (u, curl u; curl_x formed here,
// as in ky_inv_rhs), the half-axis lines with u x curl u (two real lines per complex FFT, as
// in line_cross2) and the y forward of the three products, kept rows only, to du. A plane's
// six fields (123 KB at 64^3) fit shared memory, so the three passes meet there instead of in
// global memory, in one launch instead of three. Warps work alone inside a phase: a warp
// takes 32 / T neighbouring columns (y transforms) or 32 / T lines, T = N / 8 lanes each.
// ct8: compact twiddle table of the N-point FFT (line2_ct_offset).
// ------------------------------------------------------------------------------
template <int N>
struct YzCfg {
  static constexpr int T = N / 8;                 // lanes per transform
  static constexpr int XC = 32 / T;               // columns (lines) per warp
  static constexpr int H = N / 2 + 1;
  static constexpr int WARPS = N == 64 ? 16 : N == 32 ? 8 : 6;
  static constexpr int THREADS = 32 * WARPS;
  // row length of a field: the lines of a half warp's loads fall into different banks
  static constexpr int LD = N == 64 ? 40 : N == 32 ? 20 : 12;
  static constexpr int FIELD = N * LD;
  static constexpr int XS1 = XC * xpad_len<1>(N), XSC = XC * xpad_len<XC>(N);
  static constexpr int XS = XS1 > XSC ? XS1 : XSC;  // exchange slots per warp
  static constexpr int SMEM = (6 * FIELD + WARPS * XS) * (int)sizeof(float2);
};

template <int D>
struct Dir {
  static constexpr int value = D;
};

// Z = X_ext + i Y_ext (c2r_pair_load) from two half-spectrum rows in shared memory
template <int N>
__device__ __forceinline__ void c2r_pair_row(const float2* X, const float2* Y, int t, float2 (&z)[8]) {
  constexpr int T = N / 8;
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const int n = t + T * e;
    const bool lo = e < 4;
    float2 x = X[lo ? n : N - n], y = Y[lo ? n : N - n];
    if ((e == 0 || e == 4) && t == 0) {  // n = 0 and n = N/2: real parts only
      x.y = 0.f;
      y.y = 0.f;
    }
    z[e] = lo ? make_float2(x.x - y.y, x.y + y.x) : make_float2(x.x + y.y, y.x - x.y);
  }
}

// Half-axis lines of a plane in shared memory (six fields, rows of LD): u x curl u of every
// row into the first kt columns of fields 0..2. Slot y of T lanes takes row y; the z
// products of rows y and y + PB/2 of a block of PB rows share one transform. All threads; xs: the warp's exchange
// buffer.
template <int N, int ROWS = N, int PB = ROWS>
__device__ __forceinline__ void plane_lines(float2* s_yz, float2* xs, int kt, int kd, float s2,
                                            const float2* __restrict__ ct8) {
  using C = YzCfg<N>;
  constexpr int T = C::T, LD = C::LD, FIELD = ROWS * LD;
  const int lane = threadIdx.x & 31;
  const int y = threadIdx.x / T, t = threadIdx.x % T;
  float2* xl = xs + lane / T * xpad_len<1>(N);
  float2* row = s_yz + (y < ROWS ? y : 0) * LD;
  float pz[8];
  auto put = [&](float2* dst, const float2 (&X)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = t + T * e;
      if (k < kt) dst[k] = k <= kd ? X[e] : make_float2(0.f, 0.f);
    }
  };
  if (y < ROWS) {  // whole warps
    float2 h1[8], h2[8], z[8];
    c2r_pair_row<N>(row, row + FIELD, t, z);  // u_x + i u_y
    warp_fft<N, 8, kInv>(z, xl, t, ct8);
#pragma unroll
    for (int e = 0; e < 8; ++e) h1[e] = z[e];
    __syncwarp();
    c2r_pair_row<N>(row + 2 * FIELD, row + 3 * FIELD, t, z);  // u_z + i curl_x
    warp_fft<N, 8, kInv>(z, xl, t, ct8);
#pragma unroll
    for (int e = 0; e < 8; ++e) h2[e] = z[e];
    __syncwarp();
    c2r_pair_row<N>(row + 4 * FIELD, row + 5 * FIELD, t, z);  // curl_y + i curl_z
    warp_fft<N, 8, kInv>(z, xl, t, ct8);
    __syncwarp();
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float ux = h1[e].x, uy = h1[e].y, uz = h2[e].x, wx_ = h2[e].y, wy = z[e].x, wz = z[e].y;
      pz[e] = fmaf(ux, wy, -uy * wx_);
      z[e] = make_float2(fmaf(uy, wz, -uz * wy), fmaf(uz, wx_, -ux * wz));
    }
    warp_fft<N, 8, kFwd>(z, xl, t, ct8);
    float2 X[4], Y[4];
    r2c_pair_unpack<N>(z, t, s2, X, Y);
    // this line's rows are read: they take its products
    put(row, X);
    put(row + FIELD, Y);
    if (y % PB >= PB / 2) {
      float* zr = reinterpret_cast<float*>(row + 3 * FIELD);
#pragma unroll
      for (int e = 0; e < 8; ++e) zr[t + T * e] = pz[e];
    }
  }
  __syncthreads();
  if (y < ROWS && (y % PB < PB / 2 || PB / 2 * T < 32)) {  // whole warps
    const bool lower = y % PB < PB / 2;
    const float* zr = reinterpret_cast<const float*>(s_yz + 3 * FIELD + (lower ? y + PB / 2 : y) * LD);
    float2 z[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) z[e] = make_float2(pz[e], zr[t + T * e]);
    warp_fft<N, 8, kFwd>(z, xl, t, ct8);
    float2 X[4], Y[4];
    r2c_pair_unpack<N>(z, t, s2, X, Y);
    if (lower) {
      put(row + 2 * FIELD, X);
      put(row + 2 * FIELD + PB / 2 * LD, Y);
    }
  }
}

template <int N>
__global__ void __launch_bounds__(YzCfg<N>::THREADS)
k_yz_plane(const float2* __restrict__ w, const float2* __restrict__ wx, long long fs, float2* __restrict__ du,
           long long ds, int kt, int kd, float s2, const float2* __restrict__ tw, const float2* __restrict__ ct8) {
  pdl_begin();
  using C = YzCfg<N>;
  constexpr int T = C::T, XC = C::XC, H = C::H, LD = C::LD;
  extern __shared__ __align__(16) float2 s_yz[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* xs = s_yz + 6 * C::FIELD + warp * C::XS;
  const long long plane = (long long)blockIdx.x * N * H;
  // y inverse: warp jobs (column tile, field), the field varying fastest
  {
    const float2* wb = w + (long long)blockIdx.y * 6 * fs + plane;
    const float2* xb = wx + (long long)blockIdx.y * 2 * fs + plane;
    const int p = lane % XC, t = lane / XC;
    constexpr int TILES = (H + XC - 1) / XC;
    for (int j = warp; j < 6 * TILES; j += C::WARPS) {
      const int f = j % 6, col = j / 6 * XC + p;
      const bool ok = col < H;
      float2 v[8];
      if (f == 3) {
        const float kz = (float)col;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int o = (t + T * e) * H + col;
          const float2 wy = ok ? __ldg(xb + o) : make_float2(0.f, 0.f);
          const float2 wz = ok ? __ldg(xb + fs + o) : make_float2(0.f, 0.f);
          const float ky = (float)kfull(t + T * e, N);
          v[e] = mul_i<kInv>(make_float2(ky * wz.x - kz * wy.x, ky * wz.y - kz * wy.y));
        }
      } else {
        const float2* src = f == 1 || f == 2 ? xb + (f - 1) * fs : wb + f * fs;
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = ok ? __ldg(src + (t + T * e) * H + col) : make_float2(0.f, 0.f);
      }
      block_fft<N, 8, kInv, XC, kSyncWarp>(v, xs + p, t, tw, 1);
      if (ok) {
#pragma unroll
        for (int e = 0; e < 8; ++e) s_yz[f * C::FIELD + (t + T * e) * LD + col] = v[e];
      }
      __syncwarp();
    }
  }
  __syncthreads();
  plane_lines<N>(s_yz, xs, kt, kd, s2, ct8);
  __syncthreads();
  // y forward of the products' kept columns, rows |ky| <= kd to du
  {
    const int p = lane % XC, t = lane / XC;
    const int tiles = (kt + XC - 1) / XC;
    float2* db = du + (long long)blockIdx.y * 3 * ds + (long long)blockIdx.x * N * kt;
    for (int j = warp; j < 3 * tiles; j += C::WARPS) {
      const int c = j % 3, col = j / 3 * XC + p;
      const bool ok = col < kt;
      float2 v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e)
        v[e] = ok ? s_yz[c * C::FIELD + (t + T * e) * LD + col] : make_float2(0.f, 0.f);
      block_fft<N, 8, kFwd, XC, kSyncWarp>(v, xs + p, t, tw, 1);
      if (ok) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int ky = t + T * e;
          if ((unsigned)(kfull(ky, N) + kd) <= 2u * (unsigned)kd) db[c * ds + (long long)ky * kt + col] = v[e];
        }
      }
      __syncwarp();
    }
  }
}

// ------------------------------------------------------------------------------
// k_yz_plane with a plane shared by two CTAs, one for the even rows y and one for the odd: the
// inverse y transform gives a CTA its rows from the folded columns (V[k] + V[k + N/2] or their
// difference: half_rows_inv), the lines of its rows need nothing else, and the halves of the
// forward transform (half_rows_fwd) meet where kx_stage reads them:
//   X[k] = E[k] + exp(-2 pi i k / N) O[k],  X[k + N/2] = E[k] - exp(-2 pi i k / N) O[k],
// E and the turned O in rows k and N/2 + k of du. Twice the CTAs, for launches that leave SMs
// idle. Bound by latency: the 16 loads of a column stay unbranched so that
// they are in flight together, and a CTA has twice the warps that the lines need, for the
// columns (ten 64^3 steps 705 us with half of them, 532 us; 676 us by k_yz_plane).
//
// The halves are the halves of an N-point transform of radix 8 and N/8 (8 x 8, 8 x 4): the fold
// is the first level of its radix-8 butterflies, whose outputs of one parity are four of
// eight, and the turn by exp(2 pi i k / N) goes into the twiddles between its stages and the
// eighth turns of the butterfly. A turn of its own beside an N/2-point transform took one
// more rounding per value: the error of 64^3 and 32^3 steps against 64 bits was 0.7 and 1.2 %
// above the unsplit transforms' in nearly every field, now it is level with theirs, and ten
// 64^3 steps take 513 us instead of 532 (32^3 320 and 324).
// ------------------------------------------------------------------------------
// x times the k-th eighth turn, exp(DIR 2 pi i k / 8), k = 0..3
template <int DIR>
__device__ __forceinline__ float2 turn8(float2 x, int k) {
  const float c = 0.70710678118654752f;
  return k == 0 ? x : k == 2 ? mul_i<DIR>(x) : cmul(x, make_float2(k == 1 ? c : -c, DIR * c));
}

// Rows 2 m + odd (m = t + T e of N/2) of the inverse N-point transform, T = N / 16 lanes; v, b:
// its inputs k = t + T e and k + N/2. XC interleaved columns; sm: N/2 + N/8 slots of them.
template <int N, int XC>
__device__ __forceinline__ void half_rows_inv(const float2 (&v)[8], const float2 (&b)[8], int odd, float2 (&z)[8],
                                              float2* sm, int t, const float2* __restrict__ tw) {
  constexpr int T = N / 16, R2 = N / 8, B2 = 8 / R2;
  // one slot of padding in four: the lanes' writes, four slots apart, fall into different banks
  auto slot = [&](int n) { return sm + (n + n / 4) * XC; };
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    float2 x[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int e = q + 2 * r;
      x[r] = odd ? turn8<kInv>(csub(v[e], b[e]), r) : cadd(v[e], b[e]);
    }
    Dft<4, kInv, true>::run(x);
#pragma unroll
    for (int r = 0; r < 4; ++r) *slot(4 * (t + T * q) + r) = x[r];
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < B2; ++q) {
    const int j = t + T * q;
    float2 x[R2];
#pragma unroll
    for (int r = 0; r < R2; ++r) {
      x[r] = *slot(j + 4 * r);
      if (r > 0) x[r] = cmul(x[r], twid<kInv>(tw, r * (2 * j + odd)));
    }
    Dft<R2, kInv, true>::run(x);
#pragma unroll
    for (int r = 0; r < R2; ++r) z[q + r * B2] = x[r];
  }
}

// The half of the forward N-point transform that rows 2 m + odd give, m = t + T e of N/2, in
// place: outputs k = t + T e < N/2, those of the odd rows turned by exp(-2 pi i k / N).
template <int N, int XC>
__device__ __forceinline__ void half_rows_fwd(float2 (&v)[8], int odd, float2* sm, int t,
                                              const float2* __restrict__ tw) {
  constexpr int T = N / 16, R1 = N / 8, B1 = 8 / R1;
  auto slot = [&](int n) { return sm + (n + n / 8) * XC; };
#pragma unroll
  for (int q = 0; q < B1; ++q) {
    float2 x[R1];
#pragma unroll
    for (int r = 0; r < R1; ++r) x[r] = v[q + r * B1];
    Dft<R1, kFwd, true>::run(x);
#pragma unroll
    for (int r = 0; r < R1; ++r) *slot((t + T * q) * R1 + r) = x[r];
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int j = t + T * q;
    float2 x[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) x[r] = cmul(*slot(j + R1 * r), twid<kFwd>(tw, j * (2 * r + odd)));
    Dft<4, kFwd, true>::run(x);
#pragma unroll
    for (int r = 0; r < 4; ++r) v[q + 2 * r] = odd ? turn8<kFwd>(x[r], r) : x[r];
  }
}

template <int N, int CTAS>
struct YzHalfCfg {
  static constexpr int R = N / 2;                 // rows of a half
  static constexpr int T = R / 8;                 // lanes per y transform
  static constexpr int XC = 32 / T;               // columns per warp
  static constexpr int ROWS = N / CTAS;
  static constexpr int THREADS = YzCfg<N>::THREADS;  // at least a slot per row in the lines
  static constexpr int WARPS = THREADS / 32;
  static constexpr int FIELD = ROWS * YzCfg<N>::LD;
  static constexpr int XSC = XC * (R + R / 4);
  static constexpr int XS = YzCfg<N>::XS1 > XSC ? YzCfg<N>::XS1 : XSC;
  static constexpr int SMEM = (6 * FIELD + WARPS * XS) * (int)sizeof(float2);
};

// CTAS: per plane, 2 or 1 (both halves in turn: the same arithmetic, so that a trajectory's
// result does not depend on the batch)
template <int N, int CTAS>
__global__ void __launch_bounds__(YzHalfCfg<N, CTAS>::THREADS)
k_yz_half(const float2* __restrict__ w, const float2* __restrict__ wx, long long fs, float2* __restrict__ du,
          long long ds, int kt, int kd, float s2, const float2* __restrict__ tw, const float2* __restrict__ ct8) {
  pdl_begin();
  using C = YzHalfCfg<N, CTAS>;
  constexpr int R = C::R, T = C::T, XC = C::XC, H = YzCfg<N>::H, LD = YzCfg<N>::LD;
  extern __shared__ __align__(16) float2 s_yz[];
  const int first = CTAS == 2 ? blockIdx.x & 1 : 0, x = blockIdx.x / CTAS;  // the CTA's first half
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int p = lane % XC, t = lane / XC;
  float2* xs = s_yz + 6 * C::FIELD + warp * C::XS;
  {
    const long long plane = (long long)x * N * H;
    const float2* wb = w + (long long)blockIdx.y * 6 * fs + plane;
    const float2* xb = wx + (long long)blockIdx.y * 2 * fs + plane;
    constexpr int TILES = (H + XC - 1) / XC;
    for (int j = warp; j < 6 * TILES; j += C::WARPS) {
      const int f = j % 6, col = j / 6 * XC + p;
      const bool ok = col < H;
      float2 v[8], b[8];
      if (f == 3) {
        const float kz = (float)col;
        float2 y[16], z[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const int o = (t + T * (e & 7) + R * (e >> 3)) * H + col;
          y[e] = ok ? __ldg(xb + o) : make_float2(0.f, 0.f);
          z[e] = ok ? __ldg(xb + fs + o) : make_float2(0.f, 0.f);
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float ky = (float)kfull(t + T * (e & 7) + R * (e >> 3), N);
          (e < 8 ? v[e & 7] : b[e & 7]) =
              mul_i<kInv>(make_float2(ky * z[e].x - kz * y[e].x, ky * z[e].y - kz * y[e].y));
        }
      } else {
        const float2* src = f == 1 || f == 2 ? xb + (f - 1) * fs : wb + f * fs;
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = ok ? __ldg(src + (t + T * e) * H + col) : make_float2(0.f, 0.f);
#pragma unroll
        for (int e = 0; e < 8; ++e) b[e] = ok ? __ldg(src + (t + T * e + R) * H + col) : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int h = 0; h < 3 - CTAS; ++h) {
        float2 z[8];
        half_rows_inv<N, XC>(v, b, first + h, z, xs + p, t, tw);
        if (ok) {
#pragma unroll
          for (int e = 0; e < 8; ++e) s_yz[f * C::FIELD + (h * R + t + T * e) * LD + col] = z[e];
        }
        __syncwarp();
      }
    }
  }
  __syncthreads();
  plane_lines<N, C::ROWS, R>(s_yz, xs, kt, kd, s2, ct8);
  __syncthreads();
  // y forward of the CTA's halves, kept columns
  {
    const int tiles = (kt + XC - 1) / XC;
    float2* db = du + (long long)blockIdx.y * 3 * ds + (long long)x * N * kt;
    for (int j = warp; j < 3 * (3 - CTAS) * tiles; j += C::WARPS) {
      const int c = j % 3, h = j / 3 / tiles, odd = first + h, col = j / 3 % tiles * XC + p;
      const bool ok = col < kt;
      float2 v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e)
        v[e] = ok ? s_yz[c * C::FIELD + (h * R + t + T * e) * LD + col] : make_float2(0.f, 0.f);
      half_rows_fwd<N, XC>(v, odd, xs + p, t, tw);
      if (ok) {
#pragma unroll
        for (int e = 0; e < 8; ++e) db[c * ds + (long long)(odd * R + t + T * e) * kt + col] = v[e];
      }
      __syncwarp();
    }
  }
}

// ------------------------------------------------------------------------------
// Whole RK4 steps of a 2D grid up to 32^2, one CTA per trajectory: the six fields of a
// stage (31 KB at 32^2), its field and the accumulator on the band fit shared memory, and a
// thread keeps the step's initial state of its modes in registers, so nsteps steps (up to
// kStep2dSteps) are one launch that reads and writes the state once. A stage is the transforms
// and the combination of kx_stage and the lines of k_yz_plane (the plane's rows are x here, its
// columns the half axis), four block barriers in place of two launches. Ten steps at 32^2 x 9 took 266 us by
// kx_stage and 82 us a single step from the start of plain launches; here 152 and 18 us. At
// 64^2 one SM's issue rate is the bound (46 us a step; kx_stage over 17 SMs 33 us).
// ------------------------------------------------------------------------------
constexpr int kStep2dMax = 32;
// Steps of one launch: 1024 take some 15 ms, so that a long run is not one kernel that nothing
// else gets in between, and the stages' count stays far from overflow; the state's trip through
// memory per launch is nothing beside them.
constexpr int kStep2dSteps = 1024;

template <int N>
struct Step2dCfg {
  using Y = YzCfg<N>;
  static constexpr int MODES = N * Y::H;
  static constexpr int PER = (MODES + Y::THREADS - 1) / Y::THREADS;  // modes per thread
  // the stage field and the accumulator live on the band only: [component][kx + KD][kh < KT]
  static constexpr int KD = (N + 1) / 3, KT = (KD + 8) / 8 * 8;  // the plan's kd, kt at N = 16, 32
  static constexpr int BAND = (2 * KD + 1) * KT;
  static constexpr int SMEM = Y::SMEM + 2 * 3 * BAND * (int)sizeof(float2);
};

struct Step2d {
  long long cs;
  int nsteps;
  float a_dt[4], b_dt[4];
  EpiParams prm;  // what the stages share
  double inv_n2d, eps_inj;
  const float* nu_b;
  int* err;
};

template <int N>
__global__ void __launch_bounds__(YzCfg<N>::THREADS)
k_step2d(float2* __restrict__ S, const __grid_constant__ Step2d a, float s2, const float2* __restrict__ tw,
         const float2* __restrict__ ct8) {
  pdl_begin();
  using C = YzCfg<N>;
  using K = Step2dCfg<N>;
  constexpr int T = C::T, XC = C::XC, H = C::H, LD = C::LD, PER = K::PER;
  extern __shared__ __align__(16) float2 s_step[];
  __shared__ double red[32];
  __shared__ double s_scale;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float2* xs = s_step + 6 * C::FIELD + warp * C::XS;
  float2* us = s_step + 6 * C::FIELD + C::WARPS * C::XS;  // stage field and, behind it, accumulator
  float2* acc = us + 3 * K::BAND;
  float2* Sb = S + (long long)blockIdx.x * 3 * a.cs;
  constexpr int kd = K::KD, kt = K::KT;
  constexpr unsigned ukd = 2u * (unsigned)kd;
  EpiParams prm = a.prm;
  prm.nu = a.nu_b[blockIdx.x];
  // this thread's modes threadIdx.x + i THREADS
  auto row_of = [&](int i) { return (int)(threadIdx.x + i * C::THREADS) / H; };
  auto col_of = [&](int i) { return (int)(threadIdx.x + i * C::THREADS) % H; };
  auto has = [&](int i) { return (int)(threadIdx.x + i * C::THREADS) < K::MODES; };
  float2 u0[PER][3];
  // the stage field of mode i: kept on the band, and with its curl put on the plane
  auto open = [&](int i, const float2 (&v)[3]) {
    const int row = row_of(i), kh = col_of(i), kxb = kfull(row, N) + kd;
    if (kh < kt && (unsigned)kxb <= ukd) {
#pragma unroll
      for (int c = 0; c < 3; ++c) us[c * K::BAND + kxb * kt + kh] = v[c];
    }
    float2* f = s_step + row * LD + kh;
    float k0, k1, k2;
    kvec<2>(kfull(row, N), 0, kh, k0, k1, k2);
#pragma unroll
    for (int c = 0; c < 3; ++c) f[c * C::FIELD] = v[c];
    f[3 * C::FIELD] = mul_i<kInv>(make_float2(k1 * v[2].x - k2 * v[1].x, k1 * v[2].y - k2 * v[1].y));
    f[4 * C::FIELD] = mul_i<kInv>(make_float2(k2 * v[0].x - k0 * v[2].x, k2 * v[0].y - k0 * v[2].y));
    f[5 * C::FIELD] = mul_i<kInv>(make_float2(k0 * v[1].x - k1 * v[0].x, k0 * v[1].y - k1 * v[0].y));
  };
  // x transforms of the first cols columns of nf fields, in place, 32 / T columns per warp
  const int p = lane % XC, t = lane / XC;
  auto x_pass = [&](auto dir, int nf, int cols) {
    constexpr int D = decltype(dir)::value;
    const int jobs = nf * ((cols + XC - 1) / XC);
    for (int j = warp; j < jobs; j += C::WARPS) {
      const int f = j % nf, col = j / nf * XC + p;
      const bool ok = col < cols;
      float2* q = s_step + f * C::FIELD + t * LD + (ok ? col : 0);
      float2 v[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = ok ? q[T * e * LD] : make_float2(0.f, 0.f);
      block_fft<N, 8, D, XC, kSyncWarp>(v, xs + p, t, tw, 1);
      if (ok) {
#pragma unroll
        for (int e = 0; e < 8; ++e) q[T * e * LD] = v[e];
      }
      __syncwarp();
    }
  };
#pragma unroll
  for (int i = 0; i < PER; ++i) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
      u0[i][c] = has(i) ? Sb[c * a.cs + threadIdx.x + i * C::THREADS] : make_float2(0.f, 0.f);
    if (has(i)) open(i, u0[i]);
  }
  bool bad = false;
#pragma unroll 1
  for (int q = 0; q < 4 * a.nsteps; ++q) {
    const int rk = q & 3;
    __syncthreads();
    x_pass(Dir<kInv>{}, 6, H);
    __syncthreads();
    plane_lines<N>(s_step, xs, kt, kd, s2, ct8);
    __syncthreads();
    x_pass(Dir<kFwd>{}, 3, kt);
    float fscale = 0.f;
    if (prm.band_kf2 > 0) {  // constant-power coefficient of the stage field
      double lo = 0.0;
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int kx = kfull(row_of(i), N), kh = col_of(i), ik2 = kx * kx + kh * kh;
        if (!has(i) || ik2 == 0 || ik2 > prm.band_kf2) continue;  // kf <= N/4 < kd
        const int wg = kh == 0 || kh == N / 2 ? 1 : 2;
        for (int c = 0; c < 3; ++c) {
          const float2 v = us[c * K::BAND + (kx + kd) * kt + kh];
          lo += wg * ((double)v.x * v.x + (double)v.y * v.y);
        }
      }
      for (int o = 16; o > 0; o >>= 1) lo += __shfl_xor_sync(0xffffffffu, lo, o);
      if (lane == 0) red[warp] = lo;
      __syncthreads();
      if (threadIdx.x == 0) {
        double sum = 0.0;
        for (int i = 0; i < C::WARPS; ++i) sum += red[i];
        s_scale = a.eps_inj / (2.0 * (0.5 * sum * a.inv_n2d) + 1e-30);
      }
    }
    __syncthreads();
    if (prm.band_kf2 > 0) fscale = (float)s_scale;
    prm.rk = rk;
    prm.a_dt = a.a_dt[rk];
    prm.b_dt = a.b_dt[rk];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      if (!has(i)) continue;
      const int row = row_of(i), kh = col_of(i), kx = kfull(row, N);
      const int ik2 = kx * kx + kh * kh;
      float2 nv[3];
      if (kh < kt && (unsigned)(kx + kd) <= ukd) {
        const float2* f = s_step + row * LD + kh;
        const bool keep = kh <= kd;
        float2 d[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) d[c] = keep ? f[c * C::FIELD] : make_float2(0.f, 0.f);
        const float k0 = (float)kx, k1 = (float)kh;
        const float inv = 1.0f / (ik2 == 0 ? 1.0f : (float)ik2);
        const float pr = (d[0].x * k0 + d[1].x * k1) * inv, pi_ = (d[0].y * k0 + d[1].y * k1) * inv;
        d[0] = make_float2(d[0].x - pr * k0, d[0].y - pi_ * k0);
        d[1] = make_float2(d[1].x - pr * k1, d[1].y - pi_ * k1);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int o = c * K::BAND + (kx + kd) * kt + kh;
          const float2 ra = rk_core_r<N, 2, false>(row, 0, kh, ik2, c, d[c], us[o], rk >= 2 ? acc[o] : d[c], u0[i][c], prm,
                                                   fscale, nv[c]);
          if (rk == 1 || rk == 2) acc[o] = ra;
        }
      } else {
        const float z = (prm.nu * (float)ik2 + prm.drag) * prm.dt;
        const float f = lin_stage_factor(rk, z);
#pragma unroll
        for (int c = 0; c < 3; ++c) nv[c] = make_float2(f * u0[i][c].x, f * u0[i][c].y);
      }
      if (rk == 3) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          u0[i][c] = nv[c];
          bad |= !isfinite(nv[c].x + nv[c].y);
        }
      }
      open(i, nv);
    }
  }
  if (bad) atomicOr(a.err, kErrNonFinite);
#pragma unroll
  for (int i = 0; i < PER; ++i)
    if (has(i)) {
#pragma unroll
      for (int c = 0; c < 3; ++c) Sb[c * a.cs + threadIdx.x + i * C::THREADS] = u0[i][c];
    }
}

// Constant-power coefficient of a stage field (one CTA per trajectory): the low modes of
// S (stage 0) or T.
template <int DIM>
__global__ void __launch_bounds__(256)
k_band_coefficient(const float2* __restrict__ us, long long cs, int N, int kf, double inv_n2d, double eps_inj,
                   double* __restrict__ band_scale) {
  pdl_begin();
  band_coefficient<DIM, 256>(us + (long long)blockIdx.x * 3 * cs, cs, N, kf, inv_n2d, eps_inj, 1e-30,
                             band_scale + blockIdx.x);
}

}  // namespace l3es
