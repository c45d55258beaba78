// Host launch wrappers for the DNS kernels of one grid size N. Each dns_n*.cu
// translation unit instantiates make_dns_table<N>() for its sizes, so the sizes
// compile in parallel.
#pragma once

#include "l3es_internal.h"

namespace l3es {

template <int N>
struct DnsOps {
  static constexpr int H = N / 2 + 1;
  static constexpr int TX = TW * Fft<N>::T;  // threads of the strided x passes
  // 2D x passes in narrow tiles (schedule entry [0] in 2D): XN columns per CTA, so a
  // 256^2 field's 129 columns spread over 65 CTAs instead of 17
  static constexpr int XN = 2;
  static constexpr int TXN = XN * Fft<N>::T;
  using L = LineCfg<N>;
  using KY = KyCfg<N>;
  static constexpr unsigned ky_tiles(int ncols) { return (unsigned)((ncols + KY::TWY - 1) / KY::TWY); }

  static unsigned line_blocks(long long lines) { return (unsigned)((lines + L::LPC - 1) / L::LPC); }

  // persistent CTAs of the bulk-copy x inverse pass (0: use kx_inv)
  static inline int tma_ctas = 0;

  static inline int tma_band_ctas = 0;
  static inline int tma_plain_ctas = 0;  // x inverse without curl (irfftn)
  static inline int tma_band_fused_ctas = 0;  // band pass of the band-fused RK step

  // resident CTAs (all SMs) of a persistent kernel with K::SMEM dynamic shared memory
  template <typename F>
  static int persistent_ctas(F kernel) {
    int nb = 0;
    const int smem = KxTma<N>::SMEM;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, TX, smem) == cudaSuccess)
      return nb * sm_count();
    cudaGetLastError();
    return 0;
  }

  static inline bool lc3_staged_ok = false;  // dynamic shared memory of the staged line pass granted

  static void init_attrs() {
    if constexpr (N == 256) {
      lc3_staged_ok = cudaFuncSetAttribute(line_cross3<N, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           Line3Cfg<N>::SMEM_STAGED) == cudaSuccess &&
                      cudaFuncSetAttribute(line_cross3<N, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           Line3Cfg<N>::SMEM_STAGED) == cudaSuccess;
      cudaGetLastError();
    }
    if constexpr (N >= 64) {
      tma_ctas = persistent_ctas(kx_inv_tma<N, true, true>);
      tma_band_ctas = persistent_ctas(kx_fwd_band_tma<N>);
      tma_plain_ctas = persistent_ctas(kx_inv_tma<N, false>);
    }
    if constexpr (N > kStageMax3d) {
      tma_band_fused_ctas = persistent_ctas(kx_fwd_band_tma<N, true>);
    }
    if constexpr (N > kStep2dMax) stage_attrs<2>();
    if constexpr (N >= 16 && N <= kStep2dMax) {
      cudaFuncSetAttribute(k_step2d<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, Step2dCfg<N>::SMEM);
      cudaGetLastError();
    }
    if constexpr (N >= 16 && N <= kStageMax3d) {
      stage_attrs<3>();
      if constexpr (yz_by_halves(N)) {
        cudaFuncSetAttribute(k_yz_half<N, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, YzHalfCfg<N, 1>::SMEM);
        cudaFuncSetAttribute(k_yz_half<N, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, YzHalfCfg<N, 2>::SMEM);
      } else {
        cudaFuncSetAttribute(k_yz_plane<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, YzCfg<N>::SMEM);
      }
      cudaGetLastError();
    }
  }

  // kx_stage's shape: columns per CTA and values per thread in each transform
  template <int DIM>
  static constexpr int XS = DIM == 2 ? XN : TW;
  template <int DIM>
  static constexpr int ES = N <= (DIM == 2 ? 64 : 32) ? 4 : 8;
  template <int DIM>
  using Stage = XStageCfg<N, XS<DIM>, ES<DIM>>;

  template <int DIM>
  static void stage_attrs() {
    if constexpr (Stage<DIM>::SMEM > 48 * 1024) {
      auto set = [](auto kernel) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Stage<DIM>::SMEM);
      };
      set(kx_stage<N, DIM, XS<DIM>, ES<DIM>, -1, true>);
      set(kx_stage<N, DIM, XS<DIM>, ES<DIM>, 0, true>);
      set(kx_stage<N, DIM, XS<DIM>, ES<DIM>, 1, true>);
      set(kx_stage<N, DIM, XS<DIM>, ES<DIM>, 2, true>);
      set(kx_stage<N, DIM, XS<DIM>, ES<DIM>, 3, true>);
      set(kx_stage<N, DIM, XS<DIM>, ES<DIM>, 3, false>);
      cudaGetLastError();
    }
  }

  // y pass of `nz` fields (columns [0, ncols) of rows of ncols values) in the plan's
  // y schedule (KyCfg variant)
  template <int DIR>
  static void y_pass(const Ctx& c, int kind, double bytes, float2* w, long long fs, int ncols, int kd_store, int nz,
                     cudaStream_t s) {
    const dim3 g(ky_tiles(ncols), N, nz);
    if (c.sched.y_var == 1)
      L3ES_LAUNCH(c, kind, bytes, s,
                  pdl_launch(ky_pass<N, DIR, 1>, g, KyCfg<N, 1>::THREADS, 0, s, w, fs, ncols, ncols, kd_store, c.tw));
    else
      L3ES_LAUNCH(c, kind, bytes, s, pdl_launch(ky_pass<N, DIR, 0>, g, KY::THREADS, 0, s, w, fs, ncols, ncols,
                                                kd_store, c.tw));
  }

  // the RHS's y inverse (six one-FFT jobs per tile) in the plan's y schedule
  static void y_inv_rhs(const Ctx& c, double bytes, cudaStream_t s) {
    const dim3 g(6 * ky_tiles(H), N, c.batch);
    if (c.sched.y_var == 1)
      L3ES_LAUNCH(c, KK_Y_INV, bytes, s, pdl_launch(ky_inv_rhs<N, 1>, g, KyCfg<N, 1>::THREADS, 0, s, c.W, c.Wx, c.fs,
                                                    c.tw));
    else
      L3ES_LAUNCH(c, KK_Y_INV, bytes, s, pdl_launch(ky_inv_rhs<N, 0>, g, KY::THREADS, 0, s, c.W, c.Wx, c.fs, c.tw));
  }

  // x inverse pass with curl prologue: us -> W (6 fields); xl: the x inverse of a
  // band-fused RK stage (us is then the state xl->S)
  template <int DIM>
  static void x_inverse(const Ctx& c, const float2* us, double bytes, cudaStream_t s, const XLin* xl = nullptr) {
    const long long mc = c.nmid * H;
    if constexpr (DIM == 3 && N >= 64) {
      CUtensorMap map;
      const unsigned long long dims[3] = {(unsigned long long)mc, N, 3ull * c.batch};
      const unsigned long long strides[2] = {8ull * mc, 8ull * c.cs};
      const unsigned box[3] = {TW, KxTma<N>::NY, 3};
      // (the scaling of a band-fused stage always runs in the one-tile kernel, which has no
      // register cap: per 256^3 launch 116 against 127 us, 512^3 1140 against 1360 us)
      if (!xl && c.sched.x_bulk && tma_ctas > 0 && tma_encode(&map, us, 3, dims, strides, box)) {
        const int ntiles = (int)(mc / TW);
        const int gx = std::max(1, std::min(ntiles, tma_ctas / c.batch));
        L3ES_LAUNCH(c, KK_X_INV, bytes, s,
                    pdl_launch(kx_inv_tma<N, true, true>, dim3(gx, c.batch), TX, KxTma<N>::SMEM, s, map, c.W, c.fs,
                               c.tw, ntiles, c.err, c.Wx));
        return;
      }
    }
    if constexpr (DIM == 2) {
      if (c.sched.x_bulk) {
        const dim3 gn((unsigned)((mc + XN - 1) / XN), c.batch);
        L3ES_LAUNCH(c, KK_X_INV, bytes, s,
                    pdl_launch(kx_inv<N, 2, true, false, false, XN>, gn, TXN, 0, s, us, c.cs, c.W, c.fs, c.tw, c.Wx,
                               XLin{}, nullptr));
        return;
      }
    }
    const dim3 g((unsigned)((mc + TW - 1) / TW), c.batch);
    if constexpr (DIM == 3 && N > kStageMax3d)
      if (xl) {
        L3ES_LAUNCH(c, KK_X_INV, bytes, s,
                    pdl_launch(kx_inv<N, 3, true, true, true>, g, TX, 0, s, us, c.cs, c.W, c.fs, c.tw, c.Wx, *xl,
                               c.err));
        return;
      }
    L3ES_LAUNCH(c, KK_X_INV, bytes, s,
                pdl_launch(kx_inv<N, DIM, true, DIM == 3>, g, TX, 0, s, us, c.cs, c.W, c.fs, c.tw, c.Wx, XLin{},
                           nullptr));
  }

  // W (u, curl u after the x inverse) -> DU (the nonlinear term before its x transform):
  // y inverse, half-axis line pass, y forward
  template <int DIM>
  static void nonlinear(const Ctx& c, cudaStream_t s) {
    const long long lines = c.nmid * N;
    const float scale = (float)(1.0 / (DIM == 3 ? (double)N * N * N : (double)N * N));
    const double B = c.batch, A = 8.0 * 3.0 * c.cs * B;  // bytes of one 3-component spectrum
    const double Adu = 8.0 * 3.0 * c.ds * B;               // bytes of the truncated DU field
    const double rows = DIM == 3 ? (2.0 * c.kd + 1.0) / N : 1.0;  // kept y rows
    if (DIM == 3) y_inv_rhs(c, 11.0 / 3.0 * A, s);
    bool line_done = false;
    if constexpr (N >= 64 && N <= 256) {  // two real lines per complex FFT, persistent
      if constexpr (N == 256) {
        if (c.sched.line_pair >= 2) {  // radix-16 lines, 16 lanes per line
          using L3 = Line3Cfg<N>;
          const float s2 = 0.5f * scale * scale;
          const long long tiles = (lines + L3::LPC - 1) / L3::LPC;
          if (c.sched.line_pair == 3 && lc3_staged_ok && lines % L3::LPC == 0)
            L3ES_LAUNCH(c, KK_LINE_CROSS, 2.0 * A + Adu, s,
                        pdl_launch(tiles * c.batch <= c.sms ? line_cross3<N, true, true> : line_cross3<N, true>,
                                   dim3((unsigned)tiles, c.batch), L3::THREADS, L3::SMEM_STAGED, s, c.W, c.fs, c.DU,
                                   c.ds, c.kt, c.kd, s2, c.tw + line2_ct_offset<N>(),
                                   c.tw + line3_ct16_offset<N>(), (int)lines, c.err));
          else
            L3ES_LAUNCH(c, KK_LINE_CROSS, 2.0 * A + Adu, s,
                        pdl_launch(line_cross3<N, false>, dim3((unsigned)tiles, c.batch), L3::THREADS, 0, s, c.W,
                                   c.fs, c.DU, c.ds, c.kt, c.kd, s2, c.tw + line2_ct_offset<N>(),
                            c.tw + line3_ct16_offset<N>(), (int)lines, c.err));
          line_done = true;
        }
      }
      if (!line_done && c.sched.line_pair) {
        using L2 = Line2Cfg<N>;
        const float s2 = 0.5f * scale * scale;
        const long long tiles = (lines + L2::LPC - 1) / L2::LPC;
        L3ES_LAUNCH(c, KK_LINE_CROSS, 2.0 * A + Adu, s,
                    pdl_launch(line_cross2<N>, dim3((unsigned)tiles, c.batch), L2::THREADS, 0, s, c.W, c.fs, c.DU,
                               c.ds, c.kt, c.kd, s2, c.tw + line2_ct_offset<N>(), (int)lines));
        line_done = true;
      }
    }
    if (!line_done)
      L3ES_LAUNCH(c, KK_LINE_CROSS, 2.0 * A + Adu, s,
                  pdl_launch(line_cross<N>, dim3(line_blocks(lines), c.batch), L::THREADS, 0, s, c.W, c.fs, c.DU,
                             c.ds, c.kt, c.kd, scale, c.tw, (int)lines));
    if (DIM == 3) y_pass<kFwd>(c, KK_Y_FWD, Adu * (1.0 + rows), c.DU, c.ds, c.kt, c.kd, 3 * c.batch, s);
  }

  // us: field the RHS is evaluated on; S: state; out: RK stage field (or du for rk=-1)
  template <int DIM>
  static void stage_dim(const Ctx& c, const float2* us, float2* S, float2* out, int rk, const EpiParams& prm,
                        cudaStream_t s) {
    const double B = c.batch, A = 8.0 * 3.0 * c.cs * B;  // bytes of one 3-component spectrum
    const double Adu = 8.0 * 3.0 * c.ds * B;               // bytes of the truncated DU field
    const double rows = DIM == 3 ? (2.0 * c.kd + 1.0) / N : 1.0;  // kept y rows
    const double inv_n2d = 1.0 / (DIM == 3 ? std::pow((double)N, 6) : std::pow((double)N, 4));
    // band-fused RK step (XLin): us == S; fb = the band's share of the modes
    const bool fused = DIM == 3 && N > kStageMax3d && prm.band_rk && rk >= 0;
    const double fb = (double)c.pcs / (double)c.cs;
    XLin xl{};
    if (fused) {
      xl.S = S;
      xl.cs = c.cs;
      xl.nu_b = c.nu_b;
      xl.drag = prm.drag;
      xl.dt = prm.dt;
      xl.kd = c.kd;
      xl.kt = c.kt;
      xl.rk = rk;
      xl.band_kf = prm.band_kf2 > 0 ? c.kf : 0;
      xl.inv_n2d = inv_n2d;
      xl.eps_inj = c.eps_inj;
      xl.band_scale = c.band;
    }
    // 3D: the x pass stores u_x, curl_y, curl_z in W and u_y, u_z in the side buffer
    // Wx (curl_x is not stored); the y pass writes all six fields of W. The last
    // band-fused stage also writes the new state outside the band.
    x_inverse<DIM>(c, us, (DIM == 3 ? 8.0 : 9.0) / 3.0 * A + (fused && rk == 3 ? (1.0 - fb) * A : 0.0), s,
                   fused ? &xl : nullptr);
    nonlinear<DIM>(c, s);
    // band x-FFT + projection into P, then the elementwise RK update
    const int nb = 2 * c.kd + 1;
    const double Ap = 8.0 * 3.0 * c.pcs * B;
    if constexpr (DIM == 3 && N > kStageMax3d) if (fused) {
      // the stage combination on the band: rk 0 reads S and writes P (= u0) and S; rk 1
      // reads S, P and writes acc, S; rk 2 reads S, P, acc and writes acc, S; rk 3 reads
      // S, acc and writes S
      const BandRk br{S, c.C, c.cs, prm, c.band, c.nu_b, c.err};
      const double bb = Adu * rows + Ap * (rk == 0 ? 3.0 : rk == 1 ? 4.0 : rk == 2 ? 5.0 : 3.0);
      {
        const bool bulk = c.sched.band_bulk < 0 ? N == 256 : c.sched.band_bulk != 0;
        CUtensorMap map;
        const unsigned long long dims[4] = {(unsigned long long)c.kt, N, N, 3ull * c.batch};
        const unsigned long long strides[3] = {8ull * c.kt, 8ull * N * c.kt, 8ull * c.ds};
        const unsigned box[4] = {TW, 1, KxTma<N>::NY, 3};
        if (bulk && tma_band_fused_ctas > 0 && tma_encode(&map, c.DU, 4, dims, strides, box)) {
          const int ntiles = (c.kt / TW) * nb;
          const int gx = std::max(1, std::min(ntiles, tma_band_fused_ctas / c.batch));
          L3ES_LAUNCH(c, KK_X_EPI, bb, s,
                      pdl_launch(kx_fwd_band_tma<N, true>, dim3(gx, c.batch), TX, KxTma<N>::SMEM, s, map, c.kt, c.kd,
                                 c.P, c.pcs, c.tw, us, c.cs, 0, inv_n2d, c.eps_inj, c.band, c.err, br));
          return;
        }
      }
      L3ES_LAUNCH(c, KK_X_EPI, bb, s,
                  pdl_launch(kx_fwd_band<N, 3, true>, dim3(c.kt / TW, nb, c.batch), TX, 0, s, c.DU, c.ds, c.kt, c.kd,
                             c.P, c.pcs, c.tw, us, c.cs, 0, inv_n2d, c.eps_inj, c.band, br));
      return;
    }
    // (block 0 of each trajectory also computes the constant-power coefficient of us)
    bool band_done = false;
    // by default at 256^3: smaller grids have too few band tiles per persistent CTA to
    // pipeline (a band-fused step at 128^3: 309 us persistent, 286 us one-shot), at 512^3 a
    // CTA fills its SM either way (20.1 ms persistent, 19.7 ms one-shot; 256^3 2053, 2069 us)
    if constexpr (DIM == 3 && N >= 64) {
      const bool bulk = c.sched.band_bulk < 0 ? N == 256 : c.sched.band_bulk != 0;
      CUtensorMap map;
      const unsigned long long dims[4] = {(unsigned long long)c.kt, N, N, 3ull * c.batch};
      const unsigned long long strides[3] = {8ull * c.kt, 8ull * N * c.kt, 8ull * c.ds};
      const unsigned box[4] = {TW, 1, KxTma<N>::NY, 3};
      if (bulk && tma_band_ctas > 0 && tma_encode(&map, c.DU, 4, dims, strides, box)) {
        const int ntiles = (c.kt / TW) * nb;
        const int gx = std::max(1, std::min(ntiles, tma_band_ctas / c.batch));
        L3ES_LAUNCH(c, KK_X_EPI, Adu * rows + Ap, s,
                    pdl_launch(kx_fwd_band_tma<N>, dim3(gx, c.batch), TX, KxTma<N>::SMEM, s, map, c.kt, c.kd, c.P,
                               c.pcs, c.tw, us, c.cs, prm.band_kf2 > 0 ? c.kf : 0, inv_n2d,
                        c.eps_inj, c.band, c.err, BandRk{}));
        band_done = true;
      }
    }
    if (!band_done && DIM == 2 && c.sched.x_bulk)
      L3ES_LAUNCH(c, KK_X_EPI, Adu * rows + Ap, s,
                  pdl_launch(kx_fwd_band<N, DIM, false, XN>, dim3(c.kt / XN, 1, c.batch), TXN, 0, s, c.DU, c.ds, c.kt,
                             c.kd, c.P, c.pcs, c.tw, us, c.cs, prm.band_kf2 > 0 ? c.kf : 0, inv_n2d,
                      c.eps_inj, c.band, BandRk{}));
    else if (!band_done)
      L3ES_LAUNCH(c, KK_X_EPI, Adu * rows + Ap, s,
                  pdl_launch(kx_fwd_band<N, DIM>, dim3(c.kt / TW, DIM == 3 ? nb : 1, c.batch), TX, 0, s, c.DU, c.ds,
                             c.kt, c.kd, c.P, c.pcs, c.tw, us, c.cs, prm.band_kf2 > 0 ? c.kf : 0, inv_n2d,
                      c.eps_inj, c.band, BandRk{}));
    // rk -1: us -> du; 0: us -> out; 1: us, u0 -> acc, out; 2: us, u0, acc -> acc, out;
    // 3: us, acc -> fin
    double upd = Ap + A * (rk < 0 ? 2.0 : rk == 0 ? 2.0 : rk == 1 ? 4.0 : rk == 2 ? 5.0 : 3.0);
    if (prm.lin && rk >= 0 && !(prm.if_h > 0.f)) {  // outside the stage region: u0 in, one field out
      const double fr = DIM == 3 ? (2.0 * c.kd + 1.0) / N : (double)c.kt / H;
      upd = Ap + A * (fr * (rk == 0 ? 2.0 : rk == 1 ? 4.0 : rk == 2 ? 5.0 : 3.0) + (1.0 - fr) * 2.0);
    }
    const long long pairs = 3 * c.cs / 2;
    const dim3 ug((unsigned)((pairs + 255) / 256), c.batch);
    if (prm.lin && rk >= 0 && !(prm.if_h > 0.f))
      L3ES_LAUNCH(c, KK_RK_UPDATE, upd, s,
                  pdl_launch(k_rk_update_lin<N, DIM>, ug, 256, 0, s, c.P, c.pcs, c.kt, c.kd, us, S, c.C, out, S, c.cs,
                             prm,
                                                            c.band, c.nu_b, c.err));
    else if (prm.if_h > 0.f && rk >= 0)
      L3ES_LAUNCH(c, KK_RK_UPDATE, upd, s,
                  pdl_launch(k_rk_update<N, DIM, true>, ug, 256, 0, s, c.P, c.pcs, c.kt, c.kd, us, S, c.C, out, S,
                             c.cs, prm,
                                                                c.band, c.nu_b, c.err));
    else
      L3ES_LAUNCH(c, KK_RK_UPDATE, upd, s,
                  pdl_launch(k_rk_update<N, DIM>, ug, 256, 0, s, c.P, c.pcs, c.kt, c.kd, us, S, c.C, out, S, c.cs, prm,
                                                          c.band, c.nu_b, c.err));
  }

  // One kx_stage launch: RK = -1 opens a step, RK = 0..3 closes that stage (XStage)
  template <int DIM, int RK, bool INV>
  static void x_stage(const Ctx& c, float2* S, const EpiParams& prm, cudaStream_t s) {
    const double A = 8.0 * 3.0 * c.cs * c.batch;
    // share of the columns (du is read there) and of the modes that the band holds
    const double fc = (DIM == 3 ? (2.0 * c.kd + 1.0) / N : 1.0) * c.kt / H, fb = (double)c.pcs / (double)c.cs;
    double b = INV ? (DIM == 3 ? 5.0 : 6.0) / 3.0 * A : 0.0;  // lines out
    if (RK < 0) b += A;
    if (RK == 0) b += (fc + 1.0 + fb) * A;              // du, S -> T
    if (RK == 1) b += (fc + 1.0 + 3.0 * fb) * A;        // du, S, T -> T, C
    if (RK == 2) b += (fc + 2.0 + 3.0 * fb) * A;        // du, S, T, C -> T, C, S outside the band
    if (RK == 3) b += (fc + 3.0 * fb + (INV ? 1.0 - fb : 0.0)) * A;  // du, T, C -> S
    if (RK >= 0 && prm.band_kf2 > 0) {
      const double inv_n2d = 1.0 / std::pow((double)N, 2 * DIM);
      L3ES_LAUNCH(c, KK_FORCE, 0.0, s,
                  pdl_launch(k_band_coefficient<DIM>, c.batch, 256, 0, s, RK == 0 ? S : c.Tb, c.cs, N, c.kf, inv_n2d,
                             c.eps_inj,
                                                                  c.band));
    }
    using K = Stage<DIM>;
    const XStage st{c.cs, c.kd, c.kt, prm, c.band, c.nu_b, c.err};
    const dim3 g((unsigned)((c.nmid * H + XS<DIM> - 1) / XS<DIM>), c.batch);
    L3ES_LAUNCH(c, KK_X_STAGE, b, s,
                pdl_launch(kx_stage<N, DIM, XS<DIM>, ES<DIM>, RK, INV>, g, K::THREADS, K::SMEM, s, c.DU, c.ds, S,
                           c.Tb, c.C, st, c.W, c.Wx, c.fs, c.tw));
  }

  // Whether two CTAs share a plane between two kx_stage launches (k_yz_half): while the
  // doubled grid still has an SM per CTA. Ten steps with one CTA per plane and with two:
  // 64^3 640 and 513 us, 32^3 342 and 320, 32^3 x 2 419 and 365; 64^3 x 2 802 and 901, 32^3 x 8
  // 501 and 602 (between them 32^3 x 3 and x 4 would gain a little from two: 437 and 430, 484 and
  // 428).
  static bool two_ctas(const Ctx& c) { return 2LL * N * c.batch <= c.sms; }

  // W -> DU between two kx_stage launches: in 3D one kernel per x plane
  template <int DIM>
  static void between(const Ctx& c, cudaStream_t s) {
    if constexpr (DIM == 3 && N >= 16 && N <= kStageMax3d) {
      const double A = 8.0 * 3.0 * c.cs * c.batch, Adu = 8.0 * 3.0 * c.ds * c.batch;
      const float scale = (float)(1.0 / ((double)N * N * N));
      const double bytes = 5.0 / 3.0 * A + Adu * (yz_by_halves(N) ? 1.0 : (2.0 * c.kd + 1.0) / N);
      const float2* ct = c.tw + line2_ct_offset<N>();
      const float s2 = 0.5f * scale * scale;
      if constexpr (yz_by_halves(N)) {
        using Y1 = YzHalfCfg<N, 1>;
        using Y2 = YzHalfCfg<N, 2>;
        if (two_ctas(c))
          L3ES_LAUNCH(c, KK_YZ_PLANE, bytes, s,
                      pdl_launch(k_yz_half<N, 2>, dim3(2 * N, c.batch), Y2::THREADS, Y2::SMEM, s, c.W, c.Wx, c.fs,
                                 c.DU, c.ds, c.kt, c.kd, s2, c.tw, ct));
        else
          L3ES_LAUNCH(c, KK_YZ_PLANE, bytes, s,
                      pdl_launch(k_yz_half<N, 1>, dim3(N, c.batch), Y1::THREADS, Y1::SMEM, s, c.W, c.Wx, c.fs, c.DU,
                                 c.ds, c.kt, c.kd, s2, c.tw, ct));
      } else {
        L3ES_LAUNCH(c, KK_YZ_PLANE, bytes, s,
                    pdl_launch(k_yz_plane<N>, dim3(N, c.batch), YzCfg<N>::THREADS, YzCfg<N>::SMEM, s, c.W, c.Wx, c.fs,
                               c.DU, c.ds, c.kt, c.kd, s2, c.tw, ct));
      }
    } else if constexpr (DIM == 2 && N > kStep2dMax && N <= 128) {
      const double A = 8.0 * 3.0 * c.cs * c.batch, Adu = 8.0 * 3.0 * c.ds * c.batch;
      const float scale = (float)(1.0 / ((double)N * N));
      constexpr int LPC = 128 / (N / 8);
      L3ES_LAUNCH(c, KK_LINE_CROSS, 2.0 * A + Adu, s,
                  pdl_launch(line_cross_slots<N>, dim3((N + LPC - 1) / LPC, c.batch), 128, 0, s, c.W, c.fs, c.DU, c.ds,
                             c.kt, c.kd, 0.5f * scale * scale, c.tw + line2_ct_offset<N>(), N));
    } else {
      nonlinear<DIM>(c, s);
    }
  }

  // One RK4 step in place on S by kx_stage (stage_kernels.cuh). first: the x inverse of S
  // is not in W yet; last: nothing follows that needs the new state's.
  template <int DIM>
  static void step_dim(const Ctx& c, float2* S, const EpiParams* prm, bool first, bool last, cudaStream_t s) {
    if constexpr (DIM == 2 ? N > kStep2dMax : N >= 16 && N <= kStageMax3d) {
      if (first) x_stage<DIM, -1, true>(c, S, prm[0], s);
      between<DIM>(c, s);
      x_stage<DIM, 0, true>(c, S, prm[0], s);
      between<DIM>(c, s);
      x_stage<DIM, 1, true>(c, S, prm[1], s);
      between<DIM>(c, s);
      x_stage<DIM, 2, true>(c, S, prm[2], s);
      between<DIM>(c, s);
      if (last)
        x_stage<DIM, 3, false>(c, S, prm[3], s);
      else
        x_stage<DIM, 3, true>(c, S, prm[3], s);
    }
  }

  // nsteps RK4 steps of a 2D grid in one launch (k_step2d)
  static void steps2d(const Ctx& c, float2* S, const EpiParams* prm, int nsteps, cudaStream_t s) {
    if constexpr (N >= 16 && N <= kStep2dMax) {
      Step2d a{};
      a.cs = c.cs;
      a.nsteps = nsteps;
      a.prm = prm[0];
      for (int rk = 0; rk < 4; ++rk) {
        a.a_dt[rk] = prm[rk].a_dt;
        a.b_dt[rk] = prm[rk].b_dt;
      }
      a.inv_n2d = 1.0 / std::pow((double)N, 4);
      a.eps_inj = c.eps_inj;
      a.nu_b = c.nu_b;
      a.err = c.err;
      const float scale = (float)(1.0 / ((double)N * N));
      L3ES_LAUNCH(c, KK_X_STAGE, 2.0 * 8.0 * 3.0 * c.cs * c.batch, s,
                  pdl_launch(k_step2d<N>, c.batch, YzCfg<N>::THREADS, Step2dCfg<N>::SMEM, s, S, a, 0.5f * scale * scale,
                             c.tw, c.tw + line2_ct_offset<N>()));
    }
  }

  static void step(const Ctx& c, float2* S, const EpiParams* prm, bool first, bool last, cudaStream_t s) {
    if (c.dim == 3)
      step_dim<3>(c, S, prm, first, last, s);
    else
      step_dim<2>(c, S, prm, first, last, s);
  }

  static void stage(const Ctx& c, const float2* us, float2* S, float2* out, int rk, const EpiParams& prm,
                    cudaStream_t s) {
    if (c.dim == 3)
      stage_dim<3>(c, us, S, out, rk, prm, s);
    else
      stage_dim<2>(c, us, S, out, rk, prm, s);
  }

  template <int DIM>
  static void irfftn_dim(const Ctx& c, const float2* uh, float* u, cudaStream_t s) {
    const long long mc = c.nmid * H;
    const long long lines = c.nmid * N;
    const float scale = (float)(1.0 / (DIM == 3 ? (double)N * N * N : (double)N * N));
    const double A = 8.0 * 3.0 * c.cs * c.batch, P = 4.0 * 3.0 * c.ps * c.batch;
    bool x_done = false;
    if constexpr (DIM == 3 && N >= 64) {  // persistent, next tile by one bulk tensor load
      CUtensorMap map;
      const unsigned long long dims[3] = {(unsigned long long)mc, N, 3ull * c.batch};
      const unsigned long long strides[2] = {8ull * mc, 8ull * c.cs};
      const unsigned box[3] = {TW, KxTma<N>::NY, 3};
      if (c.sched.x_bulk && tma_plain_ctas > 0 && tma_encode(&map, uh, 3, dims, strides, box)) {
        const int ntiles = (int)(mc / TW);
        const int gx = std::max(1, std::min(ntiles, tma_plain_ctas / c.batch));
        L3ES_LAUNCH(c, KK_X_INV_PLAIN, 2.0 * A, s,
                    pdl_launch(kx_inv_tma<N, false>, dim3(gx, c.batch), TX, KxTma<N>::SMEM, s, map, c.W, c.fs, c.tw,
                               ntiles,
                                                                                        c.err, nullptr));
        x_done = true;
      }
    }
    if (!x_done)
      L3ES_LAUNCH(c, KK_X_INV_PLAIN, 2.0 * A, s,
                  pdl_launch(kx_inv<N, DIM, false>, dim3((unsigned)((mc + TW - 1) / TW), c.batch), TX, 0, s, uh, c.cs,
                             c.W, c.fs, c.tw, nullptr, XLin{}, nullptr));
    if (DIM == 3) y_pass<kInv>(c, KK_Y_INV, 2.0 * A, c.W, c.fs, H, N / 2, 3 * c.batch, s);
    L3ES_LAUNCH(c, KK_LINE_C2R, A + P, s,
                pdl_launch(line_c2r<N>, dim3(line_blocks(lines), c.batch), L::THREADS, 0, s, c.W, c.fs, u, c.ps,
                           scale, c.tw, (int)lines));
  }

  static void irfftn(const Ctx& c, const float2* uh, float* u, cudaStream_t s) {
    if (c.dim == 3)
      irfftn_dim<3>(c, uh, u, s);
    else
      irfftn_dim<2>(c, uh, u, s);
  }

  template <int DIM>
  static void rfftn_dim(const Ctx& c, const float* u, float2* uh, cudaStream_t s) {
    const long long mc = c.nmid * H;
    const long long lines = c.nmid * N;
    const double A = 8.0 * 3.0 * c.cs * c.batch, P = 4.0 * 3.0 * c.ps * c.batch;
    L3ES_LAUNCH(c, KK_LINE_R2C, A + P, s,
                pdl_launch(line_r2c<N>, dim3(line_blocks(lines), c.batch), L::THREADS, 0, s, u, c.ps, c.W, c.fs, c.tw,
                           (int)lines));
    if (DIM == 3) y_pass<kFwd>(c, KK_Y_FWD, 2.0 * A, c.W, c.fs, H, N / 2, 3 * c.batch, s);
    L3ES_LAUNCH(c, KK_X_FWD_PLAIN, 2.0 * A, s,
                pdl_launch(kx_fwd_plain<N, DIM>, dim3((unsigned)((mc + TW - 1) / TW), c.batch), TX, 0, s, c.W, c.fs,
                           uh, c.cs, c.tw));
  }

  static void rfftn(const Ctx& c, const float* u, float2* uh, cudaStream_t s) {
    if (c.dim == 3)
      rfftn_dim<3>(c, u, uh, s);
    else
      rfftn_dim<2>(c, u, uh, s);
  }

  // Vector-Jacobian product of the RHS (adjoint_kernels.cuh): u/curl x-inverse,
  // projected-cotangent x-inverse (+ band terms), y inverse (3D), one line pass for
  // both products, y forward (3D), x forward, elementwise epilogue.
  template <int DIM>
  static void vjp_dim(const Ctx& c, const AdjEpi& a, float2* Wm, float2* Y6, cudaStream_t s) {
    const long long mc = c.nmid * H;
    const long long lines = c.nmid * N;
    const float scale = (float)(1.0 / (DIM == 3 ? (double)N * N * N : (double)N * N));
    const double A = 8.0 * 3.0 * c.cs * c.batch;  // bytes of one 3-component spectrum
    const unsigned xb = (unsigned)((mc + TW - 1) / TW);
    const double inv_n2d = 1.0 / (DIM == 3 ? std::pow((double)N, 6) : std::pow((double)N, 4));
    // u and curl u lines of the stage field: the forward RHS's x and y inverse passes, or
    // the lines the stage recomputation left (a.wlines)
    const float2* wuw = a.wlines ? a.wlines : c.W;
    if (!a.wlines) x_inverse<DIM>(c, a.us, (DIM == 3 ? 8.0 : 9.0) / 3.0 * A, s);
    const double Adu = 8.0 * 3.0 * c.ds * c.batch, rows = DIM == 3 ? (2.0 * c.kd + 1.0) / N : 1.0;
    const int nb = DIM == 3 ? 2 * c.kd + 1 : 1;
    L3ES_LAUNCH(c, KK_ADJ_X_INV, 8.0 * 3.0 * c.pcs * c.batch + Adu * rows, s,
                pdl_launch(kx_inv_adjproj<N, DIM>, dim3(c.kt / TW, nb, c.batch), TX, 0, s, a.g, c.cs, a.gscale, c.kd,
                           c.kt, Wm, c.ds, c.tw, a.us, a.band_kf2 > 0 ? c.kf : 0, inv_n2d, c.eps_inj,
                           const_cast<double*>(a.band_adj)));
    if (DIM == 3) {
      if (!a.wlines) y_inv_rhs(c, 11.0 / 3.0 * A, s);
      const dim3 g(ky_tiles(c.kt), N, 3 * c.batch);
      if (c.sched.y_var == 1)
        L3ES_LAUNCH(c, KK_Y_INV, Adu * (1.0 + rows), s,
                    pdl_launch(ky_inv_band<N, 1>, g, KyCfg<N, 1>::THREADS, 0, s, Wm, c.ds, c.kt, c.kd, c.tw));
      else
        L3ES_LAUNCH(c, KK_Y_INV, Adu * (1.0 + rows), s,
                    pdl_launch(ky_inv_band<N, 0>, g, KY::THREADS, 0, s, Wm, c.ds, c.kt, c.kd, c.tw));
    }
    L3ES_LAUNCH(c, KK_ADJ_LINE, 4.0 * A + Adu, s,
                pdl_launch(line_cross_adj<N>, dim3(line_blocks(lines), c.batch), L::THREADS, 0, s, Wm, c.ds, c.kt, wuw,
                           c.fs, Y6, c.cs, scale, c.tw, (int)lines));
    if (DIM == 3) y_pass<kFwd>(c, KK_Y_FWD, 4.0 * A, Y6, c.cs, H, N / 2, 6 * c.batch, s);
    // reads: 2 product spectra, g, lam1, lam_in; writes: lam_out, g_out
    const double epi = (3.0 + (a.lam1 ? 1.0 : 0.0) + (a.lam_in ? 1.0 : 0.0) + 1.0 + (a.g_out ? 1.0 : 0.0)) * A;
    if constexpr (DIM == 3 && N >= kAdjFusedMin3d) {
      L3ES_LAUNCH(c, KK_ADJ_EPI, epi, s,
                  pdl_launch(kx_fwd_adj<N>, dim3(xb, c.batch), TX, 0, s, Y6, c.cs, a, c.nu_b, c.tw));
      return;
    }
    // Y6 (6 fields per trajectory) -> W, as 2 * batch groups of 3 fields
    L3ES_LAUNCH(c, KK_X_FWD_PLAIN, 4.0 * A, s,
                pdl_launch(kx_fwd_plain<N, DIM>, dim3(xb, 2 * c.batch), TX, 0, s, Y6, c.cs, c.W, c.fs, c.tw));
    const long long pairs = c.cs / 2;
    L3ES_LAUNCH(c, KK_ADJ_EPI, epi, s,
                pdl_launch(k_adj_epi<N, DIM>, dim3((unsigned)((pairs + 255) / 256), c.batch), 256, 0, s, c.W, c.cs, a,
                                                                                                 c.nu_b));
  }

  static void vjp(const Ctx& c, const AdjEpi& a, float2* Wm, float2* Y6, cudaStream_t s) {
    if (c.dim == 3)
      vjp_dim<3>(c, a, Wm, Y6, s);
    else
      vjp_dim<2>(c, a, Wm, Y6, s);
  }
};

template <int N>
DnsTable make_dns_table() {
  DnsOps<N>::init_attrs();
  DnsTable t;
  t.stage = &DnsOps<N>::stage;
  t.step = &DnsOps<N>::step;
  t.steps2d = &DnsOps<N>::steps2d;
  t.irfftn = &DnsOps<N>::irfftn;
  t.rfftn = &DnsOps<N>::rfftn;
  t.vjp = &DnsOps<N>::vjp;
  return t;
}

}  // namespace l3es
