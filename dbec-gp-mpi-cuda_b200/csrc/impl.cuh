// impl.cuh -- the launches of a handle's operators, per real type and mode
// (instantiated in impl_*.cu and conv_*.cu).
#pragma once

#include "solver.cuh"

// ------------------------------------------------------------------ launches
inline Trap trap_of(const gpe_solver *s) {
   Trap t;
   t.x2 = s->x2; t.y2 = s->y2; t.z2 = s->z2;
   t.x2f = s->x2f; t.y2f = s->y2f; t.z2f = s->z2f;
   t.hp = 0.5 * s->par;
   t.vg2 = s->p.gamma * s->p.gamma;
   t.vn2 = s->p.nu * s->p.nu;
   t.vl2 = s->p.lambda * s->p.lambda;
   return t;
}

inline unsigned blocks_for(long long n, int bs) { return (unsigned) ((n + bs - 1) / bs); }

// Launch on the handle's stream with programmatic dependent launch: the
// kernel may be scheduled while its predecessor finishes its last wave (its
// CTAs call pdl_trigger / pdl_wait before touching memory), which hides the
// gap between the kernels of a step (FP64 0.880 -> 0.872 ms real, 0.722 ->
// 0.712 ms imaginary time; mixed precision 0.429 -> 0.415 ms at 256^3 and
// 0.107 -> 0.103 ms at 128^3, 512x512x256 unchanged at 1.69 ms, on B200).
template <class... KP, class... A>
gpe_status launch_pdl(void (*k)(KP...), dim3 grid, dim3 block, size_t smem, const gpe_solver *s, A... args) {
   CK(s->roomy.allow((const void *) k, smem));
   cudaLaunchAttribute at[1];
   at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
   at[0].val.programmaticStreamSerializationAllowed = 1;
   cudaLaunchConfig_t cfg{};
   cfg.gridDim = grid;
   cfg.blockDim = block;
   cfg.dynamicSmemBytes = smem;
   cfg.stream = s->st;
   cfg.attrs = at;
   cfg.numAttrs = 1;
   CK(cudaLaunchKernelEx(&cfg, k, ((KP) args)...));
   return GPE_OK;
}

// The passes on the lengths compiled for one solve only (conv_lens.cuh).
template <class R> gpe_status yfft_lens(gpe_solver *s, bool inv, unsigned grid, size_t sm);
template <class R> gpe_status xconv_lens(gpe_solver *s, unsigned grid, size_t sm);
template <class R> gpe_status zinv_lens(gpe_solver *s, size_t sm);
template <class R, bool CPLX> gpe_status zfwd_lens(gpe_solver *s, size_t sm);

// The passes of the dipolar convolution that do not see psi: y, x and inverse
// z FFTs, for one real type.
template <class R> struct Conv {
   using C = cpx<R>;

   // runs f(std::integral_constant<int, v>) for v in {2, 4, 8, 16} (tile
   // widths) or {8, 16, 32} (points per thread)
   template <class F> static gpe_status with_L(int L, F f) {
      if constexpr (std::is_same<R, float>::value)  // a tile row is 128 bytes at most
         if (L == 16) return f(std::integral_constant<int, 16>());
      if (L == 8) return f(std::integral_constant<int, 8>());
      if (L == 4) return f(std::integral_constant<int, 4>());
      return f(std::integral_constant<int, 2>());
   }
   template <class F> static gpe_status with_ppt(int ppt, F f) {
      if (ppt <= 8) return f(std::integral_constant<int, 8>());
      if (ppt <= 16) return f(std::integral_constant<int, 16>());
      return f(std::integral_constant<int, 32>());
   }
   // points per thread of the z passes: (nz/2) L over 256 threads, at least
   // 16 in FP32 (the radix-16 stages need them)
   static int zppt(const gpe_solver *s, int L) {
      const int p = (int) (((s->d.nz / 2) * L + 255) / 256);
      return s->fp32 ? std::max(p, 16) : p;
   }
   // threads of a z inverse pass CTA, and of a forward pass CTA over real
   // rows: PPT points each of the L half-length lines (the forward passes
   // over complex rows keep 256: sized CTAs measured slower there, 101 -> 105
   // us at 256^3 complex FP64)
   static unsigned z_threads(const gpe_solver *s, int L, int ppt) {
      const long t = ((long) (s->d.nz / 2) * L + ppt - 1) / ppt;
      return (unsigned) std::min<long>(256, std::max<long>(32, (t + 31) / 32 * 32));
   }

   // threads of a y / x pass CTA: PPT points each over a tile of rows x L
   // (at most 256: the kernels' register budget)
   static unsigned fft_threads(long rows, int L) {
      const long t = (rows * L + FftL<R>::PPT - 1) / FftL<R>::PPT;
      return (unsigned) std::min<long>(256, std::max<long>(32, (t + 31) / 32 * 32));
   }

   // Whether a pass runs its compile-time kernel (plan_tiles: the length has
   // one and the tile and radix choices are the defaults it is compiled for).
   static constexpr int kCols = LenCols<R>::L;
   // (the common set: the batched passes know no other)
   static bool len_x(const gpe_solver *s) { return s->fastx == 1; }
   static bool len_y(const gpe_solver *s) { return s->fasty == 1; }
   static bool len_z(const gpe_solver *s) { return s->fastz == 1; }

   // dynamic shared memory of the y and x passes on tiles of so many rows
   static size_t yfft_smem(const gpe_solver *s, int L, int rows) {
      return 128 + ((size_t) rows * L + s->d.ny) * sizeof(C);
   }
   static size_t xconv_smem(const gpe_solver *s, int L, int rows) {
      return 128 + (size_t) fft_tile_bytes<R>(rows, L) + udd_box(s->d.nx, L).bytes +
             (size_t) conv_roots(s->px) * sizeof(C);
   }

   template <bool INV, int L> static gpe_status yfft(gpe_solver *s) {
      const Dims &d = s->d;
      const unsigned grid = (unsigned) (d.nx * ((d.nzh + L - 1) / L));
      const size_t sm = yfft_smem(s, L, s->fasty ? d.ny : s->boxy * s->nboxy);
      if (s->fasty == 2) {
         CKS(yfft_lens<R>(s, INV, grid, sm));
         mark(s);
         return GPE_OK;
      }
      CKS(with_len(len_y(s) ? d.ny : 0, [&](auto nc) -> gpe_status {
         constexpr int N = decltype(nc)::value;
         if constexpr (N > 0 && L == kCols) {
            return launch_pdl(k_yfft_n<R, INV, L, N>, grid, len_threads<R>(N, L), sm, s, s->tm_spec_y, d,
                              (const C *) s->twy, s->err);
         } else {
            return launch_pdl(k_yfft<R, INV, L>, grid, fft_threads(s->boxy * s->nboxy, L), sm, s, s->tm_spec_y, d,
                              s->py, (const C *) s->twy, s->boxy, s->nboxy, s->err);
         }
      }));
      mark(s);
      return GPE_OK;
   }

   template <int L> static gpe_status xconv(gpe_solver *s) {
      const Dims &d = s->d;
      const unsigned grid = (unsigned) (d.ny * ((d.nzh + L - 1) / L));
      const size_t sm = xconv_smem(s, L, s->fastx ? d.nx : s->boxx * s->nboxx);
      if (s->fastx == 2) {
         CKS(xconv_lens<R>(s, grid, sm));
         mark(s);
         return GPE_OK;
      }
      CKS(with_len(len_x(s) ? d.nx : 0, [&](auto nc) -> gpe_status {
         constexpr int N = decltype(nc)::value;
         if constexpr (N > 0 && L == kCols) {
            return launch_pdl(k_xconv_n<R, L, N>, grid, len_threads<R>(N, L), sm, s, s->tm_spec_x,
                              s->tm_udd, d, (const C *) s->twx, s->state, s->err);
         } else {
            return launch_pdl(k_xconv<R, L>, grid, fft_threads(s->boxx * s->nboxx, L), sm, s, s->tm_spec_x,
                              s->tm_udd, d, s->px, s->pxi, (const C *) s->twx, s->state, s->boxx, s->nboxx, s->err);
         }
      }));
      mark(s);
      return GPE_OK;
   }

   template <int L> static gpe_status zinv_L(gpe_solver *s, size_t sm) {
      const Dims &d = s->d;
      return with_ppt(zppt(s, L), [&](auto pc) {
         constexpr int PPT = decltype(pc)::value;
         CKS(launch_pdl(k_zinv<R, PPT, L>, blocks_for(d.nxy, L), z_threads(s, L, PPT), sm, s, (const C *) s->spec, (R *) s->phi, d, s->ph,
                        (const C *) s->twz, s->LSo, s->err));
         CKL();
         mark(s);
         return GPE_OK;
      });
   }

   static size_t zinv_smem(const gpe_solver *s, int L) {
      const Dims &d = s->d;
      const size_t in_el = std::max((size_t) L * d.nzp, ((size_t) L * s->LSo * sizeof(R) + sizeof(C) - 1) / sizeof(C));
      return 128 + ((in_el + 7) & ~(size_t) 7) * sizeof(C) + ((size_t) (d.nz / 2) * L + ztab_len(d.nz / 2)) * sizeof(C);
   }
   template <class SM> static int zrows(const gpe_solver *s, int pref, SM smem) {
      int L = pref;
      while (L > 4 && smem(s, L) > kMaxSmem) L /= 2;
      return L;
   }
   template <class F> static gpe_status with_zrows(int L, F f) {
      if (L == 16) return f(std::integral_constant<int, 16>());
      if (L == 8) return f(std::integral_constant<int, 8>());
      return f(std::integral_constant<int, 4>());
   }

   // compile-time pass, 8-row tiles
   static size_t zinv_n_smem(const gpe_solver *s) {
      return 128 + zinv_region<R>(s->d.nz / 2, kLenRows) + ztab_len(s->d.nz / 2) * sizeof(C);
   }
   static gpe_status zinv_n(gpe_solver *s) {
      const Dims &d = s->d;
      const size_t sm = zinv_n_smem(s);
      CKS(with_len(d.nz / 2, [&](auto nc) -> gpe_status {
         constexpr int H = decltype(nc)::value;
         if constexpr (H > 0 && H <= kLenMaxH) {
            return launch_pdl(k_zinv_n<R, kLenRows, H>, blocks_for(d.nxy, kLenRows), len_threads<R>(H, kLenRows), sm, s,
                              (const C *) s->spec, (R *) s->phi, d, (const C *) s->twz, s->err);
         } else {
            return fail(GPE_ERR_STATE, "no compile-time z pass for this length");
         }
      }));
      mark(s);
      return GPE_OK;
   }

   // half spectrum of |psi|^2 (rows along z transformed) -> phi
   static gpe_status rest(gpe_solver *s);
};

template <class R> gpe_status Conv<R>::rest(gpe_solver *s) {
   CKS(with_L(s->Ly, [&](auto Lc) { return yfft<false, decltype(Lc)::value>(s); }));
   CKS(with_L(s->Lx, [&](auto Lc) { return xconv<decltype(Lc)::value>(s); }));
   CKS(with_L(s->Ly, [&](auto Lc) { return yfft<true, decltype(Lc)::value>(s); }));
   if (len_z(s)) {
      CKS(zinv_n(s));
   } else if (s->fastz == 2) {
      CKS(zinv_lens<R>(s, zinv_n_smem(s)));
      mark(s);
   } else {
      const int L = zrows(s, 8, zinv_smem);
      const size_t sm = zinv_smem(s, L);
      CKS(with_zrows(L, [&](auto lc) { return zinv_L<decltype(lc)::value>(s, sm); }));
   }
   mark(s);  // (boundary planes: stored by the inverse z pass)
   s->launches += 4;
   return GPE_OK;
}

template <class R, bool CPLX> struct Impl {
   using P = typename Tr<R, CPLX>::P;
   using C = cpx<R>;
   using CV = Conv<R>;

   // z pass kernels for a tile of L rows
   template <int L> static gpe_status zfwd_L(gpe_solver *s, size_t sm, bool sized) {
      const Dims &d = s->d;
      return CV::with_ppt(CV::zppt(s, L), [&](auto pc) {
         constexpr int PPT = decltype(pc)::value;
         const unsigned nt = sized ? CV::z_threads(s, L, PPT) : 256u;
         CKS(launch_pdl(k_zfwd<R, CPLX, PPT, L>, blocks_for(d.nxy, L), nt, sm, s, (const P *) s->psi, (C *) s->spec, d,
                        s->ph, (const C *) s->twz, s->LSr, s->err));
         CKL();
         mark(s);
         return GPE_OK;
      });
   }

   // shared memory of the z passes for L rows; the rows per CTA start at the
   // preferred value and halve (down to 4) until the tile fits
   static size_t zfwd_smem(const gpe_solver *s, int L) {
      const Dims &d = s->d;
      return 128 + (size_t) L * s->LSr * sizeof(P) + ((size_t) (d.nz / 2) * L + ztab_len(d.nz / 2)) * sizeof(C);
   }
   // compile-time pass, 8-row tiles
   static size_t zfwd_n_smem(const gpe_solver *s) {
      return 128 + zfwd_region<R, CPLX>(s->d.nz / 2, kLenRows) + ztab_len(s->d.nz / 2) * sizeof(C);
   }
   static gpe_status zfwd_n(gpe_solver *s) {
      const Dims &d = s->d;
      const size_t sm = zfwd_n_smem(s);
      CKS(with_len(d.nz / 2, [&](auto nc) -> gpe_status {
         constexpr int H = decltype(nc)::value;
         if constexpr (H > 0 && H <= kLenMaxH) {
            return launch_pdl(k_zfwd_n<R, CPLX, kLenRows, H>, blocks_for(d.nxy, kLenRows), len_threads<R>(H, kLenRows),
                              sm, s, (const P *) s->psi, (C *) s->spec, d, (const C *) s->twz, s->err);
         } else {
            return fail(GPE_ERR_STATE, "no compile-time z pass for this length");
         }
      }));
      mark(s);
      return GPE_OK;
   }
   static gpe_status psidd2(gpe_solver *s) {
      const Dims &d = s->d;
      if (CV::len_z(s)) {
         CKS(zfwd_n(s));
      } else if (s->fastz == 2) {
         CKS((zfwd_lens<R, CPLX>(s, zfwd_n_smem(s))));
         mark(s);
      } else {
         // real rows: 8-row tiles on CTAs sized to them, except FP64 rows
         // shorter than 128 points, which keep 16 rows on 256 threads (sized
         // CTAs of 32 threads measured slower at 64^3: 8.8 -> 10.8 us)
         const bool sized = !CPLX && (sizeof(R) == 4 || d.nz >= 128);
         const int L = CV::zrows(s, (!CPLX && !sized) ? 16 : zfwd_rows<R, CPLX>(), zfwd_smem);
         const size_t sm = zfwd_smem(s, L);
         CKS(CV::with_zrows(L, [&](auto lc) { return zfwd_L<decltype(lc)::value>(s, sm, sized); }));
      }
      s->launches++;
      return CV::rest(s);
   }


   template <int AXIS, bool NU, int MSEG, int S, int TWC> static gpe_status sweep_xy_launch_t(gpe_solver *s, double g, double gd) {
      auto &w = s->sw[AXIS];
      const Dims &d = s->d;
      const int nzb = (d.nz + w.TW - 1) / w.TW;
      const int ntiles = (AXIS == 0 ? d.ny : d.nx) * nzb;
      const unsigned grid = (unsigned) std::min(ntiles, w.ctas * s->nsm);
      CKS(launch_pdl(k_sweep_xy<R, CPLX, AXIS, NU, MSEG, S, TWC>, grid, ((w.TW * w.tab.P + 31) & ~31), w.smem, s,
          w.tm_psi, w.tm_phi, d, w.tab, trap_of(s), LinPhase{s->lin[0], s->lin[1], s->lin[2]}, g, gd, s->p.dt,
          s->state, w.TW, w.boxn, w.nbox, s->err));
      CKL();
      mark(s);
      s->launches++;
      return GPE_OK;
   }

   // FP64 tiles of 8 or 16 lines use kernels compiled for that width
   template <int AXIS, bool NU, int MSEG, int S> static gpe_status sweep_xy_launch(gpe_solver *s, double g, double gd) {
      if constexpr (std::is_same<R, double>::value) {
         if (s->sw[AXIS].TW == 8) return sweep_xy_launch_t<AXIS, NU, MSEG, S, 8>(s, g, gd);
         if constexpr (!kWide)
            if (s->sw[AXIS].TW == 16) return sweep_xy_launch_t<AXIS, NU, MSEG, S, 16>(s, g, gd);
      }
      return sweep_xy_launch_t<AXIS, NU, MSEG, S, 0>(s, g, gd);
   }

   // 32-point segments exist for FP32 real lines only, 16-point ones not for FP64
   // complex lines, whose tiles are 8 of them at most (sweep_candidates)
   static constexpr bool kSeg32 = std::is_same<R, float>::value && !CPLX;
   static constexpr bool kWide = std::is_same<R, double>::value && CPLX;

   template <int AXIS, bool NU> static gpe_status sweep_xy(gpe_solver *s, double g, double gd) {
      const auto &w = s->sw[AXIS];
      if constexpr (kSeg32)
         if (w.MSEG == 32)
            return w.S == 3 ? sweep_xy_launch<AXIS, NU, 32, 3>(s, g, gd) : sweep_xy_launch<AXIS, NU, 32, 2>(s, g, gd);
      if (kWide || w.MSEG == 8)
         return w.S == 3 ? sweep_xy_launch<AXIS, NU, 8, 3>(s, g, gd) : sweep_xy_launch<AXIS, NU, 8, 2>(s, g, gd);
      if constexpr (!kWide)
         return w.S == 3 ? sweep_xy_launch<AXIS, NU, 16, 3>(s, g, gd) : sweep_xy_launch<AXIS, NU, 16, 2>(s, g, gd);
   }

   // x sweep; with nu the pending 1/norm and calcnu are applied on load
   // (calcnu_kernel imag3d-mpicuda.cu:1759 fused with calclux_kernel :1802).
   static gpe_status xsweep(gpe_solver *s, bool nu, double g, double gd) {
      return nu ? sweep_xy<0, true>(s, g, gd) : sweep_xy<0, false>(s, g, gd);
   }

   static gpe_status ysweep(gpe_solver *s) { return sweep_xy<1, false>(s, 0., 0.); }

   template <int MOM, int MSEG, int S, int TWC> static gpe_status sweep_z_launch_t(gpe_solver *s, double *dev_norm) {
      auto &w = s->sw[2];
      const Dims &d = s->d;
      const long long ntiles = (d.nxy + w.TW - 1) / w.TW;
      const unsigned grid = (unsigned) std::min<long long>(ntiles, (long long) w.ctas * s->nsm);
      CKS(launch_pdl(k_sweep_z<R, CPLX, MOM, MSEG, S, TWC>, grid, ((w.TW * w.tab.P + 31) & ~31), w.smem, s,
          (P *) s->psi, d, w.tab, w.TW, w.LS, zout(s), s->p.dx, s->p.dy, s->state, dev_norm, s->err));
      CKL();
      mark(s);
      s->launches++;
      return GPE_OK;
   }

   template <int MOM, int MSEG, int S> static gpe_status sweep_z_launch(gpe_solver *s, double *nrm) {
      if constexpr (std::is_same<R, double>::value) {
         if (s->sw[2].TW == 8) return sweep_z_launch_t<MOM, MSEG, S, 8>(s, nrm);
         if constexpr (!kWide)
            if (s->sw[2].TW == 16) return sweep_z_launch_t<MOM, MSEG, S, 16>(s, nrm);
      }
      return sweep_z_launch_t<MOM, MSEG, S, 0>(s, nrm);
   }

   template <int MOM> static gpe_status zsweep_m(gpe_solver *s, double *nrm) {
      const auto &w = s->sw[2];
      if constexpr (kSeg32)
         if (w.MSEG == 32) return w.S == 3 ? sweep_z_launch<MOM, 32, 3>(s, nrm) : sweep_z_launch<MOM, 32, 2>(s, nrm);
      if (kWide || w.MSEG == 8) return w.S == 3 ? sweep_z_launch<MOM, 8, 3>(s, nrm) : sweep_z_launch<MOM, 8, 2>(s, nrm);
      if constexpr (!kWide)
         return w.S == 3 ? sweep_z_launch<MOM, 16, 3>(s, nrm) : sweep_z_launch<MOM, 16, 2>(s, nrm);
   }

   // z sweep; mom 1: also the norm of the step (dev_norm may be null) and the
   // pending renormalisation; mom 2: the rms row partials
   static gpe_status zsweep(gpe_solver *s, int mom, double *dev_norm = nullptr) {
      if (mom == 2) return zsweep_m<2>(s, nullptr);
      return mom == 1 ? zsweep_m<1>(s, dev_norm) : zsweep_m<0>(s, nullptr);
   }

   static ZOut zout(const gpe_solver *s) { return ZOut{s->wz, s->wz2, s->p.dz / 3., s->rowA, s->rowA, s->rowB}; }

   static gpe_status norm_final(gpe_solver *s, double *dev_out) {
      CKS(launch_pdl(k_norm_final, blocks_for(s->d.nx, kNormRowsPerCta), 32 * kNormRowsPerCta, 0, s,
          s->rowA, s->d, s->p.dx, s->p.dy, s->state, s->tmp, dev_out));
      CKL();
      s->launches++;
      return GPE_OK;
   }

   static gpe_status apply_scale(gpe_solver *s) {
      k_apply_scale<R, CPLX><<<592, 256, 0, s->st>>>((P *) s->psi, s->d.npts, s->state);
      CKL();
      k_state_set<<<1, 1, 0, s->st>>>(s->state, 1.);
      CKL();
      s->launches += 2;
      return GPE_OK;
   }

   static void rows_dens(gpe_solver *s, double *a, double *b) {
      k_rows_dens<R, CPLX><<<blocks_for(s->d.nxy, kRowWarps), 32 * kRowWarps, 0, s->st>>>(
          (const P *) s->psi, s->d, s->p.dz / 3., s->wz, s->wz2, a, b);
   }

   // line integrals of |psi|^2 along `axis` into rowA (z: a warp per row)
   static void lineint(gpe_solver *s, int axis, double h) {
      const Dims &d = s->d;
      if (axis == 2) return rows_dens(s, s->rowA, nullptr);
      const long long nl = (long long) (axis == 0 ? d.ny : d.nx) * d.nz;
      k_lineint_psi<R, CPLX><<<blocks_for(nl, 128), 128, 0, s->st>>>((const P *) s->psi, d, axis, h, s->rowA);
   }

   static gpe_status calcnorm(gpe_solver *s, bool renorm) {
      rows_dens(s, s->rowA, nullptr);
      CKL();
      CKS(norm_final(s, s->obs));
      s->launches++;
      if (renorm) {
         CKS(apply_scale(s));
      } else {
         k_state_set<<<1, 1, 0, s->st>>>(s->state, 1.);
         CKL();
      }
      return GPE_OK;
   }

   static gpe_status rms(gpe_solver *s, double *dev_out) {
      rows_dens(s, s->rowA, s->rowB);
      CKL();
      s->launches++;
      return rms_final(s, dev_out);
   }

   // rms from the row partials in rowA / rowB (k_rows_dens, or the z sweep
   // of the step with mom = 2)
   static gpe_status rms_final(gpe_solver *s, double *dev_out) {
      const Dims &d = s->d;
      CKS(launch_pdl(k_rms_final, blocks_for(d.nx, kNormRowsPerCta), 32 * kNormRowsPerCta, 0, s,
          s->rowA, s->rowB, d, s->p.dx, s->p.dy, s->x2, s->y2, s->state, s->tmp, dev_out));
      CKL();
      s->launches++;
      return GPE_OK;
   }

   static gpe_status muen(gpe_solver *s, double g, double gd, double *dev_out) {
      const Dims &d = s->d;
      CKS(psidd2(s));
      // chunks of x planes so that about 16 CTAs per SM run in turn (an even
      // last wave), at least 16 planes each (a chunk reads four more), with
      // room for the partials
      const unsigned bz = blocks_for(d.nz, kMuZ), by = blocks_for(d.ny, kMuY);
      const long long want = std::max<long long>(1, 16LL * s->nsm / ((long long) bz * by));
      const long long most = std::max<long long>(1, s->row_cap / (2LL * bz * by));
      const int chunk = (int) std::max<long long>(std::min<long long>(16, d.nx), (d.nx + std::min(want, most) - 1) / std::min(want, most));
      const unsigned bx = blocks_for(d.nx, chunk);
      k_muen<R, CPLX><<<dim3(bz, by, bx), kMuY * kMuZ, 0, s->st>>>((const P *) s->psi, (const R *) s->phi, d, trap_of(s),
                                                                  g, gd, s->p.dx, s->p.dy, s->p.dz, s->par, chunk,
                                                                  s->rowA);
      CKL();
      k_sum2<<<1, 256, 0, s->st>>>(s->rowA, (int) (bx * by * bz), s->p.dx * s->p.dy * s->p.dz / 27., dev_out);
      CKL();
      s->launches += 2;
      return GPE_OK;
   }

   // One split step (imag3d-mpicuda.cu:319-324): calcpsidd2, calcnu (fused
   // into the x sweep), x, y, z sweeps, and in imaginary time the norm.
   // rms_rows: (real time) the z sweep also leaves the rms row partials of
   // the new psi in rowA / rowB for rms_final.
   static gpe_status step(gpe_solver *s, double g, double gd, double *dev_norm, bool rms_rows = false) {
      CKS(psidd2(s));
      CKS(xsweep(s, true, g, gd));
      CKS(ysweep(s));
      const bool imag = !CPLX;
      CKS(zsweep(s, imag ? 1 : (rms_rows ? 2 : 0), dev_norm));
      if (imag) mark(s);  // (norm: the z sweep's last CTA)
      return GPE_OK;
   }

   static gpe_status calcnu(gpe_solver *s, double g, double gd) {
      k_calcnu<R, CPLX><<<592, 256, 0, s->st>>>((P *) s->psi, (const R *) s->phi, s->d, trap_of(s), g, gd, s->p.dt);
      CKL();
      s->launches++;
      return GPE_OK;
   }

   static gpe_status density(gpe_solver *s, int kind, long sx, long sy, long sz, double *out, long cap, long *count);

   // ---- batched launches: geometry and descriptor of this instance
   static gpe_status geom(gpe_solver *s, int Ly, int Lx, BatchGeom *g) {
      const Dims &d = s->d;
      *g = BatchGeom{};
      g->Ly = s->Ly;
      g->Lx = s->Lx;
      if (Ly <= 0 || Lx <= 0) return GPE_OK;
      // z passes: 8-row tiles
      constexpr int L = 8;
      auto fft = [&](int q, long long tiles, bool len, long pts, int lt) {
         g->tiles[q] = tiles;
         g->lens[q] = len;
         g->pts[q] = len ? 0 : pts;
         g->threads[q] = len ? (unsigned) lt : 0u;
      };
      for (int q : {kPZfwd, kPZinv})
         fft(q, (d.nxy + L - 1) / L, CV::len_z(s), (long) (d.nz / 2) * L, len_threads<R>(d.nz / 2, L));
      // y / x passes
      const long ry = (long) s->boxy * s->nboxy, rx = (long) s->boxx * s->nboxx;
      g->smem[kPZfwd] = CV::len_z(s) ? zfwd_n_smem(s) : zfwd_smem(s, L);
      g->smem[kPZinv] = CV::len_z(s) ? CV::zinv_n_smem(s) : CV::zinv_smem(s, L);
      if (g->smem[kPZfwd] > kMaxSmem || g->smem[kPZinv] > kMaxSmem)
         return fail(GPE_ERR_PARAM, "batch: z rows too long for 8-row tiles");
      // an instance with a compile-time pass keeps that pass's tile width
      Ly = CV::len_y(s) ? CV::kCols : Ly;
      Lx = CV::len_x(s) ? CV::kCols : Lx;
      if (ry * Ly > 256L * FftL<R>::PPT || rx * Lx > 256L * FftL<R>::PPT)
         return fail(GPE_ERR_PARAM, "batch: FFT tile too wide for this grid");
      for (int q : {kPYfft, kPYinv})
         fft(q, (long long) d.nx * ((d.nzh + Ly - 1) / Ly), CV::len_y(s), ry * Ly, len_threads<R>(d.ny, Ly));
      fft(kPXconv, (long long) d.ny * ((d.nzh + Lx - 1) / Lx), CV::len_x(s), rx * Lx, len_threads<R>(d.nx, Lx));
      g->smem[kPYfft] = g->smem[kPYinv] = CV::yfft_smem(s, Ly, (int) ry);
      g->smem[kPXconv] = CV::xconv_smem(s, Lx, (int) rx);
      // boundary planes of phi
      g->tiles[kPPhifix] = std::max<long>(1, (d.ny - 1) + (d.nx - 1));
      g->threads[kPPhifix] = (unsigned) std::min<long>(256, std::max<long>(32, (d.nz - 1 + 31) / 32 * 32));
      // sweeps
      const size_t esz = s->esz_psi;
      g->nxy = d.nxy;
      g->row_bytes = (size_t) d.nz * esz;
      for (int ax = 0; ax < 3; ax++) {
         const auto &w = s->sw[ax];
         const int TW = w.TW, P = w.tab.P;
         const int kp = kPXsweep + ax;
         g->mseg[ax] = w.MSEG;
         g->threads[kp] = (unsigned) ((TW * P + 31) & ~31);
         const int nzb = (d.nz + TW - 1) / TW;
         g->tiles[kp] = ax == 0 ? (long long) d.ny * nzb : (ax == 1 ? (long long) d.nx * nzb : (d.nxy + TW - 1) / TW);
         const size_t stage = ax < 2 ? sweep_stage(s, ax, w.boxn * w.nbox, TW, w.tab.skip) : (size_t) TW * w.LS * esz;
         g->stage[ax] = (uint32_t) ((stage + 127) & ~(size_t) 127);
         g->xch[ax] = (uint32_t) ((2 * (size_t) P * TW * esz + 15) & ~(size_t) 15);
         g->tabs[ax] = sweep_tab_bytes(w.tab.n, w.tab.skip, (int) esz, ax == 0 ? nu_tab_esz<R, CPLX>() : 0);
         g->tw[ax] = TW;
         g->across[ax] = nzb;
         SweepTile &r = g->tile[ax];
         r = SweepTile{};
         r.geo = sweep_geo(w.tab.n, ax < 2 ? w.boxn * w.nbox : w.LS, TW, w.tab.skip);
         r.tabs = w.tabs;
         if (ax < 2) r.st = s->state;
         else r.psi = s->psi;
         if (ax == 2) g->part = (uint32_t) (((size_t) P * TW * sizeof(double) + 15) & ~(size_t) 15);
      }
      // norm (imaginary time)
      g->tiles[kPNorm] = s->cplx ? 0 : 1;
      g->threads[kPNorm] = 256;
      return GPE_OK;
   }

   static gpe_status desc(gpe_solver *s, int Ly, int Lx, double g, double gd, BatchDesc *D) {
      const Dims &d = s->d;
      Ly = CV::len_y(s) ? CV::kCols : Ly;
      Lx = CV::len_x(s) ? CV::kCols : Lx;
      std::memset((void *) D, 0, sizeof(BatchDesc));
      D->tm_psi[0] = s->sw[0].tm_psi;
      D->tm_psi[1] = s->sw[1].tm_psi;
      D->tm_phi = s->sw[0].tm_phi;
      CKS(make_tmap(&D->tm_spec_y, s->spec, s->esz_r, 2 * d.nzh, d.ny, d.nx, 2 * Ly, s->boxy, 1, 2 * d.nzp));
      CKS(make_tmap(&D->tm_spec_x, s->spec, s->esz_r, 2 * d.nzh, d.ny, d.nx, 2 * Lx, 1, s->boxx, 2 * d.nzp));
      D->udd = s->udd;
      for (int ax = 0; ax < 3; ax++) {
         const auto &w = s->sw[ax];
         SweepView &v = D->sv[ax];
         v.tb = w.tab;
         v.trap = trap_of(s);
         v.lin = LinPhase{s->lin[0], s->lin[1], s->lin[2]};
         v.d = d;
         v.st = s->state;
         v.err = s->err;
         v.psi = s->psi;
         v.zo = zout(s);
         v.g = g;
         v.gd = gd;
         v.dt = s->p.dt;
         v.TW = w.TW;
         v.boxn = w.boxn;
         v.nbox = w.nbox;
         v.LS = w.LS;
      }
      D->px = s->px;
      D->pxi = s->pxi;
      D->fastx = CV::len_x(s);
      D->fasty = CV::len_y(s);
      D->fastz = CV::len_z(s);
      D->py = s->py;
      D->ph = s->ph;
      D->d = d;
      D->psi = s->psi;
      D->spec = s->spec;
      D->phi = s->phi;
      D->twx = s->twx;
      D->twy = s->twy;
      D->twz = s->twz;
      D->state = s->state;
      D->err = s->err;
      D->rowA = s->rowA;
      D->hx = s->p.dx;
      D->hy = s->p.dy;
      D->LSr = s->LSr;
      D->LSo = s->LSo;
      D->boxy = s->boxy;
      D->nboxy = s->nboxy;
      D->boxx = s->boxx;
      D->nboxx = s->nboxx;
      D->Ly = Ly;
      D->Lx = Lx;
      return GPE_OK;
   }
};

template <class R, bool CPLX>
gpe_status Impl<R, CPLX>::density(gpe_solver *s, int kind, long sx, long sy, long sz, double *out, long cap,
                                  long *count) {
   const Dims &d = s->d;
   const P *psi = (const P *) s->psi;
   const double hh[3] = {s->p.dx, s->p.dy, s->p.dz};
   const int n[3] = {d.nx, d.ny, d.nz};
   const std::vector<double> *crd[3] = {&s->hx, &s->hy, &s->hz};
   const long stp[3] = {sx, sy, sz};
   std::vector<double> buf;
   long o = 0;
   auto need = [&](long m) -> gpe_status {
      if (m > cap) return fail(GPE_ERR_PARAM, "density output buffer too small");
      return GPE_OK;
   };
   if (kind >= GPE_DEN_1D_X && kind <= GPE_DEN_1D_Z) {
      // axis integrated first, then the second one (reference nesting)
      const int keep = kind - GPE_DEN_1D_X;
      const int first = (keep == 2) ? 1 : 2;   // z (or y for the z profile)
      const int second = (keep == 0) ? 1 : 0;  // y for x profile, x otherwise
      const int o1 = first == 0 ? 1 : 0, o2 = first == 2 ? 1 : 2;  // axes of the 2D result
      if ((long long) n[o1] * n[o2] > s->row_cap) return fail(GPE_ERR_STATE, "row buffer too small");
      lineint(s, first, hh[first]);
      CKL();
      const int ax = (second == o1) ? 0 : 1;  // integrate rows (0) or columns (1)
      const int m = n[keep];
      k_lineint_arr<<<blocks_for(m, 128), 128, 0, s->st>>>(s->rowA, n[o1], n[o2], ax == 0 ? 0 : 1, hh[second], s->tmp);
      CKL();
      s->launches += 2;
      buf.resize(m);
      CK(cudaMemcpyAsync(buf.data(), s->tmp, sizeof(double) * m, cudaMemcpyDeviceToHost, s->st));
      CK(cudaStreamSynchronize(s->st));
      for (long c = 0; c < m; c += stp[keep]) {
         CKS(need(o + 2));
         out[o++] = (*crd[keep])[c];
         out[o++] = buf[c];
      }
   } else if (kind >= GPE_DEN_2D_XY && kind <= GPE_DEN_2D_YZ) {
      const int integ = 2 - (kind - GPE_DEN_2D_XY);  // xy -> z, xz -> y, yz -> x
      const int a1 = integ == 0 ? 1 : 0, a2 = integ == 2 ? 1 : 2;
      if ((long long) n[a1] * n[a2] > s->row_cap) return fail(GPE_ERR_STATE, "row buffer too small");
      lineint(s, integ, hh[integ]);
      CKL();
      s->launches++;
      buf.resize((size_t) n[a1] * n[a2]);
      CK(cudaMemcpyAsync(buf.data(), s->rowA, sizeof(double) * buf.size(), cudaMemcpyDeviceToHost, s->st));
      CK(cudaStreamSynchronize(s->st));
      for (long u = 0; u < n[a1]; u += stp[a1])
         for (long v = 0; v < n[a2]; v += stp[a2]) {
            CKS(need(o + 3));
            out[o++] = (*crd[a1])[u];
            out[o++] = (*crd[a2])[v];
            out[o++] = buf[(size_t) u * n[a2] + v];
         }
   } else if (kind >= GPE_DEN_3D_XY0 && kind <= GPE_DEN_3D_0YZ) {
      const int fixed = 2 - (kind - GPE_DEN_3D_XY0);  // xy0 -> z fixed, x0z -> y, 0yz -> x
      const int a1 = fixed == 0 ? 1 : 0, a2 = fixed == 2 ? 1 : 2;
      int lo[3] = {0, 0, 0}, hi[3] = {d.nx, d.ny, d.nz}, sp[3] = {(int) sx, (int) sy, (int) sz};
      lo[fixed] = n[fixed] / 2; hi[fixed] = lo[fixed] + 1; sp[fixed] = 1;
      const long na = (n[a1] + stp[a1] - 1) / stp[a1], nb = (n[a2] + stp[a2] - 1) / stp[a2];
      double *dv = nullptr;
      CK(cudaMalloc(&dv, sizeof(double) * na * nb));
      k_gather_dens<R, CPLX><<<blocks_for(na * nb, 256), 256, 0, s->st>>>(psi, d, lo[0], hi[0], sp[0], lo[1], hi[1], sp[1],
                                                                         lo[2], hi[2], sp[2], dv);
      s->launches++;
      buf.resize(na * nb);
      cudaError_t e1 = cudaGetLastError();
      cudaError_t e2 = cudaMemcpyAsync(buf.data(), dv, sizeof(double) * buf.size(), cudaMemcpyDeviceToHost, s->st);
      cudaError_t e3 = cudaStreamSynchronize(s->st);
      cudaFree(dv);
      if (e1 != cudaSuccess || e2 != cudaSuccess || e3 != cudaSuccess) return fail(GPE_ERR_CUDA, "density cut failed");
      for (long u = 0; u < na; u++)
         for (long v = 0; v < nb; v++) {
            CKS(need(o + 3));
            out[o++] = (*crd[a1])[u * stp[a1]];
            out[o++] = (*crd[a2])[v * stp[a2]];
            out[o++] = buf[(size_t) u * nb + v];
         }
   } else if (kind == GPE_DEN_3D) {
      const long na = (d.nx + sx - 1) / sx, nb = (d.ny + sy - 1) / sy, nc = (d.nz + sz - 1) / sz;
      CKS(need(na * nb * nc));
      double *dv = nullptr;
      CK(cudaMalloc(&dv, sizeof(double) * na * nb * nc));
      k_gather_dens<R, CPLX><<<592, 256, 0, s->st>>>(psi, d, 0, d.nx, (int) sx, 0, d.ny, (int) sy, 0, d.nz, (int) sz, dv);
      s->launches++;
      cudaError_t e1 = cudaGetLastError();
      cudaError_t e2 = cudaMemcpyAsync(out, dv, sizeof(double) * na * nb * nc, cudaMemcpyDeviceToHost, s->st);
      cudaError_t e3 = cudaStreamSynchronize(s->st);
      cudaFree(dv);
      if (e1 != cudaSuccess || e2 != cudaSuccess || e3 != cudaSuccess) return fail(GPE_ERR_CUDA, "density copy failed");
      o = na * nb * nc;
   } else {
      return fail(GPE_ERR_PARAM, "unknown density kind");
   }
   if (count) *count = o;
   return GPE_OK;
}

// ------------------------------------------------------------------ Ops
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::psidd2(gpe_solver *s) {
   return Impl<R, CPLX>::psidd2(s);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::xsweep(gpe_solver *s, bool nu, double g, double gd) {
   return Impl<R, CPLX>::xsweep(s, nu, g, gd);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::ysweep(gpe_solver *s) {
   return Impl<R, CPLX>::ysweep(s);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::zsweep(gpe_solver *s, int mom) {
   return Impl<R, CPLX>::zsweep(s, mom);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::apply_scale(gpe_solver *s) {
   return Impl<R, CPLX>::apply_scale(s);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::calcnorm(gpe_solver *s, bool renorm) {
   return Impl<R, CPLX>::calcnorm(s, renorm);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::calcnu(gpe_solver *s, double g, double gd) {
   return Impl<R, CPLX>::calcnu(s, g, gd);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::rms(gpe_solver *s, double *dev_out) {
   return Impl<R, CPLX>::rms(s, dev_out);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::rms_final(gpe_solver *s, double *dev_out) {
   return Impl<R, CPLX>::rms_final(s, dev_out);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::muen(gpe_solver *s, double g, double gd, double *dev_out) {
   return Impl<R, CPLX>::muen(s, g, gd, dev_out);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::step(gpe_solver *s, double g, double gd, double *dev_norm, bool rms_rows) {
   return Impl<R, CPLX>::step(s, g, gd, dev_norm, rms_rows);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::density(gpe_solver *s, int kind, long sx, long sy, long sz, double *out, long cap,
                                  long *count) {
   return Impl<R, CPLX>::density(s, kind, sx, sy, sz, out, cap, count);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::geom(gpe_solver *s, int Ly, int Lx, BatchGeom *g) {
   return Impl<R, CPLX>::geom(s, Ly, Lx, g);
}
template <class R, bool CPLX> gpe_status Ops<R, CPLX>::desc(gpe_solver *s, int Ly, int Lx, double g, double gd, BatchDesc *D) {
   return Impl<R, CPLX>::desc(s, Ly, Lx, g, gd, D);
}
