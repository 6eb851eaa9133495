// solver.cu -- handle, tables and the C ABI (include/gpe.h) of the B200
// dipolar Gross-Pitaevskii solver.  Host code only orchestrates; every
// operator on psi runs in the kernels of step_kernels.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <type_traits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <vector>

#include <cudaTypedefs.h>

#include "gpe.h"
#include "internal.h"
#include "solver.cuh"

using namespace gpe;

// The reference's truncated pi (imag3d-mpicuda.cu:69).
static const double kRefPi = 3.14159265358979;

static thread_local std::string g_err;

namespace gpe {
void set_last_error(const std::string &msg) { g_err = msg; }

cudaError_t RoomyKernels::allow(const void *kernel, size_t bytes) {
   if (bytes <= 46 * 1024) return cudaSuccess;
   if (bytes > kMaxSmem) return cudaErrorInvalidValue;
   for (const void *k : done_)
      if (k == kernel) return cudaSuccess;
   const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kMaxSmem);
   if (e == cudaSuccess) done_.push_back(kernel);
   return e;
}
}  // namespace gpe

gpe_status fail(gpe_status st, const std::string &msg) {
   g_err = msg;
   return st;
}

// ---------------------------------------------------------------- planning
static void set_stages(FftPlan &pl) {
   int ns = 1;
   for (int st = 0; st < pl.nst; st++) {
      pl.ns[st] = ns;
      // ceil(2^32 / ns): umulhi(j, magic) == j / ns for j, ns < 2^16; ns = 1 wraps to 0
      pl.magic[st] = ns == 1 ? 0u : (unsigned) ((0x100000000ULL + (unsigned long long) ns - 1) / (unsigned long long) ns);
      ns *= pl.rad[st];
   }
}

// Stages of an n-point transform (make_radices); max_radix 8, 4 or 2 drops
// the larger powers of two.  Radix 16 is for the FP32 passes only, whose
// threads hold 16 points.
static bool make_plan(int n, FftPlan &pl, int max_radix = 8) {
   pl.n = n;
   pl.nst = make_radices(n, max_radix == 16 ? 4 : (max_radix == 8 ? 3 : (max_radix == 4 ? 2 : 1)), pl.rad);
   set_stages(pl);
   return pl.nst > 0;
}

// The same stages in the reverse order.
static FftPlan reverse_plan(const FftPlan &pl) {
   FftPlan r = pl;
   for (int st = 0; st < pl.nst; st++) r.rad[st] = pl.rad[pl.nst - 1 - st];
   set_stages(r);
   return r;
}

static gpe_status validate(const gpe_params *p) {
   if (!p) return fail(GPE_ERR_PARAM, "null parameters");
   if (p->mode != GPE_MODE_IMAG && p->mode != GPE_MODE_REAL) return fail(GPE_ERR_PARAM, "mode must be 0 (imag) or 1 (real)");
   if (p->precision != GPE_PREC_FP64 && p->precision != GPE_PREC_MIXED) return fail(GPE_ERR_PARAM, "precision must be 0 or 1");
   const long n[3] = {p->nx, p->ny, p->nz};
   for (int a = 0; a < 3; a++) {
      if (n[a] < 8 || n[a] > 1024) return fail(GPE_ERR_PARAM, "grid sizes must be in [8, 1024]");
      if (n[a] % 2) return fail(GPE_ERR_PARAM, "grid sizes must be even (k-grid of initpotdd)");
      FftPlan pl;
      if (!make_plan((int) n[a], pl)) return fail(GPE_ERR_PARAM, "grid sizes must factor into 2, 3 and 5");
   }
   if (!(p->dx > 0 && p->dy > 0 && p->dz > 0 && p->dt > 0)) return fail(GPE_ERR_PARAM, "DX, DY, DZ, DT must be positive");
   if (!(p->cutoff > 0)) return fail(GPE_ERR_PARAM, "CUTOFF must be positive");
   if (p->precision == GPE_PREC_MIXED && p->nz % 4)
      return fail(GPE_ERR_PARAM, "mixed precision needs NZ divisible by 4 (16-byte FP32 rows)");
   return GPE_OK;
}

static size_t psi_esz(const gpe_params *p) {
   size_t r = (p->precision == GPE_PREC_MIXED) ? 4 : 8;
   return p->mode == GPE_MODE_REAL ? 2 * r : r;
}

extern "C" gpe_status gpe_device_bytes(const gpe_params *p, long long *bytes) {
   CKS(validate(p));
   const long long npts = p->nx * p->ny * p->nz;
   const long long nzh = p->nz / 2 + 1;
   const size_t r = (p->precision == GPE_PREC_MIXED) ? 4 : 8;
   long long b = 0;
   b += npts * (long long) psi_esz(p);                   // psi
   const long long nzp = (p->precision == GPE_PREC_MIXED) ? (nzh + 1) & ~1LL : nzh;
   b += nzp * p->nx * p->ny * (long long) (2 * r);       // spectrum (rows padded to 16 bytes)
   b += npts * (long long) r;                            // phi
   b += udd_pitch((int) nzh) * (p->nx / 2 + 1) * (p->ny / 2 + 1) * 8;  // Udd octant
   b += 4 * std::max(p->nx * p->ny, std::max(p->nx * p->nz, p->ny * p->nz)) * 8;  // row sums
   b += 1 << 20;                                         // tables, state
   if (bytes) *bytes = b;
   return GPE_OK;
}

// ------------------------------------------------------------------ tables
// On the handle's stream: a copy on the legacy stream from pageable memory may
// return before its data has arrived, and nothing would order it before the
// kernels of the handle's own non-blocking stream.
template <class T> static gpe_status upload(const gpe_solver *s, void **dst, const T *src, size_t n) {
   CK(cudaMalloc(dst, sizeof(T) * n));
   CK(cudaMemcpyAsync(*dst, src, sizeof(T) * n, cudaMemcpyHostToDevice, s->st));
   return GPE_OK;
}

// The same into a table that a later plan fills again (at most `cap` bytes): it
// is allocated once, by gpe_create, so that no plan after that can fail halfway
// and leave a handle without tables.
template <class T> static gpe_status replace(const gpe_solver *s, void **dst, const T *src, size_t n, size_t cap) {
   if (!*dst) CK(cudaMalloc(dst, cap));
   CK(cudaMemcpyAsync(*dst, src, sizeof(T) * n, cudaMemcpyHostToDevice, s->st));
   return GPE_OK;
}

// Roots of unity of the stages of pl in the order fft_lines / conv_lines read
// them: per stage after the first, exp(-2 pi i t k / (Ns r)) at [t - 1][k].
static void stage_roots(const FftPlan &pl, std::vector<double2> &out) {
   const size_t at = out.size();
   for (int st = 1; st < pl.nst; st++)
      for (int t = 1; t < pl.rad[st]; t++)
         for (int k = 0; k < pl.ns[st]; k++) {
            // the root of the n-point table the run-time stages read
            const long m = (long) t * k * (pl.n / (pl.ns[st] * pl.rad[st]));
            const long double a = -2.0L * 3.141592653589793238462643383279502884L * (long double) m / (long double) pl.n;
            out.push_back(make_double2((double) cosl(a), (double) sinl(a)));
         }
   out.resize(at + pl.n, make_double2(0., 0.));
}

// The tables of roots (ztab_roots in step_kernels.cuh) for the plans in use.
static gpe_status make_roots(gpe_solver *s) {
   const Dims &d = s->d;
   auto put = [&](const std::vector<double2> &t, void **dst) -> gpe_status {
      if (!s->fp32) return replace(s, dst, t.data(), t.size(), t.size() * sizeof(double2));
      std::vector<float2> f(t.size());
      for (size_t e = 0; e < t.size(); e++) f[e] = make_float2((float) t[e].x, (float) t[e].y);
      return replace(s, dst, f.data(), f.size(), f.size() * sizeof(float2));
   };
   std::vector<double2> t;
   stage_roots(s->px, t);
   stage_roots(s->pxi, t);
   CKS(put(t, &s->twx));
   t.clear();
   stage_roots(s->py, t);
   CKS(put(t, &s->twy));
   t.clear();
   const int h = d.nz / 2;
   stage_roots(s->ph, t);
   t.resize(ztab_roots(h), make_double2(0., 0.));
   for (int k = 0; k <= h; k++) {
      const long double a = -2.0L * 3.141592653589793238462643383279502884L * (long double) k / (long double) d.nz;
      t.push_back(make_double2((double) cosl(a), (double) sinl(a)));
   }
   t.resize(ztab_len(h), make_double2(0., 0.));
   return put(t, &s->twz);
}

// gencoef (imag3d-mpicuda.cu:894-931, real3d-mpicuda.cu:991-1035).
static void make_coef(gpe_solver *s, int ax, long n, double d2) {
   const double c = s->p.dt / d2 / (3. - s->par);
   typedef std::complex<double> Z;
   const Z A0 = s->cplx ? Z(1., c) : Z(1. + c), A = s->cplx ? Z(0., -0.5 * c) : Z(-0.5 * c);
   std::vector<Z> al(n - 1), ga(n - 1);
   al[n - 2] = 0.;
   ga[n - 2] = Z(-1.) / A0;
   for (long i = n - 2; i > 0; i--) {
      al[i - 1] = A * ga[i];
      ga[i - 1] = Z(-1.) / (A0 + A * al[i - 1]);
   }
   s->A[ax] = make_double2(A.real(), A.imag());
   if (!s->cplx)
      for (auto *v : {&al, &ga})
         for (Z &z : *v) z = z.real();
   s->alpha[ax] = std::move(al);
   s->gamma[ax] = std::move(ga);
}

// Segment tables of the parallel Thomas sweep of axis ax (line length n, P
// segments of m points; segment p holds recurrence indices lo .. lo + m - 1,
// lo = p m - skip, zero coefficients below index 0):
//   M[i] = prod_{j=i+1}^{lo+m} gamma[j] A   in every segment but the top one
//   N[k] = prod_{j=lo}^{k-1} alpha[j]        for k in (lo, lo + m], but the bottom one
// computed in long double and rounded once.
static gpe_status make_segtab(gpe_solver *s, int ax, long n, int m, int P) {
   // the z sweep's Simpson partials take the weight of a point from its
   // parity within the segment, so segments start at even indices
   if (m % 2 || n % 2) return fail(GPE_ERR_PARAM, "segment and line lengths must be even");
   typedef std::complex<long double> Z;
   const int E = s->cplx ? 2 : 1;
   std::vector<Z> al(s->alpha[ax].begin(), s->alpha[ax].end()), ga(s->gamma[ax].begin(), s->gamma[ax].end());
   const Z A(s->A[ax].x, s->A[ax].y);
   const long skip = (long) P * m - (n - 2), ne = (long) P * m;
   std::vector<Z> tg(ne, Z(0)), tma(2 * ne, Z(0)), tn(ne, Z(0));
   long double amax = 0, nmax = 0;  // largest decay of a segment's backward and forward map
   for (int p = 0; p < P; p++) {
      const long lo = (long) p * m - skip;
      const long q0 = std::max(0L, -lo);
      Z r = 1;
      for (long q = m - 1; q >= q0; q--) {
         const long e = (long) p * m + q, i = lo + q;
         tg[e] = ga[i + 1];
         r *= ga[i + 1] * A;
         if (p < P - 1) tma[2 * e] = r;
         tma[2 * e + 1] = al[i];
      }
      if (p < P - 1) amax = std::max(amax, std::abs(r));
      r = 1;
      for (long q = q0; q < m; q++) {
         r *= al[lo + q];
         if (p > 0) tn[(long) p * m + q] = r;
      }
      if (p > 0) nmax = std::max(nmax, std::abs(r));
   }
   // segments whose maps a thread composes: the carry from farther away is
   // scaled by a product of D decays, dropped below 2^-64 (FP64) or 2^-40
   // (FP32), under the rounding of the carry itself
   const long double drop = s->fp32 ? ldexpl(1.L, -40) : ldexpl(1.L, -64), dec = std::max(amax, nmax);
   int D = 1;
   for (long double r = dec; D < P && r > drop; r *= dec) D++;
   auto &w = s->sw[ax];
   // gamma | (M, alpha) | N, and for the x sweep calcnu's table behind `skip`
   // zero entries, in one block (the batched sweeps copy it whole)
   const size_t r = s->esz_r;
   const int xe = ax == 0 ? (int) (s->nu_x.size() / (size_t) n) : 0;
   std::vector<unsigned char> blk(sweep_tab_bytes((int) n, (int) skip, (int) s->esz_psi, xe), 0);
   const std::vector<Z> *src[3] = {&tg, &tma, &tn};
   size_t at = 0;
   for (int q = 0; q < 3; q++)
      for (const Z &z : *src[q]) {
         double h[2] = {(double) z.real(), (double) z.imag()};
         for (int c = 0; c < E; c++, at += r) {
            if (s->fp32) {
               // FP32 copies of the FP64 values, rounded once.  In real time the gamma copy holds gamma + 1
               // (SegOps::back_step): gamma is -1 plus a small number, which
               // FP32 keeps to its own relative precision.
               const float f = (float) (q == 0 && s->cplx && c == 0 ? h[c] + 1. : h[c]);
               std::memcpy(&blk[at], &f, 4);
            } else {
               std::memcpy(&blk[at], &h[c], 8);
            }
         }
      }
   if (ax == 0) std::memcpy(&blk[at + (size_t) skip * xe], s->nu_x.data(), s->nu_x.size());
   // (skip < m <= 32)
   CKS(replace(s, &w.tabs, blk.data(), blk.size(), sweep_tab_bytes((int) n, 31, (int) s->esz_psi, xe)));
   SegTab &t = w.tab;
   t.ga = w.tabs;
   t.ma = (unsigned char *) w.tabs + (size_t) ne * s->esz_psi;
   t.nn = (unsigned char *) w.tabs + 3 * (size_t) ne * s->esz_psi;
   t.A = s->A[ax];
   t.n = (int) n;
   t.m = m;
   t.P = P;
   t.D = D;
   t.skip = (int) skip;
   return GPE_OK;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static gpe_status encoder(EncodeTiledFn *fn) {
   static EncodeTiledFn cached = nullptr;
   if (!cached) {
      void *f = nullptr;
      cudaDriverEntryPointQueryResult q;
      CK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q));
      if (!f || q != cudaDriverEntryPointSuccess) return fail(GPE_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled unavailable");
      cached = (EncodeTiledFn) f;
   }
   *fn = cached;
   return GPE_OK;
}

gpe_status make_tmap(CUtensorMap *m, void *base, size_t esz, long w_nz, long ny, long nx, int bw, int by, int bx,
                     long pitch) {
   EncodeTiledFn enc;
   CKS(encoder(&enc));
   if (pitch == 0) pitch = w_nz;
   cuuint64_t dims[3] = {(cuuint64_t) w_nz, (cuuint64_t) ny, (cuuint64_t) nx};
   cuuint64_t strides[2] = {(cuuint64_t) (pitch * esz), (cuuint64_t) (pitch * esz * ny)};
   cuuint32_t box[3] = {(cuuint32_t) bw, (cuuint32_t) by, (cuuint32_t) bx};
   cuuint32_t es[3] = {1, 1, 1};
   CUresult r = enc(m, esz == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, base, dims,
                    strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
   if (r != CUDA_SUCCESS) return fail(GPE_ERR_CUDA, "cuTensorMapEncodeTiled failed (" + std::to_string((int) r) + ")");
   return GPE_OK;
}

// Candidates (lines per CTA TW, segment length MSEG, segments P) for a sweep
// over lines of length n, widest tile first: TW from `tw_base` (a 128-byte
// row) down to 2, and for each TW every segment length with at most 256
// threads (TW * P), shortest first; prim[c] marks the shortest segment of
// each TW (the most threads), the built-in choice.  Lines of 16-byte elements
// keep 8-point segments (16 would spill registers); 4-byte elements may use
// 32-point segments, which keep 64-byte tile rows on 512-point lines.
constexpr int kSweepCand = 16;
static int sweep_candidates(int n, int tw_base, int esz, int *TW, int *MSEG, int *P, bool *prim) {
   const bool wide = esz == 16;
   const int ms[3] = {8, 16, 32};
   const int nms = wide ? 1 : (esz == 4 ? 3 : 2);
   int k = 0;
   for (int tw = tw_base; tw >= 2 && k < kSweepCand; tw /= 2) {
      bool first = true;
      for (int mi = 0; mi < nms && k < kSweepCand; mi++) {
         const int p = (n - 2 + ms[mi] - 1) / ms[mi];
         if (tw * p <= 256) {
            TW[k] = tw; MSEG[k] = ms[mi]; P[k] = p; prim[k] = first;
            first = false;
            k++;
         }
      }
   }
   if (k == 0) {
      TW[0] = 2; MSEG[0] = wide ? 8 : 16; P[0] = (n - 2 + MSEG[0] - 1) / MSEG[0]; prim[0] = true;
      k = 1;
   }
   return k;
}

// Tile configuration of the sweeps and of the y / x FFT passes, and the FFT
// plans: the heuristics below, or the values of s->tune where set.  May be
// called again (gpe_set_tuning); it uploads the segment tables, calcnu's x table
// and the roots of unity anew, in the order of the handle's stream and without
// an allocation.
static gpe_status plan_tiles(gpe_solver *s) {
   s->plan_gen++;
   const Dims &d = s->d;
   const size_t esz = s->esz_psi, rsz = s->esz_r;
   const int E = s->cplx ? 2 : 1;
   const int tw_base = (int) (128 / esz);
   const long nn[3] = {d.nx, d.ny, d.nz};
   const size_t sm_cap = 227 * 1024;
   for (int ax = 0; ax < 3; ax++) {
      auto &w = s->sw[ax];
      // the widest tile for which as many CTAs as the kernels are compiled for
      // fit on an SM with a 2-stage pipeline (else the widest tile, fewer CTAs)
      int cTW[kSweepCand], cM[kSweepCand], cP[kSweepCand];
      bool prim[kSweepCand];
      const int nc = sweep_candidates((int) nn[ax], tw_base, (int) esz, cTW, cM, cP, prim);
      auto ctas_of = [&](int c) { return sweep_ctas(s->fp32, s->cplx, cM[c]); };
      auto sizes = [&](int TW, int MS, int P, size_t &stage, size_t &fixed) {
         const int skip = P * MS - (int) (nn[ax] - 2);
         const size_t xch = (2 * (size_t) P * TW * esz + 15) & ~(size_t) 15;
         if (ax < 2) {
            const int rows = (int) (std::min<long>(nn[ax], 256) * ((nn[ax] + 255) / 256));
            stage = sweep_stage(s, ax, rows, TW, skip);
            // FP64 x sweep: calcnu's per-x table staged in shared memory
            fixed = 128 + xch + (ax == 0 && !s->fp32 ? (size_t) (nn[0] + skip) * (s->cplx ? 16 : 8) : 0);
         } else {
            stage = ((size_t) TW * zrow_stride(d.nz, skip, (int) esz) * esz + 127) & ~(size_t) 127;
            // FP64: the coefficient tables staged in shared memory
            fixed = 128 + xch + 2 * (size_t) P * TW * sizeof(double) + (s->fp32 ? 0 : 4 * (size_t) P * MS * esz);
         }
      };
      auto fits = [&](int c) {
         size_t st_, fx_;
         sizes(cTW[c], cM[c], cP[c], st_, fx_);
         return (fx_ + 2 * st_) * 2 <= sm_cap;
      };
      const int want_tw = s->tune.sweep_tw[ax], want_ms = s->tune.sweep_seg[ax];
      // a candidate matching the fields that are set (an unset segment
      // length means the shortest of that TW; an unset TW the widest tile
      // that fits, else the widest)
      auto match = [&](int c) { return (want_tw <= 0 || cTW[c] == want_tw) && (want_ms <= 0 ? prim[c] : cM[c] == want_ms); };
      int pick = -1;
      if (want_tw > 0 || want_ms > 0) {
         for (int c = 0; c < nc && pick < 0; c++)
            if (match(c) && (want_tw > 0 || fits(c))) pick = c;
         for (int c = 0; c < nc && pick < 0; c++)
            if (match(c)) pick = c;
         if (pick < 0) return fail(GPE_ERR_PARAM, "tuning: sweep_tw / sweep_seg not available for this line length");
      } else {
         // measured on B200 (us, choice against the widest tile with the
         // shortest segments): FP64 real lines of 96 points or more: x and z 8
         // lines of 16-point segments (256^3: x 93 -> 85, z 71 -> 62; 128^3: z
         // 20.5 -> 18.5), y 16 of 16 (128^3: 14.4 -> 12.3); FP32 complex x 8
         // of 8 (256^3: 121 -> 96; 160 points 27 -> 23); FP32 real z 16 of 32
         // where that leaves 8 segments (512x512x256: 143 -> 138), else 16 of
         // 16 (128^3: 16.1 -> 14.4)
         auto want = [&](int tw, int m) {
            for (int c = 0; c < nc && pick < 0; c++)
               if (cTW[c] == tw && cM[c] == m && fits(c)) pick = c;
         };
         if (!s->fp32 && !s->cplx && nn[ax] >= 96) want(ax == 1 ? 16 : 8, 16);
         if (s->fp32 && s->cplx && ax == 0) want(8, 8);
         if (s->fp32 && !s->cplx && ax == 2 && nn[ax] >= 96) {
            if (nn[ax] - 2 > 7 * 32) want(16, 32);
            want(16, 16);
         }
         for (int c = 0; c < nc && pick < 0; c++)
            if (prim[c] && fits(c)) pick = c;
         if (pick < 0) pick = 0;
      }
      w.TW = cTW[pick];
      w.MSEG = cM[pick];
      const int P = cP[pick];
      CKS(make_segtab(s, ax, nn[ax], w.MSEG, P));
      size_t stage = 0, fixed = 0;
      sizes(w.TW, w.MSEG, P, stage, fixed);
      if (ax < 2) {
         w.boxn = (int) std::min<long>(nn[ax], 256);
         w.nbox = (int) ((nn[ax] + w.boxn - 1) / w.boxn);
         const int by = ax == 1 ? w.boxn : 1, bx = ax == 0 ? w.boxn : 1;
         CKS(make_tmap(&w.tm_psi, s->psi, s->fp32 ? 4 : 8, E * d.nz, d.ny, d.nx, E * w.TW, by, bx));
         CKS(make_tmap(&w.tm_phi, s->phi, rsz, d.nz, d.ny, d.nx, w.TW, by, bx));
      } else {
         w.LS = zrow_stride(d.nz, w.tab.skip, (int) esz);
      }
      // as many resident CTAs as allowed, then the deepest pipeline (2 or 3
      // stages) that keeps them
      // default depth: 3 for the TMA tensor tiles of the x / y sweeps, 2 for
      // the z sweep's bulk-copied rows (measured faster on B200 at 256^3, both
      // modes)
      // (FP32 real z sweeps on 16-row tiles of 32-point segments: 3)
      const bool z16 = ax == 2 && esz == 4 && w.TW == 16 && w.MSEG == 32;
      const int s_hi = s->tune.sweep_stages[ax] > 0 ? s->tune.sweep_stages[ax] : ((ax == 2 && !z16) ? 2 : 3);
      const int s_lo = s->tune.sweep_stages[ax] > 0 ? s->tune.sweep_stages[ax] : 2;
      if (s_lo < 2 || s_hi > 3) return fail(GPE_ERR_PARAM, "tuning: sweep_stages must be 2 or 3");
      // the register budget of ctas_of() CTAs of 256 threads holds more CTAs
      // of fewer threads
      const int thr = (w.TW * P + 31) & ~31;
      const int ct_max = std::min(32, 256 * ctas_of(pick) / thr);
      // a third stage only where it leaves the tables that are read through L1
      // (all but the FP64 z sweep's) their room there: us with three -> two,
      // FP32 complex x of 720 points 43 -> 37, FP64 complex y of 1024 points 74 ->
      // 66 and of 512 points 30 -> 28, FP64 real x of 1024 points 80 -> 70
      const size_t l1 = ax == 2 && !s->fp32 ? 0 : 4 * (size_t) P * w.MSEG * esz;
      auto stages_fit = [&](int ct, int S) {
         const size_t b = fixed + S * stage;
         if (b > kMaxSmem || smem_ctas(b, kSweepFixed) < ct) return false;
         return S == s_lo || ct * (b + kSweepFixed + kCtaReserved) + l1 <= kSmSmem;
      };
      w.ctas = 0;
      for (int ct = ct_max; ct >= 1 && !w.ctas; ct--)
         for (int S = s_hi; S >= s_lo && !w.ctas; S--)
            if (stages_fit(ct, S)) {
               w.ctas = ct;
               w.S = S;
            }
      if (!w.ctas) return fail(GPE_ERR_PARAM, "grid too large for the sweep tiles (shared memory)");
      w.smem = fixed + w.S * stage;
   }
   // spectrum tiles: spec[x][y][kz] viewed as [nx][ny][2 nzh] scalars; L kz
   // columns (at most a 128-byte row) per tile, halved (down to 2) until a
   // tile of a whole line holds at most 256 PPT points (32 KB), the in-place
   // FFT's register budget; the CTA has one thread per PPT points of its tile
   {
      s->boxy = (int) std::min<long>(d.ny, 256);
      s->nboxy = (d.ny + s->boxy - 1) / s->boxy;
      s->boxx = (int) std::min<long>(d.nx, 256);
      s->nboxx = (d.nx + s->boxx - 1) / s->boxx;
      const long ppt = s->fp32 ? 16 : 8;  // FftL<R>::PPT
      // FP64 starts from 4 columns: on B200 the 128-thread CTAs of 4-column
      // tiles (eight per SM) measured faster than 8-column tiles (four per
      // SM): y pass 60 -> 56 us, 256^3 step 0.870 -> 0.863 ms.  FP32 starts
      // from 8 columns (64-byte rows): mixed 256^3 step 0.412 -> 0.403 ms
      // against 16 columns, 128^3 0.103 -> 0.102 ms, 512x512x256 (8 columns
      // either way) unchanged
      auto pickL = [&](long rows) {
         int L = s->fp32 ? 8 : 4;
         while (L > 2 && rows * L > 256 * ppt) L /= 2;
         return L;
      };
      s->Ly = pickL((long) s->boxy * s->nboxy);
      s->Lx = pickL((long) s->boxx * s->nboxx);
      const long rows[2] = {(long) s->boxy * s->nboxy, (long) s->boxx * s->nboxx};
      int *Ls[2] = {&s->Ly, &s->Lx};
      for (int a = 0; a < 2; a++) {
         const int L = s->tune.fft_tile[a];
         if (L == 0) continue;
         if ((L & (L - 1)) || L < 2 || L > 128 / (int) s->esz_c || rows[a] * L > 256 * ppt)
            return fail(GPE_ERR_PARAM, "tuning: fft_tile must be a power of two, >= 2, at most a 128-byte row and "
                                       "at most 256 PPT points per tile");
         *Ls[a] = L;
      }
      // FP32 passes hold 16 points per thread and default to radix-16 stages
      // (two stages instead of three for 128- and 256-point lines)
      const int mr = s->tune.fft_max_radix > 0 ? s->tune.fft_max_radix : (s->fp32 ? 16 : 8);
      if (mr != 16 && mr != 8 && mr != 4 && mr != 2)
         return fail(GPE_ERR_PARAM, "tuning: fft_max_radix must be 16, 8, 4 or 2");
      if (mr == 16 && !s->fp32) return fail(GPE_ERR_PARAM, "tuning: radix 16 is for mixed precision only");
      // compile-time passes (fftn.cuh) where the tile and radix choices are the
      // defaults; the common set takes radices up to 16 in both precisions
      const bool plain = s->tune.fft_max_radix <= 0 || s->tune.fft_max_radix == (s->fp32 ? 16 : 8);
      auto level = [&](bool common, bool own) { return !plain ? 0 : (common ? 1 : (own ? 2 : 0)); };
      const int h = d.nz / 2;
      s->fastx = s->Lx == len_cols(s->fp32) ? level(has_len(d.nx), has_len_xy(d.nx)) : 0;
      s->fasty = s->Ly == len_cols(s->fp32) ? level(has_len(d.ny), has_len_xy(d.ny)) : 0;
      s->fastz = level(has_len(h) && h <= kLenMaxH, has_len_z(h));
      const int rx = s->fastx == 1 ? 16 : mr, ry = s->fasty == 1 ? 16 : mr, rz = s->fastz == 1 ? 16 : mr;
      make_plan(d.nx, s->px, rx);
      s->pxi = reverse_plan(s->px);
      make_plan(d.ny, s->py, ry);
      make_plan(d.nz / 2, s->ph, rz);
      CKS(make_roots(s));
      // a line over 256 points compiled for one solve arrives in two halves,
      // without padded rows (a batch's run-time pass has boxes of its own)
      const int by = s->fasty == 2 && d.ny > 256 ? d.ny / 2 : s->boxy, bx = s->fastx == 2 && d.nx > 256 ? d.nx / 2 : s->boxx;
      CKS(make_tmap(&s->tm_spec_y, s->spec, rsz, 2 * d.nzh, d.ny, d.nx, 2 * s->Ly, by, 1, 2 * d.nzp));
      CKS(make_tmap(&s->tm_spec_x, s->spec, rsz, 2 * d.nzh, d.ny, d.nx, 2 * s->Lx, 1, bx, 2 * d.nzp));
      CKS(make_udd_tmap(s, &s->tm_udd, s->Lx));
   }
   return GPE_OK;
}

// Simpson weights along z and the device status word (once per handle).
static gpe_status setup_static(gpe_solver *s) {
   const Dims &d = s->d;
   // Simpson weights along z: sum_k wz[k] f[k] * dz / 3 equals simpint (diffint.cu:37-66)
   std::vector<double> wz(d.nz, 0.);
   const int N = d.nz, mm = (N % 2) ? N : N - 1;
   for (int k = 0; k < mm; k++) wz[k] = (k == 0 || k == mm - 1) ? 1. : ((k % 2) ? 4. : 2.);
   if (N % 2 == 0) { wz[N - 1] += 5. / 4.; wz[N - 2] += 8. / 4.; wz[N - 3] -= 1. / 4.; }
   void *t = nullptr;
   // (kTabPad zero entries before index 0, for the sweeps' rows below the line)
   wz.insert(wz.begin(), kTabPad, 0.);
   CKS(upload(s, &t, wz.data(), wz.size()));
   s->wz = (double *) t + kTabPad;
   std::vector<double> wz2(kTabPad + d.nz, 0.);
   for (int k = 0; k < N; k++) {
      const double z = (k - d.nz / 2) * s->p.dz;  // the mesh of initpsi
      wz2[kTabPad + k] = wz[kTabPad + k] * (z * z);
   }
   CKS(upload(s, &t, wz2.data(), wz2.size()));
   s->wz2 = (double *) t + kTabPad;
   CK(cudaMalloc(&s->err, sizeof(uint32_t)));
   CK(cudaMemsetAsync(s->err, 0, sizeof(uint32_t), s->st));
   return GPE_OK;
}

// initpotdd (imag3d-mpicuda.cu:945-980) on the octant |kx| <= nx/2,
// |ky| <= ny/2, kz <= nz/2, stored [|kx|][|ky|][kz] (udd_pitch): Udd depends on kx^2,
// ky^2, kz^2 only, and the squares of the reference's negative k values equal
// those of the octant.
static gpe_status make_udd(gpe_solver *s) {
   const long nx = s->p.nx, ny = s->p.ny, nz = s->p.nz;
   const long nxh = nx / 2 + 1, nyh = ny / 2 + 1, nzh = nz / 2 + 1;
   const double pi = kRefPi, cutoff = s->p.cutoff;
   const double dkx = 2. * pi / (nx * s->p.dx), dky = 2. * pi / (ny * s->p.dy), dkz = 2. * pi / (nz * s->p.dz);
   std::vector<double> kx2(nxh), ky2(nyh), kz2(nzh);
   for (long i = 0; i < nxh; i++) { double k = i * dkx; kx2[i] = k * k; }
   for (long i = 0; i < nyh; i++) { double k = i * dky; ky2[i] = k * k; }
   for (long i = 0; i < nzh; i++) { double k = i * dkz; kz2[i] = k * k; }
   const long nzu = udd_pitch((int) nzh);
   std::vector<double> u((size_t) (nzu * nxh * nyh), 0.);
   for (long i = 0; i < nxh; i++)
      for (long j = 0; j < nyh; j++)
         for (long k = 0; k < nzh; k++) {
            const double xk = std::sqrt(kz2[k] + kx2[i] + ky2[j]);
            const double tmp = 1. + 3. * std::cos(xk * cutoff) / (xk * xk * cutoff * cutoff) -
                               3. * std::sin(xk * cutoff) / (xk * xk * xk * cutoff * cutoff * cutoff);
            u[(size_t) ((i * nyh + j) * nzu + k)] = (4. * pi * (3. * kz2[k] / (kx2[i] + ky2[j] + kz2[k]) - 1.) / 3.) * tmp;
         }
   u[0] = 0.;  // imag3d-mpicuda.cu:975-977
   void *dp = nullptr;
   CKS(upload(s, &dp, u.data(), u.size()));
   s->udd = (double *) dp;
   return GPE_OK;
}

static void free_all(gpe_solver *s) {
   void *ptrs[] = {s->psi, s->spec, s->phi, s->twx, s->twy, s->twz, s->udd, s->x2, s->y2, s->z2,
                   s->rowA, s->rowB, s->tmp, s->obs, s->state, s->rms_buf};
   for (void *q : ptrs)
      if (q) cudaFree(q);
   for (int a = 0; a < 3; a++) {
      if (s->sw[a].tabs) cudaFree(s->sw[a].tabs);
   }
   if (s->wz) cudaFree(s->wz - kTabPad);
   for (float *q : {s->x2f, s->y2f, s->z2f})
      if (q) cudaFree(q - kTabPad);
   for (void *q : s->lin)
      if (q) cudaFree(s->fp32 ? (void *) ((float *) q - kTabPad) : q);
   if (s->wz2) cudaFree(s->wz2 - kTabPad);
   if (s->err) cudaFree(s->err);
   if (s->own_stream && s->st) cudaStreamDestroy(s->st);
}

static gpe_status create_impl(const gpe_params *p, void *stream, gpe_solver *s) {
   s->p = *p;
   s->cplx = p->mode == GPE_MODE_REAL;
   s->fp32 = p->precision == GPE_PREC_MIXED;
   s->par = (p->opt == 2) ? 2. : 1.;
   if (p->device >= 0) CK(cudaSetDevice(p->device));
   CK(cudaGetDevice(&s->dev));
   CK(cudaDeviceGetAttribute(&s->nsm, cudaDevAttrMultiProcessorCount, s->dev));
   if (stream) {
      s->st = (cudaStream_t) stream;
   } else {
      CK(cudaStreamCreateWithFlags(&s->st, cudaStreamNonBlocking));
      s->own_stream = true;
   }
   Dims &d = s->d;
   d.nx = (int) p->nx; d.ny = (int) p->ny; d.nz = (int) p->nz; d.nzh = d.nz / 2 + 1;
   d.nzp = s->fp32 ? (d.nzh + 1) & ~1 : d.nzh;
   d.nxy = (long long) d.nx * d.ny;
   d.npts = d.nxy * d.nz;
   const size_t r = s->fp32 ? 4 : 8;
   s->esz_r = r;
   s->esz_c = 2 * r;
   s->esz_psi = psi_esz(p);
   s->LSr = (int) (d.nz + 16 / s->esz_psi);
   s->LSo = (int) (d.nz + 16 / s->esz_r);

   CK(cudaMalloc(&s->psi, s->esz_psi * d.npts));
   CK(cudaMalloc(&s->spec, s->esz_c * (size_t) d.nzp * d.nxy));
   CK(cudaMalloc(&s->phi, r * d.npts));
   CK(cudaMemsetAsync(s->psi, 0, s->esz_psi * d.npts, s->st));
   s->row_cap = std::max(d.nxy, std::max((long long) d.nx * d.nz, (long long) d.ny * d.nz));
   CK(cudaMalloc(&s->rowA, sizeof(double) * s->row_cap));
   CK(cudaMalloc(&s->rowB, sizeof(double) * s->row_cap));
   CK(cudaMalloc(&s->tmp, sizeof(double) * std::max<long long>(d.nxy, std::max(d.nx, std::max(d.ny, d.nz))) * 2));
   CK(cudaMalloc(&s->obs, sizeof(double) * 64));
   CK(cudaMalloc(&s->rms_buf, sizeof(double) * 4 * kRmsSlots));
   CK(cudaMalloc(&s->state, sizeof(State)));
   State st0{};
   st0.norm = 1.; st0.scale = 1.; st0.scale2 = 1.;
   CK(cudaMemcpyAsync(s->state, &st0, sizeof(State), cudaMemcpyHostToDevice, s->st));

   make_coef(s, 0, d.nx, p->dx * p->dx);
   make_coef(s, 1, d.ny, p->dy * p->dy);
   make_coef(s, 2, d.nz, p->dz * p->dz);
   CKS(make_udd(s));
   // space mesh (initpsi, imag3d-mpicuda.cu:842-855)
   const long nx2 = d.nx / 2, ny2 = d.ny / 2, nz2 = d.nz / 2;
   s->hx.resize(d.nx); s->hy.resize(d.ny); s->hz.resize(d.nz);
   s->hx2.resize(d.nx); s->hy2.resize(d.ny); s->hz2.resize(d.nz);
   for (long i = 0; i < d.nx; i++) { s->hx[i] = (i - nx2) * p->dx; s->hx2[i] = s->hx[i] * s->hx[i]; }
   for (long j = 0; j < d.ny; j++) { s->hy[j] = (j - ny2) * p->dy; s->hy2[j] = s->hy[j] * s->hy[j]; }
   for (long k = 0; k < d.nz; k++) { s->hz[k] = (k - nz2) * p->dz; s->hz2[k] = s->hz[k] * s->hz[k]; }
   void *t = nullptr;
   auto keep_x = [&](const void *p, size_t n) { s->nu_x.assign((const unsigned char *) p, (const unsigned char *) p + n); };
   CKS(upload(s, &t, s->hx2.data(), d.nx)); s->x2 = (double *) t;
   CKS(upload(s, &t, s->hy2.data(), d.ny)); s->y2 = (double *) t;
   CKS(upload(s, &t, s->hz2.data(), d.nz)); s->z2 = (double *) t;
   if (s->fp32) {
      const std::vector<double> *sq[3] = {&s->hx2, &s->hy2, &s->hz2};
      float **dst[3] = {&s->x2f, &s->y2f, &s->z2f};
      for (int a = 0; a < 3; a++) {
         std::vector<float> f(kTabPad, 0.f);
         f.insert(f.end(), sq[a]->begin(), sq[a]->end());
         CKS(upload(s, &t, f.data(), f.size()));
         *dst[a] = (float *) t + kTabPad;
         if (a == 0 && s->cplx) keep_x(f.data() + kTabPad, sizeof(float) * sq[a]->size());
      }
   }
   // trap factors per axis for calcnu: exp(-dt 0.5 par c x^2) in imaginary
   // time; in real time (FP64) the phases exp(-i dt 0.5 par c x^2), stored as
   // (cos, sin) pairs
   if (s->cplx && !s->fp32) {
      const long double hp = 0.5L * (long double) s->par, dt = (long double) p->dt;
      const long double cf[3] = {(long double) p->gamma * p->gamma, (long double) p->nu * p->nu,
                                 (long double) p->lambda * p->lambda};
      const std::vector<double> *sq[3] = {&s->hx2, &s->hy2, &s->hz2};
      for (int a = 0; a < 3; a++) {
         const size_t n = sq[a]->size();
         std::vector<double2> tab(n);
         for (size_t i = 0; i < n; i++) {
            const long double th = -dt * hp * cf[a] * (long double) (*sq[a])[i];
            tab[i] = make_double2((double) cosl(th), (double) sinl(th));
         }
         CKS(upload(s, &s->lin[a], tab.data(), tab.size()));
         if (a == 0) keep_x(tab.data(), sizeof(double2) * tab.size());
      }
   }
   if (!s->cplx) {
      const long double hp = 0.5L * (long double) s->par, dt = (long double) p->dt;
      const long double cf[3] = {(long double) p->gamma * p->gamma, (long double) p->nu * p->nu,
                                 (long double) p->lambda * p->lambda};
      const std::vector<double> *sq[3] = {&s->hx2, &s->hy2, &s->hz2};
      for (int a = 0; a < 3; a++) {
         const size_t n = sq[a]->size();
         std::vector<double> tab(n);
         for (size_t i = 0; i < n; i++) tab[i] = (double) expl(-dt * hp * cf[a] * (long double) (*sq[a])[i]);
         if (s->fp32) {
            std::vector<float> f(kTabPad, 0.f);
            f.insert(f.end(), tab.begin(), tab.end());
            CKS(upload(s, &t, f.data(), f.size()));
            s->lin[a] = (float *) t + kTabPad;
            if (a == 0) keep_x(f.data() + kTabPad, sizeof(float) * n);
         } else {
            CKS(upload(s, &s->lin[a], tab.data(), tab.size()));
            if (a == 0) keep_x(tab.data(), sizeof(double) * n);
         }
      }
   }
   CKS(plan_tiles(s));
   CKS(setup_static(s));

   // (the stream, not the device: another thread may be capturing a batch step)
   CK(cudaStreamSynchronize(s->st));
   return GPE_OK;
}

extern "C" gpe_status gpe_create(const gpe_params *p, void *stream, gpe_solver **out) {
   if (!out) return fail(GPE_ERR_PARAM, "null output handle");
   *out = nullptr;
   CKS(validate(p));
   gpe_solver *s = new gpe_solver();
   gpe_status st = create_impl(p, stream, s);
   if (st != GPE_OK) {
      std::string keep = g_err;
      free_all(s);
      delete s;
      g_err = keep;
      return st;
   }
   *out = s;
   return GPE_OK;
}

extern "C" void gpe_destroy(gpe_solver *s) {
   if (!s) return;
   if (s->st) cudaStreamSynchronize(s->st);
   free_all(s);
   delete s;
}

extern "C" const char *gpe_last_error(void) { return g_err.c_str(); }

#define DISPATCH(s, CALL)                                                                 \
   (((s)->fp32) ? (((s)->cplx) ? Ops<float, true>::CALL : Ops<float, false>::CALL)     \
                : (((s)->cplx) ? Ops<double, true>::CALL : Ops<double, false>::CALL))

#define CHECK_HANDLE(s) \
   if (!(s)) return fail(GPE_ERR_PARAM, "null solver handle")

// ------------------------------------------------------------------ psi I/O
// FP64 arrays are copied as they are (the host layout equals the device
// layout).  A mixed-precision handle converts on the device, through the
// spectrum buffer in pieces (its contents live only inside one convolution):
// converting on the host, through a buffer allocated for the call, took 220
// ms for 512x512x256 points, whose copy takes 10 ms.
static gpe_status fetch(gpe_solver *s, double *host, const void *dev, size_t nd) {
   if (!s->fp32) {
      CK(cudaMemcpyAsync(host, dev, sizeof(double) * nd, cudaMemcpyDeviceToHost, s->st));
   } else {
      const size_t cap = spec_doubles(s);
      for (size_t at = 0; at < nd; at += cap) {
         const size_t m = std::min(cap, nd - at);
         k_convert<<<(unsigned) std::min<size_t>(592, (m + 255) / 256), 256, 0, s->st>>>(
             (double *) s->spec, (const float *) dev + at, (long long) m);
         CKL();
         CK(cudaMemcpyAsync(host + at, s->spec, sizeof(double) * m, cudaMemcpyDeviceToHost, s->st));
         s->launches++;
      }
   }
   CK(cudaStreamSynchronize(s->st));
   return GPE_OK;
}

extern "C" gpe_status gpe_set_psi(gpe_solver *s, const double *psi) {
   CHECK_HANDLE(s);
   if (!psi) return fail(GPE_ERR_PARAM, "null psi");
   CK(cudaSetDevice(s->dev));
   const size_t nd = (size_t) s->d.npts * (s->cplx ? 2 : 1);
   if (s->fp32) {
      const size_t cap = spec_doubles(s);
      for (size_t at = 0; at < nd; at += cap) {
         const size_t m = std::min(cap, nd - at);
         CK(cudaMemcpyAsync(s->spec, psi + at, sizeof(double) * m, cudaMemcpyHostToDevice, s->st));
         k_convert<<<(unsigned) std::min<size_t>(592, (m + 255) / 256), 256, 0, s->st>>>(
             (float *) s->psi + at, (const double *) s->spec, (long long) m);
         CKL();
         s->launches++;
      }
   } else {
      CK(cudaMemcpyAsync(s->psi, psi, sizeof(double) * nd, cudaMemcpyHostToDevice, s->st));
   }
   CK(cudaStreamSynchronize(s->st));
   k_state_set<<<1, 1, 0, s->st>>>(s->state, 1.);
   CKL();
   return GPE_OK;
}

extern "C" gpe_status gpe_get_psi(gpe_solver *s, double *psi) {
   CHECK_HANDLE(s);
   if (!psi) return fail(GPE_ERR_PARAM, "null psi");
   CK(cudaSetDevice(s->dev));
   return fetch(s, psi, s->psi, (size_t) s->d.npts * (s->cplx ? 2 : 1));
}

// initpsi Gaussian (imag3d-mpicuda.cu:835-867), evaluated on the host like
// the reference and uploaded.
extern "C" gpe_status gpe_init_gaussian(gpe_solver *s) {
   CHECK_HANDLE(s);
   const double pi = kRefPi;
   const double cpsi = std::sqrt(pi * std::sqrt(pi / (s->p.gamma * s->p.nu * s->p.lambda)));
   const Dims &d = s->d;
   std::vector<double> re((size_t) d.npts * (s->cplx ? 2 : 1), 0.);
   for (long i = 0; i < d.nx; i++)
      for (long j = 0; j < d.ny; j++)
         for (long k = 0; k < d.nz; k++) {
            const double tmp = std::exp(-0.5 * (s->p.gamma * s->hx2[i] + s->p.nu * s->hy2[j] + s->p.lambda * s->hz2[k]));
            re[(size_t) ((i * d.ny + j) * d.nz + k) * (s->cplx ? 2 : 1)] = tmp / cpsi;
         }
   return gpe_set_psi(s, re.data());
}

extern "C" gpe_status gpe_init_density(gpe_solver *s, const double *rho) {
   CHECK_HANDLE(s);
   if (!rho) return fail(GPE_ERR_PARAM, "null density");
   CK(cudaSetDevice(s->dev));
   double *dr = nullptr;
   CK(cudaMalloc(&dr, sizeof(double) * s->d.npts));
   cudaError_t e = cudaMemcpyAsync(dr, rho, sizeof(double) * s->d.npts, cudaMemcpyHostToDevice, s->st);
   if (e == cudaSuccess) {
      if (s->fp32)
         s->cplx ? k_init_density<float, true><<<592, 256, 0, s->st>>>((float2 *) s->psi, dr, s->d.npts)
                 : k_init_density<float, false><<<592, 256, 0, s->st>>>((float *) s->psi, dr, s->d.npts);
      else
         s->cplx ? k_init_density<double, true><<<592, 256, 0, s->st>>>((double2 *) s->psi, dr, s->d.npts)
                 : k_init_density<double, false><<<592, 256, 0, s->st>>>((double *) s->psi, dr, s->d.npts);
      e = cudaGetLastError();
   }
   cudaError_t e2 = cudaStreamSynchronize(s->st);
   cudaFree(dr);
   if (e != cudaSuccess || e2 != cudaSuccess) return fail(GPE_ERR_CUDA, "init from density failed");
   s->launches++;
   k_state_set<<<1, 1, 0, s->st>>>(s->state, 1.);
   CKL();
   return GPE_OK;
}

// -------------------------------------------------------------- operators
// Reads and clears the device status word; a bounded wait that gave up turns
// into GPE_ERR_TIMEOUT.
static gpe_status check_err(gpe_solver *s) {
   uint32_t e = 0;
   CK(cudaMemcpyAsync(&e, s->err, sizeof(e), cudaMemcpyDeviceToHost, s->st));
   CK(cudaStreamSynchronize(s->st));
   if (e) {
      CK(cudaMemsetAsync(s->err, 0, sizeof(uint32_t), s->st));
      return fail(GPE_ERR_TIMEOUT, "a bounded device wait for a bulk copy gave up");
   }
   return GPE_OK;
}

static gpe_status read_obs(gpe_solver *s, double *dst, int n, int off = 0) {
   CK(cudaMemcpyAsync(dst, s->obs + off, sizeof(double) * n, cudaMemcpyDeviceToHost, s->st));
   CK(cudaStreamSynchronize(s->st));
   return GPE_OK;
}

extern "C" gpe_status gpe_calcnorm(gpe_solver *s, int renormalize, double *norm) {
   CHECK_HANDLE(s);
   CK(cudaSetDevice(s->dev));
   CKS(DISPATCH(s, calcnorm(s, renormalize != 0)));
   double v = 0;
   CKS(read_obs(s, &v, 1));
   if (norm) *norm = v;
   return GPE_OK;
}

extern "C" gpe_status gpe_run(gpe_solver *s, long nsteps, double *g, double *gd, double g_inc, double gd_inc,
                              double *last_norm, long rms_every, double *rms_out) {
   CHECK_HANDLE(s);
   if (!g || !gd) return fail(GPE_ERR_PARAM, "null coupling pointers");
   if (nsteps < 0) return fail(GPE_ERR_PARAM, "negative step count");
   CK(cudaSetDevice(s->dev));
   const bool imag = !s->cplx;
   const long nrms = (rms_every > 0) ? (nsteps + rms_every - 1) / rms_every : 0;
   if (nrms > 0 && !rms_out) return fail(GPE_ERR_PARAM, "rms_out required when rms_every > 0");
   // rms samples land in the handle's preallocated slots (no allocation and
   // no implicit synchronisation inside the run); every kRmsSlots samples the
   // full batch is copied out
   long flushed = 0;  // samples already copied to rms_out
   auto flush = [&](long upto) -> gpe_status {
      if (upto <= flushed) return GPE_OK;
      CK(cudaMemcpyAsync(rms_out + 4 * flushed, s->rms_buf, sizeof(double) * 4 * (upto - flushed),
                         cudaMemcpyDeviceToHost, s->st));
      CK(cudaStreamSynchronize(s->st));
      flushed = upto;
      return GPE_OK;
   };
   gpe_status st = GPE_OK;
   for (long c = 0; c < nsteps && st == GPE_OK; c++) {
      *g += g_inc;
      *gd += gd_inc;
      const bool rms_here = rms_every > 0 && c % rms_every == 0;
      double *slot = nullptr;
      if (rms_here) {
         const long idx = c / rms_every;
         if (idx - flushed == kRmsSlots) st = flush(idx);
         slot = s->rms_buf + 4 * (idx - flushed);
      }
      // real time: the step's z sweep leaves the rms row partials (no extra
      // pass over psi); imaginary time: renormalise first, then a full rms
      if (st == GPE_OK) st = DISPATCH(s, step(s, *g, *gd, s->obs, rms_here && !imag));
      if (st == GPE_OK && rms_here) {
         if (imag) {
            st = DISPATCH(s, apply_scale(s));
            if (st == GPE_OK) st = DISPATCH(s, rms(s, slot));
         } else {
            st = DISPATCH(s, rms_final(s, slot));
         }
      }
   }
   if (st == GPE_OK && imag && nsteps > 0) st = DISPATCH(s, apply_scale(s));
   if (st == GPE_OK && last_norm && imag && nsteps > 0) st = read_obs(s, last_norm, 1);
   if (st == GPE_OK && nrms > 0) st = flush(nrms);
   if (st == GPE_OK) {
      cudaError_t e = cudaStreamSynchronize(s->st);
      if (e != cudaSuccess) st = fail(GPE_ERR_CUDA, cudaGetErrorString(e));
   }
   if (st == GPE_OK) st = check_err(s);
   return st;
}

extern "C" gpe_status gpe_calcmuen(gpe_solver *s, double g, double gd, double *mu, double *en) {
   CHECK_HANDLE(s);
   CK(cudaSetDevice(s->dev));
   CKS(DISPATCH(s, muen(s, g, gd, s->obs + 8)));
   double v[2];
   CKS(read_obs(s, v, 2, 8));
   if (mu) *mu = v[0];
   if (en) *en = v[1];
   return GPE_OK;
}

extern "C" gpe_status gpe_calcrms(gpe_solver *s, double *rms) {
   CHECK_HANDLE(s);
   if (!rms) return fail(GPE_ERR_PARAM, "null rms");
   CK(cudaSetDevice(s->dev));
   CKS(DISPATCH(s, rms(s, s->obs + 16)));
   return read_obs(s, rms, 4, 16);
}

extern "C" gpe_status gpe_psi_center2(gpe_solver *s, double *value) {
   CHECK_HANDLE(s);
   CK(cudaSetDevice(s->dev));
   const Dims &d = s->d;
   const long long q = ((long long) (d.nx / 2) * d.ny + d.ny / 2) * d.nz + d.nz / 2;
   double v[2] = {0, 0};
   if (s->fp32) {
      float f[2] = {0, 0};
      CK(cudaMemcpyAsync(f, (char *) s->psi + q * s->esz_psi, s->esz_psi, cudaMemcpyDeviceToHost, s->st));
      CK(cudaStreamSynchronize(s->st));
      v[0] = f[0]; v[1] = s->cplx ? f[1] : 0.;
   } else {
      CK(cudaMemcpyAsync(v, (char *) s->psi + q * s->esz_psi, s->esz_psi, cudaMemcpyDeviceToHost, s->st));
      CK(cudaStreamSynchronize(s->st));
      if (!s->cplx) v[1] = 0.;
   }
   if (value) *value = v[0] * v[0] + v[1] * v[1];
   return GPE_OK;
}

extern "C" gpe_status gpe_density(gpe_solver *s, int kind, long sx, long sy, long sz, double *out, long cap,
                                  long *count) {
   CHECK_HANDLE(s);
   if (!out) return fail(GPE_ERR_PARAM, "null output");
   if (sx < 1 || sy < 1 || sz < 1) return fail(GPE_ERR_PARAM, "OUTSTPX/Y/Z must be >= 1");
   CK(cudaSetDevice(s->dev));
   return DISPATCH(s, density(s, kind, sx, sy, sz, out, cap, count));
}

extern "C" gpe_status gpe_calcpsidd2(gpe_solver *s) {
   CHECK_HANDLE(s);
   CK(cudaSetDevice(s->dev));
   return DISPATCH(s, psidd2(s));
}

extern "C" gpe_status gpe_get_phi(gpe_solver *s, double *phi) {
   CHECK_HANDLE(s);
   if (!phi) return fail(GPE_ERR_PARAM, "null phi");
   CK(cudaSetDevice(s->dev));
   return fetch(s, phi, s->phi, (size_t) s->d.npts);
}

extern "C" gpe_status gpe_calcnu(gpe_solver *s, double g, double gd) {
   CHECK_HANDLE(s);
   CK(cudaSetDevice(s->dev));
   return DISPATCH(s, calcnu(s, g, gd));
}

extern "C" gpe_status gpe_calclux(gpe_solver *s) {
   CHECK_HANDLE(s);
   CK(cudaSetDevice(s->dev));
   return DISPATCH(s, xsweep(s, false, 0., 0.));
}

extern "C" gpe_status gpe_calcluy(gpe_solver *s) {
   CHECK_HANDLE(s);
   CK(cudaSetDevice(s->dev));
   return DISPATCH(s, ysweep(s));
}

extern "C" gpe_status gpe_calcluz(gpe_solver *s) {
   CHECK_HANDLE(s);
   CK(cudaSetDevice(s->dev));
   return DISPATCH(s, zsweep(s, 0));
}

extern "C" gpe_status gpe_synchronize(gpe_solver *s) {
   CHECK_HANDLE(s);
   CK(cudaStreamSynchronize(s->st));
   return check_err(s);
}

extern "C" gpe_status gpe_selftest_wait_timeout(gpe_solver *s, unsigned spins) {
   CHECK_HANDLE(s);
   if (spins < 1 || spins > (1u << 16)) return fail(GPE_ERR_PARAM, "spins must be in [1, 65536]");
   CK(cudaSetDevice(s->dev));
   k_wait_selftest<<<1, 32, 0, s->st>>>(spins, s->err);
   CKL();
   s->launches++;
   return GPE_OK;
}

extern "C" gpe_status gpe_launch_count(gpe_solver *s, long long *count) {
   CHECK_HANDLE(s);
   if (count) *count = s->launches;
   return GPE_OK;
}

extern "C" gpe_status gpe_time_steps(gpe_solver *s, long nsteps, double g, double gd, double *ms) {
   CHECK_HANDLE(s);
   CK(cudaSetDevice(s->dev));
   cudaEvent_t a, b;
   CK(cudaEventCreate(&a));
   CK(cudaEventCreate(&b));
   CK(cudaEventRecord(a, s->st));
   gpe_status st = GPE_OK;
   for (long c = 0; c < nsteps && st == GPE_OK; c++) st = DISPATCH(s, step(s, g, gd, nullptr));
   if (st == GPE_OK && !s->cplx) st = DISPATCH(s, apply_scale(s));
   CK(cudaEventRecord(b, s->st));
   CK(cudaEventSynchronize(b));
   float f = 0;
   CK(cudaEventElapsedTime(&f, a, b));
   cudaEventDestroy(a);
   cudaEventDestroy(b);
   if (ms) *ms = f;
   return st;
}

extern "C" gpe_status gpe_time_calcpsidd2(gpe_solver *s, long nrep, double *ms) {
   CHECK_HANDLE(s);
   if (nrep < 1) return fail(GPE_ERR_PARAM, "nrep must be >= 1");
   CK(cudaSetDevice(s->dev));
   CKS(DISPATCH(s, psidd2(s)));  // untimed warm-up
   cudaEvent_t a, b;
   CK(cudaEventCreate(&a));
   CK(cudaEventCreate(&b));
   CK(cudaEventRecord(a, s->st));
   gpe_status st = GPE_OK;
   for (long c = 0; c < nrep && st == GPE_OK; c++) st = DISPATCH(s, psidd2(s));
   CK(cudaEventRecord(b, s->st));
   CK(cudaEventSynchronize(b));
   float f = 0;
   CK(cudaEventElapsedTime(&f, a, b));
   cudaEventDestroy(a);
   cudaEventDestroy(b);
   if (ms) *ms = f / nrep;
   if (st == GPE_OK) st = check_err(s);
   return st;
}

// ------------------------------------------------------------ profiling
static const char *kStepKernels[] = {"zfwd_r2c", "yfft_fwd", "xconv_udd", "yfft_inv", "zinv_c2r",
                                     "phi_boundary", "xsweep_calcnu", "ysweep", "zsweep", "norm_final"};

extern "C" const char *gpe_step_kernel_name(gpe_solver *s, int i) {
   const int n = (s && s->cplx) ? 9 : 10;
   if (i < 0 || i >= n) return nullptr;
   if (i == 8 && s && !s->cplx) return "zsweep_norm";
   return kStepKernels[i];
}

// Compulsory bytes of one launch of kernel i for this pass structure.
extern "C" double gpe_step_kernel_bytes(gpe_solver *s, int i) {
   if (!s) return 0.;
   const Dims &d = s->d;
   const double sp = (double) s->esz_psi, sc = (double) s->esz_c, r = (double) s->esz_r;
   const double npts = (double) d.npts, half = (double) d.nzh * (double) d.nxy;
   const double oct = (double) d.nzh * (d.nx / 2 + 1) * (d.ny / 2 + 1) * 8.;
   switch (i) {
   case 0: return npts * sp + half * sc;
   case 1: case 3: return 2. * half * sc;
   case 2: return 2. * half * sc + oct;
   case 4: return half * sc + npts * r;  // with the boundary planes (a rewrite of rows it stores anyway)
   case 5: return 0.;                    // folded into case 4
   case 6: return npts * (2. * sp + r);
   case 7: return 2. * npts * sp;
   case 8: return 2. * npts * sp;
   case 9: return 0.;  // folded into case 8
   default: return 0.;
   }
}

extern "C" gpe_status gpe_profile_step(gpe_solver *s, long nsteps, double g, double gd, double *ms, int cap,
                                       int *count) {
   CHECK_HANDLE(s);
   if (!ms || nsteps < 1) return fail(GPE_ERR_PARAM, "profile needs an output array and nsteps >= 1");
   CK(cudaSetDevice(s->dev));
   const int nk = s->cplx ? 9 : 10;
   if (cap < nk) return fail(GPE_ERR_PARAM, "profile output array too small");
   std::vector<cudaEvent_t> ev((size_t) (nsteps * (nk + 1)));
   for (auto &e : ev) CK(cudaEventCreate(&e));
   std::vector<double> acc(nk, 0.);
   gpe_status st = GPE_OK;
   for (long c = 0; c < nsteps && st == GPE_OK; c++) {
      cudaEvent_t *base = ev.data() + c * (nk + 1);
      cudaEventRecord(base[0], s->st);
      s->prof_ev = base + 1;
      s->prof_i = 0;
      s->prof_cap = nk;
      st = DISPATCH(s, step(s, g, gd, nullptr));
      s->prof_ev = nullptr;
   }
   if (st == GPE_OK && !s->cplx) st = DISPATCH(s, apply_scale(s));
   cudaError_t e = cudaStreamSynchronize(s->st);
   if (st == GPE_OK && e != cudaSuccess) st = fail(GPE_ERR_CUDA, cudaGetErrorString(e));
   if (st == GPE_OK) {
      for (long c = 0; c < nsteps; c++) {
         cudaEvent_t *base = ev.data() + c * (nk + 1);
         for (int i = 0; i < nk; i++) {
            float f = 0.f;
            cudaEventElapsedTime(&f, base[i], base[i + 1]);
            acc[i] += f;
         }
      }
      for (int i = 0; i < nk; i++) ms[i] = acc[i] / (double) nsteps;
      if (count) *count = nk;
   }
   for (auto &x : ev) cudaEventDestroy(x);
   return st;
}

// ------------------------------------------------------------------ tuning
extern "C" gpe_status gpe_get_tuning(gpe_solver *s, gpe_tuning *t) {
   CHECK_HANDLE(s);
   if (!t) return fail(GPE_ERR_PARAM, "null tuning");
   for (int a = 0; a < 3; a++) {
      t->sweep_tw[a] = s->sw[a].TW;
      t->sweep_stages[a] = s->sw[a].S;
      t->sweep_seg[a] = s->sw[a].MSEG;
   }
   t->fft_tile[0] = s->Ly;
   t->fft_tile[1] = s->Lx;
   t->fft_max_radix = s->tune.fft_max_radix > 0 ? s->tune.fft_max_radix : (s->fp32 ? 16 : 8);
   return GPE_OK;
}

extern "C" gpe_status gpe_set_tuning(gpe_solver *s, const gpe_tuning *t) {
   CHECK_HANDLE(s);
   CK(cudaSetDevice(s->dev));
   CK(cudaStreamSynchronize(s->st));  // queued kernels still read the old tables
   const gpe_tuning old = s->tune;
   s->tune = t ? *t : gpe_tuning{};
   gpe_status st = plan_tiles(s);
   if (st != GPE_OK) {
      const std::string msg = g_err;
      s->tune = old;
      plan_tiles(s);
      return fail(st, msg);
   }
   return GPE_OK;
}

// Per-kernel times of the step (index as gpe_step_kernel_name) for the
// configuration in use; psi advances by warm + nsteps steps.
static gpe_status time_kernels(gpe_solver *s, double g, double gd, int nsteps, double *ms) {
   double warm[10];
   int cnt = 0;
   CKS(gpe_profile_step(s, 1, g, gd, warm, 10, &cnt));
   return gpe_profile_step(s, nsteps, g, gd, ms, 10, &cnt);
}

extern "C" gpe_status gpe_autotune(gpe_solver *s, double g, double gd, int nsteps, gpe_tuning *best) {
   CHECK_HANDLE(s);
   if (nsteps < 1) return fail(GPE_ERR_PARAM, "autotune needs nsteps >= 1");
   CK(cudaSetDevice(s->dev));
   gpe::Stash keep;  // psi and the step state, put back at the end
   CKS(gpe::stash_take(s, &keep));
   const gpe_tuning start = s->tune;
   gpe_tuning pick = start;
   double best_sweep[3] = {1e30, 1e30, 1e30}, best_y = 1e30, best_x = 1e30, best_fft = 1e30;
   const int ksw[3] = {6, 7, 8};  // x, y, z sweeps in the kernel list
   gpe_status st = GPE_OK;
   // sweeps: every available (lines per CTA, segment length) pair with both
   // pipeline depths; the three axes are timed together, candidate c of
   // each (its last one once an axis has fewer)
   {
      const long nn[3] = {s->d.nx, s->d.ny, s->d.nz};
      int cTW[3][kSweepCand], cM[3][kSweepCand], cP[kSweepCand], nc[3];
      bool prim[kSweepCand];
      for (int a = 0; a < 3; a++)
         nc[a] = sweep_candidates((int) nn[a], (int) (128 / s->esz_psi), (int) s->esz_psi, cTW[a], cM[a], cP, prim);
      const int ncmax = std::max(nc[0], std::max(nc[1], nc[2]));
      for (int c = 0; c < ncmax && st == GPE_OK; c++)
         for (int S = 2; S <= 3 && st == GPE_OK; S++) {
            gpe_tuning t = start;
            for (int a = 0; a < 3; a++) {
               t.sweep_tw[a] = cTW[a][std::min(c, nc[a] - 1)];
               t.sweep_seg[a] = cM[a][std::min(c, nc[a] - 1)];
               t.sweep_stages[a] = S;
            }
            s->tune = t;
            if (plan_tiles(s) != GPE_OK) continue;  // does not fit: skip
            double ms[10];
            st = time_kernels(s, g, gd, nsteps, ms);
            for (int a = 0; a < 3 && st == GPE_OK; a++)
               if (ms[ksw[a]] < best_sweep[a]) {
                  best_sweep[a] = ms[ksw[a]];
                  pick.sweep_tw[a] = t.sweep_tw[a];
                  pick.sweep_seg[a] = t.sweep_seg[a];
                  pick.sweep_stages[a] = S;
               }
         }
   }
   // FFT: tile widths of the y and x passes, then the largest radix
   for (int L = 128 / (int) s->esz_c; L >= 2 && st == GPE_OK; L /= 2) {
      gpe_tuning t = pick;
      t.fft_tile[0] = t.fft_tile[1] = L;
      s->tune = t;
      if (plan_tiles(s) != GPE_OK) continue;
      double ms[10];
      st = time_kernels(s, g, gd, nsteps, ms);
      if (st != GPE_OK) break;
      if (ms[1] + ms[3] < best_y) { best_y = ms[1] + ms[3]; pick.fft_tile[0] = L; }
      if (ms[2] < best_x) { best_x = ms[2]; pick.fft_tile[1] = L; }
   }
   for (int r = s->fp32 ? 16 : 8; r >= 2 && st == GPE_OK; r /= 2) {
      gpe_tuning t = pick;
      t.fft_max_radix = r;
      s->tune = t;
      if (plan_tiles(s) != GPE_OK) continue;
      double ms[10];
      st = time_kernels(s, g, gd, nsteps, ms);
      if (st != GPE_OK) break;
      const double f = ms[0] + ms[1] + ms[2] + ms[3] + ms[4];
      if (f < best_fft) { best_fft = f; pick.fft_max_radix = r; }
   }
   // the per-kernel choices are combined: keep them only if whole steps
   // (launched as a run launches them, each kernel overlapping the drain of
   // the one before) are faster than with the configuration the tuner
   // started from (on B200 the combined picks once made the mixed real-time
   // step 13 % slower)
   if (st == GPE_OK) {
      double t_pick = 1e30, t_start = 1e30;
      const gpe_tuning cand[2] = {pick, start};
      double *tt[2] = {&t_pick, &t_start};
      for (int k = 0; k < 2 && st == GPE_OK; k++) {
         s->tune = cand[k];
         st = plan_tiles(s);
         double ms = 0.;
         if (st == GPE_OK) st = gpe_time_steps(s, 1, g, gd, &ms);
         for (int r = 0; r < 2 && st == GPE_OK; r++) {
            st = gpe_time_steps(s, 2 * nsteps, g, gd, &ms);
            *tt[k] = std::min(*tt[k], ms);
         }
      }
      if (st == GPE_OK && t_pick >= t_start) pick = start;
   }
   s->tune = st == GPE_OK ? pick : start;
   gpe_status st2 = plan_tiles(s);
   gpe_status st3 = gpe::stash_restore(s, &keep);
   if (st != GPE_OK) return st;
   if (st2 != GPE_OK) return st2;
   if (st3 != GPE_OK) return st3;
   if (best) return gpe_get_tuning(s, best);  // every field filled in
   return GPE_OK;
}

// ------------------------------------------------------ hooks (internal.h)
namespace gpe {

gpe_status queue_steps(gpe_solver *s, long nsteps, double g, double gd) {
   CHECK_HANDLE(s);
   for (long c = 0; c < nsteps; c++) CKS(DISPATCH(s, step(s, g, gd, nullptr)));
   return GPE_OK;
}

gpe_status queue_finish(gpe_solver *s) {
   CHECK_HANDLE(s);
   if (!s->cplx) return DISPATCH(s, apply_scale(s));
   return GPE_OK;
}

gpe_status queue_muen(gpe_solver *s, double g, double gd) {
   CHECK_HANDLE(s);
   return DISPATCH(s, muen(s, g, gd, s->obs + 8));
}

gpe_status read_muen(gpe_solver *s, double *mu, double *en) {
   CHECK_HANDLE(s);
   double v[2];
   CKS(read_obs(s, v, 2, 8));
   CKS(check_err(s));
   if (mu) *mu = v[0];
   if (en) *en = v[1];
   return GPE_OK;
}

cudaStream_t stream_of(gpe_solver *s) { return s->st; }
gpe_status params_of(gpe_solver *s, gpe_params *p) {
   CHECK_HANDLE(s);
   *p = s->p;
   return GPE_OK;
}
int device_of(gpe_solver *s) { return s->dev; }
unsigned long long plan_generation(gpe_solver *s) { return s->plan_gen; }
gpe_status tuning_as_set(gpe_solver *s, gpe_tuning *t) {
   CHECK_HANDLE(s);
   *t = s->tune;
   return GPE_OK;
}

gpe_status batch_geom(gpe_solver *s, int Ly, int Lx, BatchGeom *geom) {
   CHECK_HANDLE(s);
   return DISPATCH(s, geom(s, Ly, Lx, geom));
}

gpe_status batch_desc(gpe_solver *s, int Ly, int Lx, double g, double gd, BatchDesc *out) {
   CHECK_HANDLE(s);
   return DISPATCH(s, desc(s, Ly, Lx, g, gd, out));
}

static_assert(sizeof(State) <= sizeof(Stash::state), "step state larger than its stash");

gpe_status stash_take(gpe_solver *s, Stash *k) {
   CHECK_HANDLE(s);
   if (!k || k->psi) return fail(GPE_ERR_PARAM, "stash: null or already holding a copy");
   CK(cudaSetDevice(s->dev));
   k->bytes = s->esz_psi * (size_t) s->d.npts;
   CK(cudaMalloc(&k->psi, k->bytes));
   cudaError_t e = cudaMemcpyAsync(k->psi, s->psi, k->bytes, cudaMemcpyDeviceToDevice, s->st);
   if (e == cudaSuccess) e = cudaMemcpyAsync(k->state, s->state, sizeof(State), cudaMemcpyDeviceToHost, s->st);
   if (e == cudaSuccess) e = cudaStreamSynchronize(s->st);
   if (e != cudaSuccess) {
      stash_drop(k);
      return fail(GPE_ERR_CUDA, cudaGetErrorString(e));
   }
   return GPE_OK;
}

gpe_status stash_restore(gpe_solver *s, Stash *k) {
   CHECK_HANDLE(s);
   if (!k || !k->psi) return fail(GPE_ERR_PARAM, "stash: nothing to restore");
   CK(cudaSetDevice(s->dev));
   cudaError_t e = cudaMemcpyAsync(s->psi, k->psi, k->bytes, cudaMemcpyDeviceToDevice, s->st);
   if (e == cudaSuccess) e = cudaMemcpyAsync(s->state, k->state, sizeof(State), cudaMemcpyHostToDevice, s->st);
   if (e == cudaSuccess) e = cudaStreamSynchronize(s->st);
   stash_drop(k);
   if (e != cudaSuccess) return fail(GPE_ERR_CUDA, cudaGetErrorString(e));
   return GPE_OK;
}

void stash_drop(Stash *k) {
   if (k && k->psi) cudaFree(k->psi);
   if (k) k->psi = nullptr;
}

}  // namespace gpe

// --------------------------------------------------------------- snapshots
namespace {
struct SnapHeader {
   char magic[8];           // "GPESNAP1"
   uint32_t header_bytes;   // 192 (the header is zero-padded to that size)
   uint32_t version;        // 1
   gpe_params p;
   double g, gd;
   long long step;
   unsigned long long payload_bytes;
   unsigned long long fnv1a;
};
static_assert(sizeof(gpe_params) == 104, "gpe_params layout");
constexpr size_t kSnapHeaderBytes = 192;
static_assert(sizeof(SnapHeader) <= kSnapHeaderBytes, "snapshot header size");

unsigned long long fnv1a(const unsigned char *p, size_t n) {
   unsigned long long h = 1469598103934665603ULL;
   for (size_t i = 0; i < n; i++) {
      h ^= p[i];
      h *= 1099511628211ULL;
   }
   return h;
}
}  // namespace

extern "C" gpe_status gpe_snapshot_save(gpe_solver *s, const char *path, double g, double gd, long long step) {
   CHECK_HANDLE(s);
   if (!path) return fail(GPE_ERR_PARAM, "null path");
   CK(cudaSetDevice(s->dev));
   State st{};
   CK(cudaMemcpyAsync(&st, s->state, sizeof(State), cudaMemcpyDeviceToHost, s->st));
   CK(cudaStreamSynchronize(s->st));
   if (st.scale != 1.) CKS(DISPATCH(s, apply_scale(s)));
   const size_t nbytes = s->esz_psi * (size_t) s->d.npts;
   std::vector<unsigned char> buf(kSnapHeaderBytes + nbytes, 0);
   CK(cudaMemcpyAsync(buf.data() + kSnapHeaderBytes, s->psi, nbytes, cudaMemcpyDeviceToHost, s->st));
   CK(cudaStreamSynchronize(s->st));
   SnapHeader h{};
   std::memcpy(h.magic, "GPESNAP1", 8);
   h.header_bytes = (uint32_t) kSnapHeaderBytes;
   h.version = 1;
   h.p = s->p;
   h.g = g;
   h.gd = gd;
   h.step = step;
   h.payload_bytes = nbytes;
   h.fnv1a = fnv1a(buf.data() + kSnapHeaderBytes, nbytes);
   std::memcpy(buf.data(), &h, sizeof(h));
   FILE *f = std::fopen(path, "wb");
   if (!f) return fail(GPE_ERR_IO, std::string("cannot create ") + path);
   const size_t w = std::fwrite(buf.data(), 1, buf.size(), f);
   const int c = std::fclose(f);
   if (w != buf.size() || c != 0) return fail(GPE_ERR_IO, std::string("short write to ") + path);
   return GPE_OK;
}

extern "C" gpe_status gpe_snapshot_load(gpe_solver *s, const char *path, double *g, double *gd, long long *step) {
   CHECK_HANDLE(s);
   if (!path) return fail(GPE_ERR_PARAM, "null path");
   FILE *f = std::fopen(path, "rb");
   if (!f) return fail(GPE_ERR_IO, std::string("cannot open ") + path);
   SnapHeader h{};
   unsigned char hb[kSnapHeaderBytes];
   const size_t r = std::fread(hb, 1, kSnapHeaderBytes, f);
   std::memcpy(&h, hb, sizeof(h));
   if (r != kSnapHeaderBytes || std::memcmp(h.magic, "GPESNAP1", 8) != 0 || h.version != 1 ||
       h.header_bytes != kSnapHeaderBytes) {
      std::fclose(f);
      return fail(GPE_ERR_IO, std::string(path) + " is not a version-1 solver snapshot");
   }
   if (h.p.nx != s->p.nx || h.p.ny != s->p.ny || h.p.nz != s->p.nz || h.p.mode != s->p.mode ||
       h.p.precision != s->p.precision) {
      std::fclose(f);
      return fail(GPE_ERR_PARAM, "snapshot grid, mode or precision differs from the handle's");
   }
   const size_t nbytes = s->esz_psi * (size_t) s->d.npts;
   std::vector<unsigned char> buf(nbytes);
   const size_t rp = h.payload_bytes == nbytes ? std::fread(buf.data(), 1, nbytes, f) : 0;
   std::fclose(f);
   if (rp != nbytes || fnv1a(buf.data(), nbytes) != h.fnv1a)
      return fail(GPE_ERR_IO, std::string(path) + ": payload short or checksum mismatch");
   CK(cudaSetDevice(s->dev));
   CK(cudaMemcpyAsync(s->psi, buf.data(), nbytes, cudaMemcpyHostToDevice, s->st));
   CK(cudaStreamSynchronize(s->st));
   k_state_set<<<1, 1, 0, s->st>>>(s->state, 1.);
   CKL();
   if (g) *g = h.g;
   if (gd) *gd = h.gd;
   if (step) *step = h.step;
   return GPE_OK;
}
