// batch_kernels.cuh -- one launch per pass of the split step over many
// independent solves (gpe_batch_* in include/gpe.h).
//
// The reference runs one solve per MPI job; a batch steps many solves with
// their own grids, parameters and couplings together.  Every pass of the step
// (z forward FFT, y FFT, x convolution, inverse y FFT, z inverse FFT, phi
// boundary planes, x sweep with calcnu, y sweep, z sweep, norm) is ONE launch
// over the tiles of all instances of a group (same mode and precision; mixed
// precision folds the boundary planes into the z inverse pass): a
// per-instance descriptor table in device memory holds each instance's
// dimensions, pointers, FFT plans, coefficient tables, couplings and TMA
// tensor maps, and a work list per pass maps a tile to its instance and its
// place in that instance.  The per-tile arithmetic is the single
// solve's own (the *_body functions of step_kernels.cuh and the sweep helpers
// of sweep_kernels.cuh), so an instance's step is bit for bit its solo step.
//
// Tensor maps read from global memory are acquired through the tensormap
// proxy (fence.proxy.tensormap::generic.acquire) by the thread that issues
// the copies, before their first use in the CTA (and again whenever a
// persistent CTA moves on to another instance).
#pragma once

#include "step_kernels.cuh"
#include "sweep_kernels.cuh"

namespace gpe {

// Everything one sweep tile of one instance needs, next to its tables (a
// 16-byte multiple: it travels to shared memory as one bulk copy).
struct alignas(16) SweepView {
   SegTab tb;
   Trap trap;
   LinPhase lin;
   Dims d;
   const State *st;
   uint32_t *err;
   void *psi;               // z sweep: psi rows
   ZOut zo;                 // z sweep: norm and rms partials
   double g, gd, dt;
   int TW, boxn, nbox, LS;
};

// Passes of the step (work-list index).
enum BatchPass { kPZfwd = 0, kPYfft, kPXconv, kPYinv, kPZinv, kPPhifix, kPXsweep, kPYsweep, kPZsweep, kPNorm, kNPass };

// One instance of a batch.  Tensor maps need 64-byte alignment; the table is
// a cudaMalloc'd array of these.
struct alignas(64) BatchDesc {
   CUtensorMap tm_psi[2];  // x and y sweep tiles of psi
   CUtensorMap tm_phi;     // x sweep tiles of phi
   CUtensorMap tm_spec_y, tm_spec_x;
   SweepView sv[3];
   FftPlan px, pxi, py, ph;
   Dims d;
   void *psi, *spec, *phi;
   const void *twx, *twy, *twz;  // roots of unity (ztab_roots in step_kernels.cuh)
   int fastx, fasty, fastz;      // compile-time passes
   const double *udd;
   State *state;
   uint32_t *err;
   double *rowA;
   double hx, hy;
   int LSr, LSo, boxy, nboxy, boxx, nboxx, Ly, Lx;
};

// One tile of a sweep.
struct alignas(16) SweepTile {
   int inst;
   int a, b;          // x / y sweep: plane, first z column; z sweep: first row, rows
   int geo;           // sweep_geo
   const void *tabs;  // the instance's coefficient tables (and calcnu's x table)
   union {
      const State *st;   // x sweep: the pending renormalisation
      void *psi;         // z sweep: the tile's first row
   };
};
static_assert(sizeof(SweepTile) == 32, "tile record");
// Lines of n points, TW per tile; x / y: rows staged, z: row stride in `ext`.
__host__ __device__ __forceinline__ int sweep_geo(int n, int ext, int TW, int skip) {
   int lg = 0;
   while ((1 << lg) < TW) lg++;
   return n | ext << 11 | lg << 23 | skip << 26;
}
struct SweepGeo {
   int n, ext, TW, skip;
};
__device__ __forceinline__ SweepGeo sweep_geo(int g) {
   return SweepGeo{g & 2047, g >> 11 & 4095, 1 << (g >> 23 & 7), (int) ((unsigned) g >> 26)};
}
// Bytes of an instance's table block: gamma | (M, alpha) | N and, for the x
// sweep, calcnu's table along the line (xe bytes per entry) behind its zero
// entries.
__host__ __device__ __forceinline__ uint32_t sweep_tab_bytes(int n, int skip, int esz, int xe) {
   return (uint32_t) (4 * (n - 2 + skip) * esz + (((n + skip) * xe + 15) & ~15));
}
// Bytes of an entry of calcnu's x table (NuXf::T).
template <class R, bool CPLX> __host__ __device__ constexpr int nu_tab_esz() {
   return (int) sizeof(R) * (CPLX && sizeof(R) == 8 ? 2 : 1);
}

// Launch geometry of one instance under the batch's fixed tile choices (z
// passes: 8-row tiles; y / x passes: Ly / Lx kz columns; sweeps: the
// instance's own lines per CTA and segments, 2-stage pipelines).
struct BatchGeom {
   long long tiles[kNPass];  // CTAs (FFT passes, norm, planes) or tiles (sweeps)
   unsigned threads[kNPass]; // (0: an FFT pass of run-time length, whose group decides)
   long pts[kNPass];         // FFT passes: points of a tile of run-time length, else 0
   size_t smem[kNPass];      // dynamic shared memory of one CTA (FFT passes)
   bool lens[kNPass];        // FFT passes: a compile-time length
   int ppt[kNPass];          // FFT passes (group): points per thread at run-time lengths
   int mseg[3];              // compile-time segment bound of each sweep
   uint32_t stage[3];        // sweeps: bytes of one pipeline stage
   uint32_t xch[3];          // sweeps: bytes of the exchange buffer
   uint32_t tabs[3];         // sweeps: bytes of the table block
   SweepTile tile[3];        // sweeps: the tiles' geo, tabs and state or psi
   int across[3], tw[3];     // sweeps: x / y tiles per plane, lines per tile
   long long nxy;            // z sweep: rows, bytes of a row
   size_t row_bytes;
   uint32_t part;            // z sweep: bytes of one Simpson partial array
   int Ly, Lx;               // the instance's own FFT tile widths
};

__device__ __forceinline__ void tmap_acquire(const CUtensorMap *m) {
   asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(m) : "memory");
}

// Work list of a pass: entry t packs the instance owning tile t (high
// kInstBits bits) and the tile's index within that instance (low bits), so a
// CTA finds its instance with one load.
constexpr int kInstBits = 12;
constexpr int kLocalBits = 32 - kInstBits;
struct TileRef {
   int inst, local;
};
__device__ __forceinline__ TileRef tile_ref(const unsigned *__restrict__ work, int t) {
   const unsigned w = __ldg(work + t);
   return TileRef{(int) (w >> kLocalBits), (int) (w & ((1u << kLocalBits) - 1u))};
}

// Copies a plan into shared memory (every thread of the CTA calls it); the
// FFT stages index its arrays with run-time stage numbers.
__device__ __forceinline__ void stage_plan(FftPlan &dst, const FftPlan &src) {
   constexpr int W = (int) (sizeof(FftPlan) / sizeof(int));
   static_assert(sizeof(FftPlan) % sizeof(int) == 0, "plan size");
   for (int e = threadIdx.x; e < W; e += blockDim.x) ((int *) &dst)[e] = ((const int *) &src)[e];
   __syncthreads();
}

// Resident CTAs of 256 threads per SM (register budgets): 128 registers for
// the FP64 FFT passes with compile-time transforms, which hold 16 points per
// thread, 64 for the others; the sweeps as sweep_ctas, with 80 for the FP32 ones of
// up to 16-point segments, which hold the code of two segment lengths, and one
// CTA fewer for FP32 x sweeps in real time (`nu`), whose calcnu takes the whole
// view's constants into registers: at 64 registers it spilled 244 bytes a thread
// (batches of 160x144x120, 80^3, 48^3: 231, 162, 61 us; at 80 registers 138, 117,
// 48).
template <class R, bool LENS> constexpr int kb_fft_ctas() { return sizeof(R) == 8 && LENS ? 2 : 4; }
__host__ __device__ constexpr int kb_sweep_ctas(bool fp32, bool cplx, int m, bool nu) {
   if (fp32 && cplx && nu) return m == 16 ? 2 : 3;
   return fp32 && m == 16 ? 3 : sweep_ctas(fp32, cplx, m);
}

// ---------------------------------------------------------------- FFT passes
// One CTA per tile; tile numbering of each instance as its single-solve grid.
// LENS: some instance of the group has a compile-time length in this pass.  A
// group without one runs kernels that hold the run-time pass alone, on half the
// registers in FP64 (us of the FFT passes of a step: FP64 imaginary time, 16 grids
// of 72^3 355 -> 246, 24 of 40^3 124 -> 100; FP32 real time, 6 of 160x144x120 407
// -> 357).
// PPT: points per thread at run-time lengths.  Beside compile-time transforms,
// whose registers they then have, FP64 tiles of more than a warp's 256 points take
// 16 (us, 8 -> 16: y pass of 80^3 78 -> 63, x pass of 72^3 102 -> 86; tiles of one
// warp are slower with 16, z pass of 100x90x60 56 -> 63); FP32 always does.
template <class R> constexpr int batch_ppt(bool lens, long pts) {
   return sizeof(R) == 4 || pts > (lens ? 256 : 2048) ? 16 : 8;
}
template <bool LENS, class F> __device__ __forceinline__ void batch_len(int n, F f) {
   if constexpr (LENS) with_len(n, f);
   else f(std::integral_constant<int, 0>());
}

template <class R, bool CPLX, int PPT, int L, bool LENS>
__global__ void __launch_bounds__(256, kb_fft_ctas<R, LENS>()) kb_zfwd(const BatchDesc *__restrict__ tab,
                                                                const unsigned *__restrict__ work) {
   const TileRef r = tile_ref(work, blockIdx.x);
   const BatchDesc &D = tab[r.inst];
   using P = typename Tr<R, CPLX>::P;
   __shared__ FftPlan pl;
   const Dims d = D.d;
   const long long r0 = (long long) r.local * L;
   batch_len<LENS>(D.fastz ? d.nz / 2 : 0, [&](auto nc) {
      constexpr int H = decltype(nc)::value;
      if constexpr (H > 0 && H <= kLenMaxH && L == kLenRows) {
         zfwd_body_n<R, CPLX, L, H>((const P *) D.psi, (cpx<R> *) D.spec, d, (const cpx<R> *) D.twz, D.err, r0);
      } else if constexpr (H == 0) {
         stage_plan(pl, D.ph);
         zfwd_body<R, CPLX, PPT, L>((const P *) D.psi, (cpx<R> *) D.spec, d, pl, (const cpx<R> *) D.twz, D.LSr, D.err, r0);
      }
   });
}

template <class R, bool INV, int PPT, int L, bool LENS>
__global__ void __launch_bounds__(256, kb_fft_ctas<R, LENS>()) kb_yfft(const BatchDesc *__restrict__ tab,
                                                  const unsigned *__restrict__ work) {
   const TileRef r = tile_ref(work, blockIdx.x);
   const BatchDesc &D = tab[r.inst];
   __shared__ FftPlan pl;
   if (threadIdx.x == 0) tmap_acquire(&D.tm_spec_y);
   const Dims d = D.d;
   batch_len<LENS>(D.fasty ? d.ny : 0, [&](auto nc) {
      constexpr int N = decltype(nc)::value, LT = N > 0 ? LenCols<R>::L : L;
      const int nkb = (d.nzh + LT - 1) / LT;
      const int x = r.local / nkb, k0 = (r.local - x * nkb) * LT;
      if constexpr (N > 0) {
         yfft_body_n<R, INV, LT, N>(&D.tm_spec_y, (const cpx<R> *) D.twy, D.err, x, k0);
      } else {
         stage_plan(pl, D.py);
         yfft_body<R, INV, L, PPT>(&D.tm_spec_y, d, pl, (const cpx<R> *) D.twy, D.boxy, D.nboxy, D.err, x, k0);
      }
   });
}

template <class R, int PPT, int L, bool LENS>
__global__ void __launch_bounds__(256, kb_fft_ctas<R, LENS>()) kb_xconv(const BatchDesc *__restrict__ tab,
                                                   const unsigned *__restrict__ work) {
   const TileRef r = tile_ref(work, blockIdx.x);
   const BatchDesc &D = tab[r.inst];
   __shared__ FftPlan pl, pli;
   if (threadIdx.x == 0) tmap_acquire(&D.tm_spec_x);
   const Dims d = D.d;
   batch_len<LENS>(D.fastx ? d.nx : 0, [&](auto nc) {
      constexpr int N = decltype(nc)::value, LT = N > 0 ? LenCols<R>::L : L;
      const int nkb = (d.nzh + LT - 1) / LT;
      const int y = r.local / nkb, k0 = (r.local - y * nkb) * LT;
      if constexpr (N > 0) {
         xconv_body_n<R, LT, N>(&D.tm_spec_x, nullptr, D.udd, d, (const cpx<R> *) D.twx, D.state, D.err, y, k0);
      } else {
         stage_plan(pl, D.px);
         stage_plan(pli, D.pxi);
         xconv_body<R, L, PPT>(&D.tm_spec_x, nullptr, D.udd, d, pl, pli, (const cpx<R> *) D.twx, D.state, D.boxx,
                          D.nboxx, D.err, y, k0);
      }
   });
}

template <class R, int PPT, int L, bool FOLD, bool LENS>
__global__ void __launch_bounds__(256, kb_fft_ctas<R, LENS>()) kb_zinv(const BatchDesc *__restrict__ tab,
                                                                const unsigned *__restrict__ work) {
   const TileRef r = tile_ref(work, blockIdx.x);
   const BatchDesc &D = tab[r.inst];
   __shared__ FftPlan pl;
   const Dims d = D.d;
   const long long r0 = (long long) r.local * L;
   batch_len<LENS>(D.fastz ? d.nz / 2 : 0, [&](auto nc) {
      constexpr int H = decltype(nc)::value;
      if constexpr (H > 0 && H <= kLenMaxH && L == kLenRows) {
         zinv_body_n<R, L, H, FOLD>((const cpx<R> *) D.spec, (R *) D.phi, d, (const cpx<R> *) D.twz, D.err, r0);
      } else if constexpr (H == 0) {
         stage_plan(pl, D.ph);
         zinv_body<R, PPT, L, FOLD>((const cpx<R> *) D.spec, (R *) D.phi, d, pl, (const cpx<R> *) D.twz, D.LSo, D.err, r0);
      }
   });
}

template <class R>
__global__ void kb_phifix(const BatchDesc *__restrict__ tab, const unsigned *__restrict__ work) {
   const TileRef r = tile_ref(work, blockIdx.x);
   const BatchDesc &D = tab[r.inst];
   const Dims d = D.d;
   phifix_body<R>((R *) D.phi, d, r.local);
}

// The norm of one instance per CTA, from its z sweep's tile partials.
static __global__ void __launch_bounds__(256) kb_norm_final(const BatchDesc *__restrict__ tab,
                                                            const unsigned *__restrict__ work) {
   const TileRef r = tile_ref(work, blockIdx.x);
   const BatchDesc &D = tab[r.inst];
   __shared__ double red[8];
   const double sum = sum_tiles(D.rowA, (int) ((D.d.nxy + D.sv[2].TW - 1) / D.sv[2].TW), red);
   if (threadIdx.x == 0) set_norm(D.state, sum, D.hx, D.hy, nullptr);
}

// ------------------------------------------------------------------- sweeps
// Persistent pipelined CTAs over the tiles of all instances (the pipeline of
// k_sweep_xy / k_sweep_z): while a CTA sweeps tile t, tile t + gridDim.x
// (usually of another instance) is loading.  Every stage has room for the
// largest tile of the group (stage_bytes).  Nothing a tile needs is fetched
// when it is due: its record comes three tiles ahead into a ring, and where the
// instance changes its view and tables come with the tile, as bulk copies on
// the same mbarrier, into the other of two buffers (looked up in global
// memory by every tile, the records, views and tables cost a chain of L2
// latencies per tile that every warp waited for at the next barrier: 64
// mixed-precision grids, x / y / z sweep 286 / 155 / 154 -> 269 /
// 136 / 122 us).
template <class R, bool CPLX> struct BatchTabs {
   using P = typename Tr<R, CPLX>::P;
   // the view's tables in shared memory: gamma | (M, alpha) | N | calcnu's x table
   __device__ __forceinline__ static SegTab at(const SegTab &tb, unsigned char *tabs) {
      SegTab o = tb;
      const int ne = tb.P * tb.m;
      o.ga = tabs;
      o.ma = (P *) tabs + ne;
      o.nn = (P *) tabs + 3 * ne;
      return o;
   }
   __device__ __forceinline__ static const void *xt(const SegTab &tb, unsigned char *tabs) {
      return (P *) tabs + 4 * tb.P * tb.m;
   }
};

template <class R, bool CPLX, int AXIS, bool NU, int MSEG, int S>
__global__ void __launch_bounds__(256, kb_sweep_ctas(sizeof(R) == 4, CPLX, MSEG, NU)) kb_sweep_xy(
    const BatchDesc *__restrict__ tab, const SweepTile *__restrict__ tiles, int ntiles, uint32_t stage_bytes,
    uint32_t xch_bytes, uint32_t tab_bytes, int nbuf) {
   using P = typename Tr<R, CPLX>::P;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t full[S];
   __shared__ SweepView views[2];
   __shared__ SweepTile ring[8];
   __shared__ __align__(16) State states[2];
   static_assert(sizeof(State) % 16 == 0, "state size");
   constexpr int E = CPLX ? 2 : 1;
   // layout: S stages | exchange buffer | nbuf table buffers
   unsigned char *base = (unsigned char *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   P *xch = (P *) (base + S * stage_bytes);
   unsigned char *tabs = (unsigned char *) xch + xch_bytes;
   const int g = gridDim.x;
   int acq = -1;  // thread 0: the instance whose tensor maps it last acquired
   // thread 0: the view and tables of tile T into buffer vb; their bytes are
   // expected with the tile's
   auto copy_tabs = [&](const SweepTile &T, int q, int vb) {
      const SweepGeo o = sweep_geo(T.geo);
      bulk_load(&views[vb], &tab[T.inst].sv[AXIS], (uint32_t) sizeof(SweepView), &full[q]);
      bulk_load(tabs + vb * tab_bytes, T.tabs,
                sweep_tab_bytes(o.n, o.skip, (int) sizeof(P), NU ? nu_tab_esz<R, CPLX>() : 0), &full[q]);
      if (NU) bulk_load(&states[vb], T.st, (uint32_t) sizeof(State), &full[q]);
   };
   // thread 0: copies of tile T in stage q; expects view and tables too if `with`
   auto copy_tile = [&](const SweepTile &T, int q, bool load, bool with) {
      const SweepGeo o = sweep_geo(T.geo);
      const BatchDesc &D = tab[T.inst];
      const int TW = o.TW, rows = o.ext, boxn = rows <= 256 ? rows : 256;
      const XyStage lay = xy_stage<R, CPLX, NU>(rows, TW, o.skip);
      P *tile = (P *) (base + q * stage_bytes + lay.psi);
      R *ptile = (R *) (base + q * stage_bytes + lay.phi);
      const CUtensorMap *tm_psi = &D.tm_psi[AXIS];
      if (T.inst != acq) {
         tmap_acquire(tm_psi);
         if (NU) tmap_acquire(&D.tm_phi);
         acq = T.inst;
      }
      if (load) {
         uint32_t tx = (uint32_t) (rows * TW * sizeof(P)) + (NU ? (uint32_t) (rows * TW * sizeof(R)) : 0u);
         const uint32_t tb = sweep_tab_bytes(o.n, o.skip, (int) sizeof(P), NU ? nu_tab_esz<R, CPLX>() : 0);
         if (with) tx += (uint32_t) sizeof(SweepView) + tb + (NU ? (uint32_t) sizeof(State) : 0u);
         mbar_arrive_expect_tx(&full[q], tx);
      }
      for (int a0 = 0; a0 < rows; a0 += boxn) {
         if (load) {
            if (AXIS == 0) tma_load_3d(tile + a0 * TW, tm_psi, E * T.b, T.a, a0, &full[q]);
            else tma_load_3d(tile + a0 * TW, tm_psi, E * T.b, a0, T.a, &full[q]);
            if (NU) tma_load_3d(ptile + a0 * TW, &D.tm_phi, T.b, T.a, a0, &full[q]);
         } else {
            if (AXIS == 0) tma_store_3d(tm_psi, E * T.b, T.a, a0, tile + a0 * TW);
            else tma_store_3d(tm_psi, E * T.b, a0, T.a, tile + a0 * TW);
         }
      }
      if (!load) bulk_commit();
   };
   if (threadIdx.x == 0) {
      for (int q = 0; q < S; q++) mbar_init(&full[q], 1);
      fence_mbar_init();
      if ((int) blockIdx.x < ntiles) ring[0] = tiles[blockIdx.x];
      for (int k = 1; k < 3; k++)
         if ((int) blockIdx.x + k * g < ntiles) ring[k] = tiles[blockIdx.x + k * g];
      if ((int) blockIdx.x < ntiles) {
         copy_tile(ring[0], 0, true, true);
         copy_tabs(ring[0], 0, 0);
      }
   }
   __syncthreads();
   int vb = 0, it = 0;
   for (int t = blockIdx.x; t < ntiles; t += g, it++) {
      const int q = it % S;
      const SweepTile &T = ring[it & 7], &N = ring[(it + 1) & 7];
      const bool change = t + g < ntiles && N.inst != T.inst;
      const int vn = change && nbuf == 2 ? vb ^ 1 : vb;
      if (threadIdx.x == 0 && t + g < ntiles) {
         wait_stage_free<S>();
         copy_tile(N, (it + 1) % S, true, change);
         if (change && nbuf == 2) copy_tabs(N, (it + 1) % S, vn);
      }
      if (threadIdx.x == blockDim.x - 1) {
         // the record asked for one tile ago is complete before the barrier
         // below; the next one replaces a record no thread reads any more
         cp_async_wait_all();
         if (t + 3 * g < ntiles) {
            unsigned char *to = (unsigned char *) &ring[(it + 3) & 7];
            const unsigned char *from = (const unsigned char *) (tiles + t + 3 * g);
            cp_async16(to, from);
            cp_async16(to + 16, from + 16);
         }
      }
      const bool late = !mbar_wait(&full[q], (it / S) & 1, nullptr);
      if (late) atomicOr(tab[T.inst].err, kErrTmaTimeout);
      if (__syncthreads_or(late)) break;
      const SweepView &sv = views[vb];
      const SweepGeo o = sweep_geo(T.geo);
      const int TW = o.TW, c = threadIdx.x & (TW - 1), p = threadIdx.x / TW;
      const XyStage lay = xy_stage<R, CPLX, NU>(o.ext, TW, o.skip);
      P *col = (P *) (base + q * stage_bytes + lay.psi) + c;
      const SegTab tbs = BatchTabs<R, CPLX>::at(sv.tb, tabs + vb * tab_bytes);
      if constexpr (NU) {
         static_assert(AXIS == 0, "calcnu is fused into the x sweep only");
         seg_sweep_any<R, CPLX, MSEG, false, true, 0>(
             col, TW, p, tbs, xch + c, TW,
             nu_xf<R, CPLX, true>((R *) (base + q * stage_bytes + lay.phi) + c, TW, T.a, T.b, c, sv.d, sv.trap, sv.lin,
                                  BatchTabs<R, CPLX>::xt(sv.tb, tabs + vb * tab_bytes), sv.tb.skip, sv.g, sv.gd, sv.dt,
                                  states[vb].scale));
      } else {
         seg_sweep_any<R, CPLX, MSEG, false, true, 0>(col, TW, p, tbs, xch + c, TW, NoXf());
      }
      fence_proxy_async();
      __syncthreads();
      if (threadIdx.x == 0) {
         copy_tile(T, q, false, false);
         if (change && nbuf == 1) copy_tabs(N, (it + 1) % S, 0);
      }
      vb = vn;
   }
   if (threadIdx.x == 0) bulk_wait_all();
}

template <class R, bool CPLX, int MOM, int MSEG, int S>
__global__ void __launch_bounds__(256, kb_sweep_ctas(sizeof(R) == 4, CPLX, MSEG, false)) kb_sweep_z(
    const BatchDesc *__restrict__ tab, const SweepTile *__restrict__ tiles, int ntiles, uint32_t stage_bytes,
    uint32_t xch_bytes, uint32_t tab_bytes, int nbuf, uint32_t part_bytes) {
   using P = typename Tr<R, CPLX>::P;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t full[S];
   __shared__ SweepView views[2];
   __shared__ SweepTile ring[8];
   // layout: S stages of rows | exchange buffer | Simpson partials (2 arrays) | nbuf table buffers
   unsigned char *base = (unsigned char *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   P *xch = (P *) (base + S * stage_bytes);
   double *part = (double *) ((unsigned char *) xch + xch_bytes);
   double *part2 = (double *) ((unsigned char *) part + part_bytes);
   unsigned char *tabs = (unsigned char *) part2 + part_bytes;
   const int g = gridDim.x;
   // one bulk copy per row, issued by the 32 lanes of warp 0 (the short rows
   // of small grids make many small copies); every lane commits and waits
   // for its own store groups
   const int lane = threadIdx.x & 31;
   auto copy_tabs = [&](const SweepTile &T, int q, int vb) {
      if (lane != 0) return;
      const SweepGeo o = sweep_geo(T.geo);
      bulk_load(&views[vb], &tab[T.inst].sv[2], (uint32_t) sizeof(SweepView), &full[q]);
      bulk_load(tabs + vb * tab_bytes, T.tabs, sweep_tab_bytes(o.n, o.skip, (int) sizeof(P), 0), &full[q]);
   };
   auto copy_tile = [&](const SweepTile &T, int q, bool load, bool with) {
      const SweepGeo o = sweep_geo(T.geo);
      const int nz = o.n, nr = T.b;
      const uint32_t row_bytes = (uint32_t) (nz * sizeof(P));
      P *tile = (P *) (base + q * stage_bytes) + zrow_pad(o.skip, (int) sizeof(P));
      if (load && lane == 0) {
         const uint32_t more = with ? (uint32_t) sizeof(SweepView) + sweep_tab_bytes(nz, o.skip, (int) sizeof(P), 0) : 0u;
         mbar_arrive_expect_tx(&full[q], row_bytes * nr + more);
      }
      __syncwarp();
      for (int rr = lane; rr < nr; rr += 32) {
         P *gp = (P *) T.psi + (long long) rr * nz;
         if (load) bulk_load(tile + rr * o.ext, gp, row_bytes, &full[q]);
         else bulk_store(gp, tile + rr * o.ext, row_bytes);
      }
      if (!load) bulk_commit();
   };
   if (threadIdx.x == 0) {
      for (int q = 0; q < S; q++) mbar_init(&full[q], 1);
      fence_mbar_init();
      if ((int) blockIdx.x < ntiles) ring[0] = tiles[blockIdx.x];
      for (int k = 1; k < 3; k++)
         if ((int) blockIdx.x + k * g < ntiles) ring[k] = tiles[blockIdx.x + k * g];
   }
   __syncthreads();
   if (threadIdx.x < 32 && (int) blockIdx.x < ntiles) {
      copy_tile(ring[0], 0, true, true);
      copy_tabs(ring[0], 0, 0);
   }
   int vb = 0, it = 0;
   for (int t = blockIdx.x; t < ntiles; t += g, it++) {
      const int q = it % S;
      const SweepTile &T = ring[it & 7], &N = ring[(it + 1) & 7];
      const bool change = t + g < ntiles && N.inst != T.inst;
      const int vn = change && nbuf == 2 ? vb ^ 1 : vb;
      if (threadIdx.x < 32 && t + g < ntiles) {
         wait_stage_free<S>();
         copy_tile(N, (it + 1) % S, true, change);
         if (change && nbuf == 2) copy_tabs(N, (it + 1) % S, vn);
      }
      if (threadIdx.x == blockDim.x - 1) {
         // the record asked for one tile ago is complete before the barrier
         // below; the next one replaces a record no thread reads any more
         cp_async_wait_all();
         if (t + 3 * g < ntiles) {
            unsigned char *to = (unsigned char *) &ring[(it + 3) & 7];
            const unsigned char *from = (const unsigned char *) (tiles + t + 3 * g);
            cp_async16(to, from);
            cp_async16(to + 16, from + 16);
         }
      }
      const bool late = !mbar_wait(&full[q], (it / S) & 1, nullptr);
      if (late) atomicOr(tab[T.inst].err, kErrTmaTimeout);
      if (__syncthreads_or(late)) break;
      const SweepView &sv = views[vb];
      const SweepGeo o = sweep_geo(T.geo);
      const int TR = o.TW, c = threadIdx.x % TR, p = threadIdx.x / TR;
      P *rows = (P *) (base + q * stage_bytes) + zrow_pad(o.skip, (int) sizeof(P));
      // the row sums run beyond the tile's last barrier: what they need of the
      // view, whose buffer the next copies may replace, is taken before
      const Dims d = sv.d;
      const ZOut zo = sv.zo;
      zsweep_tile<R, CPLX, MOM, MSEG, true, true>(rows, T.b, TR, o.ext, c, p,
                                                  BatchTabs<R, CPLX>::at(sv.tb, tabs + vb * tab_bytes), xch, part, part2,
                                                  d, zo, T.a, T.a / TR);
      if (threadIdx.x < 32) {
         copy_tile(T, q, false, false);
         if (change && nbuf == 1) copy_tabs(N, (it + 1) % S, 0);
      }
      vb = vn;
   }
   if (threadIdx.x < 32) bulk_wait_all();
}

}  // namespace gpe
