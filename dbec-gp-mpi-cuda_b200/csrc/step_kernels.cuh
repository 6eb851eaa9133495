// step_kernels.cuh -- kernels of the split step (dipolar convolution passes,
// fused calcnu + sweeps, norm) and of the observables.
#pragma once

#include "fftn.cuh"
#include "kernels.cuh"
#include "tma.cuh"

namespace gpe {

// ===========================================================================
// Dipolar convolution phi = IFFT[Udd * FFT[|psi|^2]] (calcpsidd2_mem,
// imag3d-mpicuda.cu:1460-1510) as four FFT passes over the half spectrum
// spec[x][y][kz], kz in [0, nz/2], plus the boundary planes.
//
// z passes: each real row of length nz is transformed as a complex line of
// length h = nz/2 (z[m] = x[2m] + i x[2m+1]) and split/merged with
//   X[k] = E + W^k O,  E = (Z_k + conj Z_{h-k})/2,  O = (Z_k - conj Z_{h-k})/(2i)
// (forward) and Z_k = (X_k + conj X_{h-k}) + i (X_k - conj X_{h-k}) W^-k
// (inverse), W = exp(-2 pi i / nz).  Rows arrive and leave by bulk copies.
// y and x passes: a TMA box of L kz columns by the whole line lands in the
// interleaved layout the FFT engine works in.
// ===========================================================================

// Points per thread of the y and x passes, whose tile width (kz columns) the host
// picks so that a tile of a whole line holds at most 256 PPT points (32 KB).
template <class R> struct FftL {
   static constexpr int PPT = sizeof(R) == 8 ? 8 : 16;
};

// Preferred rows per CTA of the forward z pass: 16 over complex FP32 rows, so
// that the radix-8 stages (nz/2-point lines) keep all 256 threads busy; 8 over
// complex FP64 rows (4 KB each), which measured faster with four CTAs per SM; 8
// over real rows on a CTA sized to them (128 threads at nz = 256; 512x512x256
// FP32 280 -> 238 us, 256^3 FP64 93 -> 87 us), where the host keeps 16 rows on
// 256 threads for FP64 rows shorter than 128 points.  The inverse pass takes 8
// rows on a CTA sized to them, six per SM (256^3 FP64 82 -> 78 us, 512x512x256
// FP32 238 -> 210 us).  The host halves the rows while the tile does not fit
// shared memory.
template <class R, bool CPLX> constexpr int zfwd_rows() { return sizeof(R) == 4 && CPLX ? 16 : 8; }

// Tables of roots: a y line has n stage roots (padded to n entries), an x line
// n forward and n inverse ones (one set where the plan reads the same both
// ways), a z line of half length h its stage roots, padded to even, and then
// W^k, k <= h, padded to even.
__host__ __device__ constexpr int ztab_roots(int h) { return (h + 1) & ~1; }
__host__ __device__ constexpr int ztab_len(int h) { return ztab_roots(h) + ((h + 2) & ~1); }
__host__ __device__ __forceinline__ int conv_roots(const FftPlan &px) {
   for (int q = 0; q < px.nst / 2; q++)
      if (px.rad[q] != px.rad[px.nst - 1 - q]) return 2 * px.n;
   return px.n;
}

// Udd's columns of an x tile: nb boxes of rows |kx| rows (at most the 256 a TMA
// box may have) by L columns, FP64; of several boxes each is a multiple of 8
// rows, so that the next one lands on a 128-byte boundary.
struct UddBox {
   int nb, rows;
   uint32_t bytes;  // shared memory of one tile's columns, a multiple of 128
};
__host__ __device__ __forceinline__ constexpr UddBox udd_box(int nx, int L) {
   const int nxh = nx / 2 + 1, nb = (nxh + 255) / 256;
   const int rows = nb == 1 ? nxh : ((nxh + nb - 1) / nb + 7) & ~7;
   return UddBox{nb, rows, (uint32_t) ((nb * rows * L * 8 + 127) & ~127)};
}
// Bytes of a tile of `rows` by L columns of complex R, a multiple of 128.
template <class R> __host__ __device__ __forceinline__ constexpr uint32_t fft_tile_bytes(int rows, int L) {
   return (uint32_t) ((rows * L * 2 * (int) sizeof(R) + 127) & ~127);
}

// |psi|^2 of L rows (row stride LS elements) packed as complex lines of
// length h = nz/2 in the interleaved layout: buf[m L + l] = (rho[2m], rho[2m+1]).
template <class R, bool CPLX, int L>
__device__ __forceinline__ void zfwd_pack(const typename Tr<R, CPLX>::P *rows, int LS, cpx<R> *buf, int h) {
   for (int e = threadIdx.x; e < h * L; e += blockDim.x) {
      const int l = e % L, m = e / L;
      const typename Tr<R, CPLX>::P *rw = rows + l * LS + 2 * m;
      buf[e] = mk<R>(dens_rn(rw[0]), dens_rn(rw[1]));
   }
}

// Real-FFT split of the transformed lines Z (interleaved) into half-spectrum
// rows out[l pitch + k], k <= h, and zero padding up to nzp.  X[k] and X[h-k]
// come from the same pair of inputs: X[k] = E + W^k O, X[h-k] = conj(E - W^k O).
template <class R, int L>
__device__ __forceinline__ void zfwd_split(const cpx<R> *Z, const cpx<R> *W, int h, int nzp, cpx<R> *out,
                                           int nt) {
   using C = cpx<R>;
   for (int e = threadIdx.x; e < (h / 2 + 1) * L; e += nt) {
      const int l = e % L, k = e / L;
      const C a = Z[k * L + l];
      const C b = cconj(Z[(k == 0 ? 0 : h - k) * L + l]);
      const C E = cscale(cadd(a, b), (R) 0.5);
      const C t = csub(a, b);
      const C O = cmul(W[k], mk<R>(t.y * (R) 0.5, -t.x * (R) 0.5));
      C *o = out + l * nzp;
      o[k] = cadd(E, O);
      if (2 * k != h) o[h - k] = cconj(csub(E, O));
   }
   if (nzp > h + 1)
      for (int l = threadIdx.x; l < L; l += nt) out[l * nzp + h + 1] = mk<R>(0, 0);
}

// The same for a compile-time length, in place: every thread takes its pairs
// into registers before any output row (which overlaps the lines) is written.
template <class R, int L, int H, int NT>
__device__ __forceinline__ void zfwd_split_n(const cpx<R> *Z, const cpx<R> *W, int nzp, cpx<R> *out) {
   using C = cpx<R>;
   constexpr int NE = (H / 2 + 1) * L, U = (NE + NT - 1) / NT;
   C lo[U], hi[U];
#pragma unroll
   for (int u = 0; u < U; u++) {
      const int e = threadIdx.x + u * NT;
      if ((int) threadIdx.x < NT && e < NE) {
         const int l = e % L, k = e / L;
         const C a = Z[k * L + l];
         const C b = cconj(Z[(k == 0 ? 0 : H - k) * L + l]);
         const C E = cscale(cadd(a, b), (R) 0.5);
         const C t = csub(a, b);
         const C O = cmul(W[k], mk<R>(t.y * (R) 0.5, -t.x * (R) 0.5));
         lo[u] = cadd(E, O);
         hi[u] = cconj(csub(E, O));
      }
   }
   __syncthreads();
#pragma unroll
   for (int u = 0; u < U; u++) {
      const int e = threadIdx.x + u * NT;
      if ((int) threadIdx.x < NT && e < NE) {
         const int l = e % L, k = e / L;
         C *o = out + l * nzp;
         o[k] = lo[u];
         if (2 * k != H) o[H - k] = hi[u];
      }
   }
   if (nzp > H + 1)
      for (int l = threadIdx.x; l < L; l += NT) out[l * nzp + H + 1] = mk<R>(0, 0);
}

// Real-FFT merge: Z_k of the inverse transform from X_k and X_{h-k} (row of
// nzp half-spectrum points); the DC and Nyquist bins are real.
template <class R>
__device__ __forceinline__ cpx<R> zinv_merge(const cpx<R> *row, const cpx<R> *W, int h, int k) {
   using C = cpx<R>;
   C a = row[k], b = row[h - k];
   if (k == 0) { a.y = 0; b.y = 0; }
   b = cconj(b);
   const C E = cadd(a, b);
   const C O = cmul(csub(a, b), cconj(W[k]));
   return mk<R>(E.x - O.y, E.y + O.x);
}

// kz columns of the y and x tiles these are compiled for, rows of the z tiles
// and the longest half-length z line.
__host__ __device__ constexpr int len_cols(bool fp32) { return fp32 ? 8 : 4; }
template <class R> struct LenCols { static constexpr int L = len_cols(sizeof(R) == 4); };
constexpr int kLenRows = 8, kLenMaxH = 256;
// Threads of a CTA that transforms L lines of N points, and the resident CTAs
// its kernels are compiled for: 64 registers per FP32 thread, 128 per FP64 one.
template <class R> __host__ __device__ constexpr int len_threads(int N, int L) {
   const int t = (N * L / kLenPpt + 31) / 32 * 32;
   return t < 32 ? 32 : t;
}
template <class R> __host__ __device__ constexpr int len_ctas(int N, int L) {
   const int c = (sizeof(R) == 8 ? 512 : 1024) / len_threads<R>(N, L);
   return c < 1 ? 1 : c;
}

// Pass 1: |psi|^2 rows -> half spectrum rows (L rows per CTA).
// Register budget: four CTAs per SM for 8-row tiles, three for 16-row tiles
// (whose shared tiles allow no more; measured faster with the larger budget).
// The pass over the tile of L rows starting at row r0 (shared by the single
// solve's kernel and the batched one).
template <class R, bool CPLX, int PPT, int L>
__device__ __forceinline__ void zfwd_body(const typename Tr<R, CPLX>::P *__restrict__ psi, cpx<R> *__restrict__ spec,
                                          const Dims &d, const FftPlan &ph, const cpx<R> *__restrict__ twz, int LSr,
                                          uint32_t *err, long long r0) {
   using C = cpx<R>;
   using P = typename Tr<R, CPLX>::P;

   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t bar;
   const int nz = d.nz, h = nz / 2, nzp = d.nzp;
   // layout: rows [L][LSr] (later the output rows [L][nzp]) | FFT buffer | twiddles
   P *rows = (P *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   C *buf = (C *) (rows + L * LSr);
   C *tw = buf + h * L;
   const int nr = (int) ((d.nxy - r0) < L ? (d.nxy - r0) : L);
   const uint32_t row_bytes = (uint32_t) (nz * sizeof(P));
   // the roots do not depend on the previous kernel: their copies start
   // before it has finished
   if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
      mbar_arrive_expect_tx(&bar, row_bytes * nr + (uint32_t) (ztab_len(h) * sizeof(C)));
      bulk_load(tw, twz, (uint32_t) (ztab_len(h) * sizeof(C)), &bar);
   }
   pdl_wait();
   if (threadIdx.x == 0) {
      for (int r = 0; r < nr; r++) bulk_load(rows + r * LSr, psi + (r0 + r) * nz, row_bytes, &bar);
   }
   __syncthreads();
   for (int e = threadIdx.x; e < (L - nr) * LSr; e += blockDim.x) rows[nr * LSr + e] = zero_of<P>();
   if (__syncthreads_or(!mbar_wait(&bar, 0, err))) return;
   zfwd_pack<R, CPLX, L>(rows, LSr, buf, h);
   __syncthreads();
   fft_lines_ip<L, C, false, PPT>(buf, ph, tw);
   C *out = (C *) rows;  // [L][nzp]; the rows are no longer read
   zfwd_split<R, L>(buf, tw + ztab_roots(h), h, nzp, out, blockDim.x);
   fence_proxy_async();
   __syncthreads();
   if (threadIdx.x == 0) {
      bulk_store(spec + r0 * nzp, out, (uint32_t) (nr * nzp * sizeof(C)));
      bulk_commit();
      bulk_wait_all();
   }
}

template <class R, bool CPLX, int PPT, int L>
__global__ void __launch_bounds__(256, L >= 16 ? 3 : 4) k_zfwd(const typename Tr<R, CPLX>::P *__restrict__ psi,
                                              cpx<R> *__restrict__ spec, Dims d, FftPlan ph,
                                              const cpx<R> *__restrict__ twz, int LSr, uint32_t *err) {
   pdl_trigger();
   zfwd_body<R, CPLX, PPT, L>(psi, spec, d, ph, twz, LSr, err, (long long) blockIdx.x * L);
}

// Passes 2 and 4: FFT along y of L kz columns of one x plane.  The host sizes
// the CTA at one thread per PPT points of the tile (128 threads for the
// 4-column FP64 tiles, so that eight fit on an SM); the register budget
// (launch bounds 256 x 4) allows any of these sizes.
template <class R, bool INV, int L, int PPT = FftL<R>::PPT>
__device__ __forceinline__ void yfft_body(const CUtensorMap *tm, const Dims &d, const FftPlan &py,
                                          const cpx<R> *__restrict__ twy, int boxn, int nbox, uint32_t *err, int x,
                                          int k0) {
   using C = cpx<R>;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t bar;
   const int ny = d.ny, rows = boxn * nbox;
   C *buf = (C *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   C *tw = buf + rows * L;
   // the roots do not depend on the previous kernel: their copies start
   // before it has finished
   if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
      mbar_arrive_expect_tx(&bar, (uint32_t) (rows * L * sizeof(C) + ny * sizeof(C)));
      bulk_load(tw, twy, (uint32_t) (ny * sizeof(C)), &bar);
   }
   pdl_wait();
   if (threadIdx.x == 0) {
      for (int b = 0; b < nbox; b++) tma_load_3d(buf + b * boxn * L, tm, 2 * k0, b * boxn, x, &bar);
   }
   __syncthreads();
   if (__syncthreads_or(!mbar_wait(&bar, 0, err))) return;
   fft_lines_ip<L, C, INV, PPT>(buf, py, tw);
   fence_proxy_async();
   __syncthreads();
   if (threadIdx.x == 0) {
      for (int b = 0; b < nbox; b++) tma_store_3d(tm, 2 * k0, b * boxn, x, buf + b * boxn * L);
      bulk_commit();
      bulk_wait_all();
   }
}

template <class R, bool INV, int L>
__global__ void __launch_bounds__(256, 4) k_yfft(const __grid_constant__ CUtensorMap tm, Dims d, FftPlan py,
                                                 const cpx<R> *__restrict__ twy, int boxn, int nbox, uint32_t *err) {
   pdl_trigger();
   const int nkb = (d.nzh + L - 1) / L;
   const int x = blockIdx.x / nkb, k0 = (blockIdx.x - x * nkb) * L;
   yfft_body<R, INV, L>(&tm, d, py, twy, boxn, nbox, err, x, k0);
}

// Udd's columns of an x tile by asynchronous 8-byte copies of every thread
// (batched passes: a second tensor map in global memory costs each CTA an
// acquire, x pass of 64 grids 167 us this way and 203 us by TMA; one solve, its
// map a kernel parameter, gained by TMA, 78 -> 68 us at 256^3 FP64).
__device__ __forceinline__ void udd_copy(double *ud, const double *udd, const Dims &d, int nx, int L, int ay, int k0) {
   const int nyh = d.ny / 2 + 1, nzu = (d.nzh + 1) & ~1;
   for (int e = threadIdx.x; e < (nx / 2 + 1) * L; e += blockDim.x) {
      const int ax = e / L, k = k0 + e % L;
      cp_async8(ud + e, udd + ((long long) ax * nyh + ay) * nzu + (k < d.nzh ? k : d.nzh - 1));
   }
}

// Pass 3: FFT along x, multiply by Udd(k) * scale^2, inverse FFT along x, for
// L kz columns of one y plane.  Udd octant layout [|kx|][|ky|][kz].  CTA size
// as for the y passes.
template <class R, int L, int PPT = FftL<R>::PPT>
__device__ __forceinline__ void xconv_body(const CUtensorMap *tm, const CUtensorMap *tm_udd, const double *udd, const Dims &d,
                                           const FftPlan &px, const FftPlan &pxi, const cpx<R> *__restrict__ twx,
                                           const State *__restrict__ st, int boxn, int nbox, uint32_t *err, int y,
                                           int k0) {
   using C = cpx<R>;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t bar;
   const int nx = d.nx, ny = d.ny, rows = boxn * nbox;
   const UddBox ub = udd_box(nx, L);
   C *buf = (C *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   double *ud = (double *) ((unsigned char *) buf + fft_tile_bytes<R>(rows, L));  // [|kx|][L]
   C *tw = (C *) ((unsigned char *) ud + ub.bytes);
   const int ntw = conv_roots(px);  // stage roots, forward then inverse
   const int ay = (y <= ny / 2) ? y : ny - y;
   // the roots and Udd do not depend on the previous kernel: their copies start
   // before it has finished
   if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
      mbar_arrive_expect_tx(&bar, (uint32_t) ((rows * L + ntw) * sizeof(C)) + (tm_udd ? (uint32_t) (ub.nb * ub.rows * L * 8) : 0u));
      bulk_load(tw, twx, (uint32_t) (ntw * sizeof(C)), &bar);
      if (tm_udd)
         for (int b = 0; b < ub.nb; b++) tma_load_3d(ud + b * ub.rows * L, tm_udd, k0, ay, b * ub.rows, &bar);
   }
   if (!tm_udd) udd_copy(ud, udd, d, nx, L, ay, k0);
   pdl_wait();
   if (threadIdx.x == 0) {
      for (int b = 0; b < nbox; b++) tma_load_3d(buf + b * boxn * L, tm, 2 * k0, y, b * boxn, &bar);
   }
   __syncthreads();
   if (!tm_udd) cp_async_wait_all();
   if (__syncthreads_or(!mbar_wait(&bar, 0, err))) return;
   fft_lines_ip<L, C, false, PPT>(buf, px, tw);
   C *res = buf;
   const double s2 = st->scale2;
   for (int e = threadIdx.x; e < nx * L; e += blockDim.x) {
      const int xx = e / L, c = e - xx * L;
      const int ax = (xx <= nx / 2) ? xx : nx - xx;
      const R u = (R) (ud[ax * L + c] * s2);
      res[e] = scale_rn(res[e], u);
   }
   __syncthreads();
   fft_lines_ip<L, C, true, PPT, true>(buf, pxi, ntw > nx ? tw + nx : tw);
   fence_proxy_async();
   __syncthreads();
   if (threadIdx.x == 0) {
      for (int b = 0; b < nbox; b++) tma_store_3d(tm, 2 * k0, y, b * boxn, buf + b * boxn * L);
      bulk_commit();
      bulk_wait_all();
   }
}

template <class R, int L>
__global__ void __launch_bounds__(256, 4) k_xconv(const __grid_constant__ CUtensorMap tm,
                                                  const __grid_constant__ CUtensorMap tm_udd, Dims d, FftPlan px, FftPlan pxi,
                                                  const cpx<R> *__restrict__ twx,
                                                  const State *__restrict__ st, int boxn, int nbox, uint32_t *err) {
   pdl_trigger();
   const int nkb = (d.nzh + L - 1) / L;
   const int y = blockIdx.x / nkb, k0 = (blockIdx.x - y * nkb) * L;
   xconv_body<R, L>(&tm, &tm_udd, nullptr, d, px, pxi, twx, st, boxn, nbox, err, y, k0);
}

// Ends the inverse z pass: stores the phi rows out[l LSo + k], l < nr, with
// the boundary planes (calcpsidd2_kernel2a/2b with last = 1,
// imag3d-mpicuda.cu:1591-1625): z = nz-1 <- z = 0, x = nx-1 <- x = 0 and
// y = ny-1 <- y = 0, each excluding the other two last indices.  z is fixed
// inside the row.  With FOLD the first nz-1 points of a row (0, y) or (x, 0)
// go to the matching boundary row too and that row's own CTA stores only its
// last point; without, a pass of its own copies the planes (k_phifix).  One
// thread per row; a copied row's points beyond the last 16-byte multiple of
// nz-1 are stored one by one.  Folding the planes saves a launch of 6 us per
// step.
template <class R, bool FOLD>
__device__ __forceinline__ void zinv_finish(R *__restrict__ phi, R *out, int LSo, const Dims &d, long long r0, int nr) {
   const int nz = d.nz;
   long long x = 0, y = 0;
   if (threadIdx.x < nr) {
      const long long row = r0 + threadIdx.x;
      x = row / d.ny, y = row - x * d.ny;
      if (x < d.nx - 1 && y < d.ny - 1) out[threadIdx.x * LSo + nz - 1] = out[threadIdx.x * LSo];
   }
   fence_proxy_async();
   __syncthreads();
   if (threadIdx.x < nr) {
      const R *o = out + threadIdx.x * LSo;
      R *own = phi + (r0 + threadIdx.x) * nz;
      const bool bx = x == d.nx - 1 && y < d.ny - 1, by = y == d.ny - 1 && x < d.nx - 1;
      if (FOLD && (bx || by)) {
         own[nz - 1] = o[nz - 1];
      } else {
         bulk_store(own, o, (uint32_t) (nz * sizeof(R)));
      }
      if (FOLD) {
         constexpr int V = 16 / (int) sizeof(R);
         const int nb = (nz - 1) / V * V;  // nz is a multiple of V
         for (int q = 0; q < 2; q++) {
            if (q == 0 ? !(x == 0 && y < d.ny - 1) : !(y == 0 && x < d.nx - 1)) continue;
            R *to = phi + (q == 0 ? (long long) (d.nx - 1) * d.ny + y : x * d.ny + d.ny - 1) * nz;
            if (nb > 0) bulk_store(to, o, (uint32_t) (nb * sizeof(R)));
            for (int k = nb; k < nz - 1; k++) to[k] = o[k];
         }
      }
      bulk_commit();
      bulk_wait_all();
   }
}

// Pass 5: half spectrum rows -> phi rows (unnormalised inverse, Hermitian).
template <class R, int PPT, int L, bool FOLD>
__device__ __forceinline__ void zinv_body(const cpx<R> *__restrict__ spec, R *__restrict__ phi, const Dims &d,
                                          const FftPlan &ph, const cpx<R> *__restrict__ twz, int LSo, uint32_t *err,
                                          long long r0) {
   using C = cpx<R>;

   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t bar;
   const int nz = d.nz, h = nz / 2, nzp = d.nzp;
   // layout: input rows [L][nzp] (later the phi rows [L][LSo]) | FFT buffer | twiddles
   C *in = (C *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   const int in_elems = ((L * nzp) > (L * LSo + 1) / 2 ? (L * nzp) : (L * LSo + 1) / 2);
   C *buf = in + ((in_elems + 7) & ~7);
   C *tw = buf + h * L;
   const int nr = (int) ((d.nxy - r0) < L ? (d.nxy - r0) : L);
   // the roots do not depend on the previous kernel: their copies start
   // before it has finished
   if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
      mbar_arrive_expect_tx(&bar, (uint32_t) ((nr * nzp + ztab_len(h)) * sizeof(C)));
      bulk_load(tw, twz, (uint32_t) (ztab_len(h) * sizeof(C)), &bar);
   }
   pdl_wait();
   if (threadIdx.x == 0) {
      bulk_load(in, spec + r0 * nzp, (uint32_t) (nr * nzp * sizeof(C)), &bar);
   }
   __syncthreads();
   for (int e = threadIdx.x; e < (L - nr) * nzp; e += blockDim.x) in[nr * nzp + e] = mk<R>(0, 0);
   if (__syncthreads_or(!mbar_wait(&bar, 0, err))) return;
   for (int e = threadIdx.x; e < h * L; e += blockDim.x) {
      const int l = e % L, k = e / L;
      buf[e] = zinv_merge<R>(in + l * nzp, tw + ztab_roots(h), h, k);
   }
   __syncthreads();
   fft_lines_ip<L, C, true, PPT>(buf, ph, tw);
   const C *z = buf;
   R *out = (R *) in;  // [L][LSo]
   for (int e = threadIdx.x; e < h * L; e += blockDim.x) {
      const int l = e % L, m = e / L;
      const C v = z[e];
      out[l * LSo + 2 * m] = v.x;
      out[l * LSo + 2 * m + 1] = v.y;
   }
   __syncthreads();
   zinv_finish<R, FOLD>(phi, out, LSo, d, r0, nr);
}

template <class R, int PPT, int L>
__global__ void __launch_bounds__(256, L >= 16 ? 3 : 4) k_zinv(const cpx<R> *__restrict__ spec, R *__restrict__ phi, Dims d,
                                                 FftPlan ph, const cpx<R> *__restrict__ twz, int LSo, uint32_t *err) {
   pdl_trigger();
   zinv_body<R, PPT, L, true>(spec, phi, d, ph, twz, LSo, err, (long long) blockIdx.x * L);
}

// ---------------------------------------------------------------------------
// The passes on lines of a compile-time length (fftn.cuh): one CTA of
// len_threads(N, L) threads per tile (the batched kernels may launch more),
// the roots from the stage-ordered tables (make_roots in solver.cu).  The z
// passes take the first stage's points straight from the staged rows (|psi|^2
// or the merged half spectrum) and the inverse one ends in the phi rows.  With
// run-time lengths these passes were bound by issue, most of it index
// arithmetic (z inverse 180 instructions a complex point, now 56); they are now
// bound by the series load, stages, store of the five to eight CTAs that fit an
// SM.  256^3 on B200, run-time lengths -> these: at each kernel, with the time
// of its bytes at 6.65 TB/s.

// Bytes of the shared region of a z pass (psi or half-spectrum rows, lines,
// output rows).
template <class R, bool CPLX> __host__ __device__ constexpr int zfwd_region(int H, int L) {
   constexpr int sp = (int) sizeof(R) * (CPLX ? 2 : 1), sc = 2 * (int) sizeof(R);
   const int rows = L * (2 * H + 16 / sp) * sp, lines = L * (sizeof(R) == 4 ? (H + 2) & ~1 : H + 1) * sc;
   return ((rows > lines ? rows : lines) + 127) & ~127;
}
template <class R> __host__ __device__ constexpr int zinv_region(int H, int L) {
   constexpr int sc = 2 * (int) sizeof(R);
   const int rows = L * (2 * H + 16 / (int) sizeof(R)) * (int) sizeof(R),
             lines = L * (sizeof(R) == 4 ? (H + 2) & ~1 : H + 1) * sc;
   return ((rows > lines ? rows : lines) + 127) & ~127;
}

// z forward: H = nz / 2; twz: H stage roots, then W^k, k <= H.  us: FP64 complex
// 103 -> 73 (bytes 61), real 89 -> 57 (40), FP32 real 56 -> 29 (20).
template <class R, bool CPLX, int L, int H>
__device__ __forceinline__ void zfwd_body_n(const typename Tr<R, CPLX>::P *__restrict__ psi, cpx<R> *__restrict__ spec,
                                            const Dims &d, const cpx<R> *__restrict__ twz, uint32_t *err,
                                            long long r0) {
   using C = cpx<R>;
   using P = typename Tr<R, CPLX>::P;
   constexpr int NT = len_threads<R>(H, L), nz = 2 * H;
   constexpr int U16 = 16 / (int) sizeof(P), LSr = (nz / U16 | 1) * U16;  // an odd number of 16-byte units
   constexpr int nzp = sizeof(R) == 4 ? (H + 2) & ~1 : H + 1;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t bar;
   // one region for the psi rows, the lines being transformed and the output
   // rows in turn (each is read into registers before the next is written):
   // 37 instead of 53 KB at nz = 256 complex FP64, six CTAs per SM for four
   P *rows = (P *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   C *buf = (C *) rows;
   C *tw = (C *) ((unsigned char *) rows + zfwd_region<R, CPLX>(H, L));
   const int nr = (int) ((d.nxy - r0) < L ? (d.nxy - r0) : L);
   constexpr uint32_t row_bytes = (uint32_t) (nz * sizeof(P)), tw_bytes = (uint32_t) (ztab_len(H) * sizeof(C));
   // the roots do not depend on the previous kernel: their copies start
   // before it has finished
   if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
      mbar_arrive_expect_tx(&bar, row_bytes * nr + tw_bytes);
      bulk_load(tw, twz, tw_bytes, &bar);
   }
   pdl_wait();
   if (threadIdx.x == 0) {
      for (int r = 0; r < nr; r++) bulk_load(rows + r * LSr, psi + (r0 + r) * nz, row_bytes, &bar);
   }
   __syncthreads();
   for (int e = threadIdx.x; e < (L - nr) * LSr; e += blockDim.x) rows[nr * LSr + e] = zero_of<P>();
   if (__syncthreads_or(!mbar_wait(&bar, 0, err))) return;
   fft_lines<H, L, NT, C, false>(
       buf, tw,
       [&](int l, int m) {
          P a, b;
          ld2(rows + l * LSr + 2 * m, a, b);
          return mk<R>(dens_rn(a), dens_rn(b));
       },
       [&](int l, int i, C v) { buf[i * L + l] = v; });
   __syncthreads();
   C *out = buf;  // [L][nzp]
   zfwd_split_n<R, L, H, NT>(buf, tw + ztab_roots(H), nzp, out);
   fence_proxy_async();
   __syncthreads();
   if (threadIdx.x == 0) {
      bulk_store(spec + r0 * nzp, out, (uint32_t) (nr * nzp * sizeof(C)));
      bulk_commit();
      bulk_wait_all();
   }
}

template <class R, bool CPLX, int L, int H>
__global__ void __launch_bounds__(len_threads<R>(H, L), len_ctas<R>(H, L))
k_zfwd_n(const typename Tr<R, CPLX>::P *__restrict__ psi, cpx<R> *__restrict__ spec, Dims d,
         const cpx<R> *__restrict__ twz, uint32_t *err) {
   pdl_trigger();
   zfwd_body_n<R, CPLX, L, H>(psi, spec, d, twz, err, (long long) blockIdx.x * L);
}

// z inverse; twz as above.  us, with the boundary planes: FP64 78 + 7 -> 53
// (bytes 41), FP32 49 + 7 -> 28 (20).
template <class R, int L, int H, bool FOLD>
__device__ __forceinline__ void zinv_body_n(const cpx<R> *__restrict__ spec, R *__restrict__ phi, const Dims &d,
                                            const cpx<R> *__restrict__ twz, uint32_t *err, long long r0) {
   using C = cpx<R>;
   constexpr int NT = len_threads<R>(H, L), nz = 2 * H;
   constexpr int U16 = 16 / (int) sizeof(R), LSo = (nz / U16 | 1) * U16;  // an odd number of 16-byte units
   constexpr int nzp = sizeof(R) == 4 ? (H + 2) & ~1 : H + 1;
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t bar;
   // one region for the half-spectrum rows, the lines and the phi rows in turn
   C *in = (C *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   C *buf = in;
   C *tw = (C *) ((unsigned char *) in + zinv_region<R>(H, L));
   const int nr = (int) ((d.nxy - r0) < L ? (d.nxy - r0) : L);
   constexpr uint32_t tw_bytes = (uint32_t) (ztab_len(H) * sizeof(C));
   // the roots do not depend on the previous kernel: their copies start
   // before it has finished
   if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
      mbar_arrive_expect_tx(&bar, (uint32_t) (nr * nzp * sizeof(C)) + tw_bytes);
      bulk_load(tw, twz, tw_bytes, &bar);
   }
   pdl_wait();
   if (threadIdx.x == 0) {
      bulk_load(in, spec + r0 * nzp, (uint32_t) (nr * nzp * sizeof(C)), &bar);
   }
   __syncthreads();
   for (int e = threadIdx.x; e < (L - nr) * nzp; e += blockDim.x) in[nr * nzp + e] = mk<R>(0, 0);
   if (__syncthreads_or(!mbar_wait(&bar, 0, err))) return;
   R *out = (R *) in;  // [L][LSo], written by the last stage
   fft_lines<H, L, NT, C, true>(
       buf, tw, [&](int l, int k) { return zinv_merge<R>(in + l * nzp, tw + ztab_roots(H), H, k); },
       [&](int l, int m, C v) { st2(out + l * LSo + 2 * m, v.x, v.y); });
   __syncthreads();
   zinv_finish<R, FOLD>(phi, out, LSo, d, r0, nr);
}

template <class R, int L, int H>
__global__ void __launch_bounds__(len_threads<R>(H, L), len_ctas<R>(H, L))
k_zinv_n(const cpx<R> *__restrict__ spec, R *__restrict__ phi, Dims d, const cpx<R> *__restrict__ twz, uint32_t *err) {
   pdl_trigger();
   zinv_body_n<R, L, H, true>(spec, phi, d, twz, err, (long long) blockIdx.x * L);
}

// y passes, forward and inverse; twy: N stage roots.  us: FP64 57 -> 54 (bytes
// 41), FP32 30 -> 28 (20); they were nearest to their bytes before.
template <class R, bool INV, int L, int N>
__device__ __forceinline__ void yfft_body_n(const CUtensorMap *tm, const cpx<R> *__restrict__ twy, uint32_t *err, int x,
                                            int k0) {
   using C = cpx<R>;
   constexpr int NT = len_threads<R>(N, L), boxn = N <= 256 ? N : N / 2;
   static_assert(N <= 256 || boxn * L * 2 * (int) sizeof(R) % 128 == 0, "TMA boxes start on 128 bytes");
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t bar;
   C *buf = (C *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   C *tw = buf + N * L;
   // the roots do not depend on the previous kernel: their copies start
   // before it has finished
   if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
      mbar_arrive_expect_tx(&bar, (uint32_t) (N * L * sizeof(C) + N * sizeof(C)));
      bulk_load(tw, twy, (uint32_t) (N * sizeof(C)), &bar);
   }
   pdl_wait();
   if (threadIdx.x == 0) {
      for (int b = 0; b < N; b += boxn) tma_load_3d(buf + b * L, tm, 2 * k0, b, x, &bar);
   }
   __syncthreads();
   if (__syncthreads_or(!mbar_wait(&bar, 0, err))) return;
   fft_lines<N, L, NT, C, INV>(
       buf, tw, [&](int l, int i) { return buf[i * L + l]; }, [&](int l, int i, C v) { buf[i * L + l] = v; });
   fence_proxy_async();
   __syncthreads();
   if (threadIdx.x == 0) {
      for (int b = 0; b < N; b += boxn) tma_store_3d(tm, 2 * k0, b, x, buf + b * L);
      bulk_commit();
      bulk_wait_all();
   }
}

template <class R, bool INV, int L, int N>
__global__ void __launch_bounds__(len_threads<R>(N, L), len_ctas<R>(N, L))
k_yfft_n(const __grid_constant__ CUtensorMap tm, Dims d, const cpx<R> *__restrict__ twy, uint32_t *err) {
   pdl_trigger();
   const int nkb = (d.nzh + L - 1) / L;
   const int x = blockIdx.x / nkb, k0 = (blockIdx.x - x * nkb) * L;
   yfft_body_n<R, INV, L, N>(&tm, twy, err, x, k0);
}

// x convolution; twx: N forward and N inverse stage roots.  The multiply by
// Udd happens on the last forward stage's registers.  us: FP64 111 -> 68 (bytes
// 42), FP32 61 -> 37 (21), 512x512x256 FP32 (three stages) 166 (92); 41 % of
// its cycles are FP64 arithmetic.
template <class R, int L, int N>
__device__ __forceinline__ void xconv_body_n(const CUtensorMap *tm, const CUtensorMap *tm_udd, const double *udd, const Dims &d,
                                             const cpx<R> *__restrict__ twx, const State *__restrict__ st,
                                             uint32_t *err, int y, int k0) {
   using C = cpx<R>;
   constexpr int NT = len_threads<R>(N, L), boxn = N <= 256 ? N : N / 2;
   static_assert(N <= 256 || boxn * L * 2 * (int) sizeof(R) % 128 == 0, "TMA boxes start on 128 bytes");
   extern __shared__ __align__(16) unsigned char smem_raw[];
   __shared__ __align__(8) uint64_t bar;
   const int ny = d.ny;
   constexpr UddBox ub = udd_box(N, L);
   C *buf = (C *) (((uintptr_t) smem_raw + 127) & ~(uintptr_t) 127);
   double *ud = (double *) ((unsigned char *) buf + fft_tile_bytes<R>(N, L));  // [|kx|][L]
   C *tw = (C *) ((unsigned char *) ud + ub.bytes);
   constexpr int NTW = palin_plan<R, N>() ? N : 2 * N;  // stage roots
   const int ay = (y <= ny / 2) ? y : ny - y;
   // the roots and Udd do not depend on the previous kernel: their copies start
   // before it has finished
   if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
      mbar_arrive_expect_tx(&bar, (uint32_t) ((N * L + NTW) * sizeof(C)) + (tm_udd ? (uint32_t) (ub.nb * ub.rows * L * 8) : 0u));
      bulk_load(tw, twx, (uint32_t) (NTW * sizeof(C)), &bar);
      if (tm_udd)
         for (int b = 0; b < ub.nb; b++) tma_load_3d(ud + b * ub.rows * L, tm_udd, k0, ay, b * ub.rows, &bar);
   }
   if (!tm_udd) udd_copy(ud, udd, d, N, L, ay, k0);
   pdl_wait();
   if (threadIdx.x == 0) {
      for (int b = 0; b < N; b += boxn) tma_load_3d(buf + b * L, tm, 2 * k0, y, b, &bar);
   }
   __syncthreads();
   const double s2 = st->scale2;
   if (!tm_udd) cp_async_wait_all();
   if (__syncthreads_or(!mbar_wait(&bar, 0, err))) return;
   conv_lines<N, L, NT, C>(buf, tw, palin_plan<R, N>() ? tw : tw + N, [&](int l, int i) {
      const int ax = i <= N / 2 ? i : N - i;
      return (R) (ud[ax * L + l] * s2);
   });
   fence_proxy_async();
   __syncthreads();
   if (threadIdx.x == 0) {
      for (int b = 0; b < N; b += boxn) tma_store_3d(tm, 2 * k0, y, b, buf + b * L);
      bulk_commit();
      bulk_wait_all();
   }
}

template <class R, int L, int N>
__global__ void __launch_bounds__(len_threads<R>(N, L), len_ctas<R>(N, L))
k_xconv_n(const __grid_constant__ CUtensorMap tm, const __grid_constant__ CUtensorMap tm_udd, Dims d,
          const cpx<R> *__restrict__ twx, const State *__restrict__ st, uint32_t *err) {
   pdl_trigger();
   const int nkb = (d.nzh + L - 1) / L;
   const int y = blockIdx.x / nkb, k0 = (blockIdx.x - y * nkb) * L;
   xconv_body_n<R, L, N>(&tm, &tm_udd, nullptr, d, twx, st, err, y, k0);
}

// Boundary planes x = nx-1 and y = ny-1 of phi as a pass of their own (batched
// FP64 steps, whose inverse z pass does not fold them).  The read and write sets are disjoint, so both copies
// run concurrently.  One CTA per copied row: blocks [0, ny-1) the rows (nx-1,
// j) <- (0, j), blocks [ny-1, ny-1 + nx-1) the rows (i, ny-1) <- (i, 0), the
// first nz-1 points of each (the grid has at least one block).
template <class R>
__device__ __forceinline__ void phifix_body(R *__restrict__ phi, const Dims &d, int b) {
   long long dst, src;
   if (b < d.ny - 1) {
      dst = ((long long) (d.nx - 1) * d.ny + b) * d.nz;
      src = (long long) b * d.nz;
   } else if (b - (d.ny - 1) < d.nx - 1) {
      const long long i = b - (d.ny - 1);
      dst = (i * d.ny + d.ny - 1) * d.nz;
      src = i * d.ny * d.nz;
   } else {
      return;
   }
   for (int k = threadIdx.x; k < d.nz - 1; k += blockDim.x) phi[dst + k] = phi[src + k];
}

// Self-test of the bounded waits: one CTA waits on an mbarrier that expects
// 16 bytes of a transaction no copy will ever deliver.  No copy is issued, so
// nothing is in flight when the wait gives up after `spins` polls; the CTA
// then leaves together, exactly as a step kernel whose tile never arrived,
// and the handle's status word reports the timeout.
static __global__ void k_wait_selftest(uint32_t spins, uint32_t *err) {
   __shared__ __align__(8) uint64_t bar;
   if (threadIdx.x == 0) {
      mbar_init(&bar, 1);
      fence_mbar_init();
   }
   __syncthreads();
   if (threadIdx.x == 0) mbar_arrive_expect_tx(&bar, 16u);
   if (__syncthreads_or(!mbar_wait_n(&bar, 0, err, spins))) return;
}

// ===========================================================================
// Sweeps.
// ===========================================================================

// Standalone calcnu (operator-level entry point).
template <class R, bool CPLX>
__global__ void k_calcnu(typename Tr<R, CPLX>::P *__restrict__ psi, const R *__restrict__ phi, Dims d, Trap trap,
                         double g, double gd, double dt) {
   const R invN = (R) (1.0 / (double) d.npts);
   for (long long q = blockIdx.x * (long long) blockDim.x + threadIdx.x; q < d.npts; q += (long long) gridDim.x * blockDim.x) {
      const int k = (int) (q % d.nz);
      const long long r = q / d.nz;
      const int j = (int) (r % d.ny), i = (int) (r / d.ny);
      psi[q] = nu_op<R>(psi[q], phi[q], (R) trap.v(i, j, k), (R) g, (R) gd, (R) dt, invN);
   }
}

// ===========================================================================
// Reductions.
// ===========================================================================

// Per-row Simpson integrals along z of |psi|^2 (rowA) and, with rowB, of z^2
// |psi|^2, by a warp per row with the weights wz, wz2 (in units of h / 3): the
// loads of a warp are consecutive and four rounds of them are in flight.  One
// thread per row left the loads of a warp a row apart (96 us at 256^3 FP64,
// whose 134 MB take 20 us; a whole calcnorm call 97 -> 54 us).
constexpr int kRowWarps = 8;
template <class R, bool CPLX>
__global__ void __launch_bounds__(32 * kRowWarps) k_rows_dens(const typename Tr<R, CPLX>::P *__restrict__ psi, Dims d,
                                                              double hz3, const double *__restrict__ wz,
                                                              const double *__restrict__ wz2,
                                                              double *__restrict__ rowA, double *__restrict__ rowB) {
   const long long row = (long long) blockIdx.x * kRowWarps + threadIdx.x / 32;
   if (row >= d.nxy) return;
   const int lane = threadIdx.x % 32;
   const auto *ps = psi + row * d.nz;
   double a = 0., b = 0.;
#pragma unroll 4
   for (int k = lane; k < d.nz; k += 32) {
      const double f = (double) dens2(ps[k]);
      a = fma(wz[k], f, a);
      if (rowB) b = fma(wz2[k], f, b);
   }
   for (int o = 16; o; o >>= 1) {
      a += __shfl_xor_sync(0xffffffffu, a, o);
      if (rowB) b += __shfl_xor_sync(0xffffffffu, b, o);
   }
   if (lane == 0) {
      rowA[row] = a * hz3;
      if (rowB) rowB[row] = b * hz3;
   }
}

// Sum of n tile partials in an order that depends on n only: 256 strided
// partial sums, a shuffle tree over each 32 of them, then the eight in turn.
// Every thread of the CTA (whole warps) calls it; the result is valid in
// thread 0.  red: 8 doubles.
__device__ __forceinline__ double sum_tiles(const double *__restrict__ part, int n, double *red) {
   constexpr int U = 8;  // loads in flight per lane
   for (int v = threadIdx.x; v < 256; v += blockDim.x) {
      double acc = 0.;
      for (int k0 = v; k0 < n; k0 += 256 * U) {
         double x[U];
#pragma unroll
         for (int u = 0; u < U; u++) x[u] = k0 + 256 * u < n ? __ldcg(part + k0 + 256 * u) : 0.;
#pragma unroll
         for (int u = 0; u < U; u++) acc += x[u];
      }
      for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (v % 32 == 0) red[v / 32] = acc;
   }
   __syncthreads();
   double s = 0.;
   for (int q = 0; q < 8; q++) s += red[q];
   return s;
}

// The step's norm from S = sum w_x w_y S_z |psi|^2 into the state.
__device__ __forceinline__ void set_norm(State *st, double sum, double hx, double hy, double *out_norm) {
   const double nrm = sqrt(sum * (hx / 3.) * (hy / 3.));
   const double t = 1. / nrm;
   st->norm = nrm;
   st->scale = t;
   st->scale2 = t * t;
   if (out_norm) *out_norm = nrm;
}

// norm = sqrt(S_x S_y rowsum) (calcnorm, imag3d-mpicuda.cu:1194-1218), stores
// norm, scale = 1/norm and scale^2 in the state.  Each warp forms the
// weighted Simpson sum over y of one x row (shuffle reduction) into xs[i];
// the last CTA to finish integrates xs over x.  The kernel is latency-bound
// (a few kB of row sums): loads are issued ahead of the sums and the final
// sum uses the whole CTA (16 -> 10 us at 256^3).
constexpr int kNormRowsPerCta = 8;
// CTA `cta` of the `ncta` CTAs that reduce one solve's row sums.
__device__ __forceinline__ void norm_final_body(const double *__restrict__ rowsum, const Dims &d, double hx, double hy,
                                                State *st, double *xs, double *out_norm, int cta, int ncta) {
   const int lane = threadIdx.x & 31;
   const int i = cta * kNormRowsPerCta + (threadIdx.x >> 5);
   if (i < d.nx) {
      // a warp per x row; the loads of a lane are issued before the sums
      const double *r = rowsum + (long long) i * d.ny;
      constexpr int U = 8;
      double acc = 0.;
      for (int j0 = 0; j0 < d.ny; j0 += 32 * U) {
         double v[U];
#pragma unroll
         for (int u = 0; u < U; u++) {
            const int j = j0 + lane + 32 * u;
            v[u] = j < d.ny ? r[j] : 0.;
         }
#pragma unroll
         for (int u = 0; u < U; u++) {
            const int j = j0 + lane + 32 * u;
            if (j < d.ny) acc = fma(simp_w(j, d.ny), v[u], acc);
         }
      }
      for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) xs[i] = acc * hy / 3.;
   }
   __threadfence();
   __syncthreads();
   __shared__ bool last;
   __shared__ double red[32 * kNormRowsPerCta];
   if (threadIdx.x == 0) last = atomicAdd(&st->ticket, 1u) == (unsigned) ncta - 1;
   __syncthreads();
   if (!last) return;
   // last CTA: every thread takes its strided share of the x rows, then a
   // fixed-order tree over the CTA
   __threadfence();
   double acc = 0.;
   for (int k = threadIdx.x; k < d.nx; k += blockDim.x) acc = fma(simp_w(k, d.nx), __ldcg(xs + k), acc);
   red[threadIdx.x] = acc;
   __syncthreads();
   for (int h = blockDim.x / 2; h >= 32; h >>= 1) {
      if ((int) threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
      __syncthreads();
   }
   if (threadIdx.x >= 32) return;
   acc = red[threadIdx.x];
   for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
   if (lane == 0) {
      const double nrm = sqrt(acc * hx / 3.);
      const double t = 1. / nrm;
      st->norm = nrm;
      st->scale = t;
      st->scale2 = t * t;
      st->ticket = 0u;
      if (out_norm) *out_norm = nrm;
   }
}

static __global__ void __launch_bounds__(32 * kNormRowsPerCta) k_norm_final(const double *__restrict__ rowsum, Dims d,
                                                                     double hx, double hy, State *st, double *xs,
                                                                     double *out_norm) {
   pdl_trigger();
   pdl_wait();
   norm_final_body(rowsum, d, hx, hy, st, xs, out_norm, blockIdx.x, gridDim.x);
}

// psi *= scale (calcnorm_kernel, imag3d-mpicuda.cu:1220-1233).
template <class R, bool CPLX>
__global__ void k_apply_scale(typename Tr<R, CPLX>::P *__restrict__ psi, long long n, const State *__restrict__ st) {
   const double s = st->scale;
   for (long long q = blockIdx.x * (long long) blockDim.x + threadIdx.x; q < n; q += (long long) gridDim.x * blockDim.x)
      psi[q] = scl(psi[q], s);
}

static __global__ void k_state_set(State *st, double scale) {
   st->scale = scale;
   st->scale2 = scale * scale;
}

// calcrms (imag3d-mpicuda.cu:1639-1744) from the row partials rowA = S_z
// |psi|^2 and rowB = S_z z^2 |psi|^2: <x^2> = S_x x^2 S_y rowA, <y^2> =
// S_x S_y y^2 rowA, <z^2> = S_x S_y rowB; out = (r, rx, ry, rz).  Each warp
// forms the three weighted Simpson sums over y of one x row into xs[3 nx];
// the last CTA to finish integrates them over x.
static __global__ void __launch_bounds__(32 * kNormRowsPerCta) k_rms_final(const double *__restrict__ rowA,
                                                                    const double *__restrict__ rowB, Dims d, double hx,
                                                                    double hy, const double *__restrict__ x2,
                                                                    const double *__restrict__ y2, State *st,
                                                                    double *xs, double *__restrict__ out) {
   pdl_trigger();
   pdl_wait();
   const int lane = threadIdx.x & 31;
   const int i = blockIdx.x * kNormRowsPerCta + (threadIdx.x >> 5);
   if (i < d.nx) {
      const double *ra = rowA + (long long) i * d.ny, *rb = rowB + (long long) i * d.ny;
      double a = 0., b = 0., c = 0.;
      for (int j = lane; j < d.ny; j += 32) {
         const double w = simp_w(j, d.ny);
         a = fma(w, ra[j], a);
         b = fma(w, rb[j], b);
         c = fma(w * y2[j], ra[j], c);
      }
      for (int o = 16; o; o >>= 1) {
         a += __shfl_xor_sync(0xffffffffu, a, o);
         b += __shfl_xor_sync(0xffffffffu, b, o);
         c += __shfl_xor_sync(0xffffffffu, c, o);
      }
      if (lane == 0) {
         xs[i] = x2[i] * a * hy / 3.;
         xs[d.nx + i] = c * hy / 3.;
         xs[2 * d.nx + i] = b * hy / 3.;
      }
   }
   __threadfence();
   __syncthreads();
   __shared__ bool last;
   if (threadIdx.x == 0) last = atomicAdd(&st->ticket, 1u) == gridDim.x - 1;
   __syncthreads();
   if (!last || threadIdx.x >= 32) return;
   __threadfence();
   double m[3] = {0., 0., 0.};
   for (int k = lane; k < d.nx; k += 32) {
      const double w = simp_w(k, d.nx);
      for (int q = 0; q < 3; q++) m[q] = fma(w, __ldcg(xs + q * d.nx + k), m[q]);
   }
   for (int q = 0; q < 3; q++)
      for (int o = 16; o; o >>= 1) m[q] += __shfl_xor_sync(0xffffffffu, m[q], o);
   if (lane == 0) {
      const double rx = sqrt(m[0] * hx / 3.), ry = sqrt(m[1] * hx / 3.), rz = sqrt(m[2] * hx / 3.);
      out[1] = rx;
      out[2] = ry;
      out[3] = rz;
      out[0] = sqrt(rx * rx + ry * ry + rz * rz);
      st->ticket = 0u;
   }
}

// 4th-order first derivative with the reference's edge rules
// (calcmuen_kernel1x/1y/1z, imag3d-mpicuda.cu:1293-1422) at index i of n from
// the five values around it (those beyond the line are not used).
__device__ __forceinline__ double fd4(double m2, double m1, double p1, double p2, int i, int n, double r2h,
                                      double r12h) {
   if (i == 0 || i == n - 1) return 0.;
   if (i == 1 || i == n - 2) return (p1 - m1) * r2h;
   return (m2 - p2 + 8. * (p1 - m1)) * r12h;
}

// mu and E (calcmuen_kernel2, imag3d-mpicuda.cu:1424-1450; real time
// differentiates |psi|, real3d-mpicuda.cu:1401): a CTA owns kMuY rows of y by
// kMuZ points of z and walks along x over a ring of kMuRing planes of |psi|
// with their two-point halo, so each amplitude is loaded, and its square root
// taken, once per tile and plane.  The integrands are summed with the product
// of the Simpson weights of the three axes (the nested rule of simpint is
// that product); part[2 CTA] receives the CTA's sums, k_sum2 adds them.  One
// thread per (x, y) row walking z (32 rows apart in a warp's loads, 13 square
// roots a point) took 2.5 ms at 256^3 complex FP64; a whole calcmuen call at
// 256^3 real FP64, with its convolution, 1615 -> 680 us.
constexpr int kMuY = 8, kMuZ = 32, kMuRing = 6;
template <class R, bool CPLX>
__global__ void __launch_bounds__(kMuY *kMuZ, 4) k_muen(const typename Tr<R, CPLX>::P *__restrict__ psi,
                                                     const R *__restrict__ phi, Dims d, Trap trap, double g, double gd,
                                                     double dx, double dy, double dz, double par, int xchunk,
                                                     double *__restrict__ part) {
   constexpr int PY = kMuY + 4, PZ = kMuZ + 4, NT = kMuY * kMuZ;
   __shared__ double ring[kMuRing][PY * PZ];
   __shared__ double red[2 * NT / 32];
   const int z0 = blockIdx.x * kMuZ, y0 = blockIdx.y * kMuY, x0 = blockIdx.z * xchunk;
   const int x1 = min(x0 + xchunk, d.nx);
   const int tz = threadIdx.x % kMuZ, ty = threadIdx.x / kMuZ;
   const int j = y0 + ty, k = z0 + tz;
   const bool in = j < d.ny && k < d.nz;
   // plane x with the halo, zero outside the grid: loaded into registers one
   // plane ahead of the amplitudes' square roots and stores
   using P = typename Tr<R, CPLX>::P;
   constexpr int NE = (PY * PZ + NT - 1) / NT;
   P raw[NE];
   auto load = [&](int x) {
#pragma unroll
      for (int u = 0; u < NE; u++) {
         const int e = threadIdx.x + u * NT;
         const int jj = y0 - 2 + e / PZ, kk = z0 - 2 + e % PZ;
         raw[u] = zero_of<P>();
         if (e < PY * PZ && x >= 0 && x < d.nx && jj >= 0 && jj < d.ny && kk >= 0 && kk < d.nz)
            raw[u] = psi[((long long) x * d.ny + jj) * d.nz + kk];
      }
   };
   auto keep = [&](int x) {
      double *r = ring[(x + kMuRing) % kMuRing];
#pragma unroll
      for (int u = 0; u < NE; u++) {
         const int e = threadIdx.x + u * NT;
         if (e < PY * PZ) {
            if constexpr (CPLX) r[e] = sqrt((double) dens2(raw[u]));
            else r[e] = (double) raw[u];
         }
      }
   };
   const double invN = 1.0 / (double) d.npts, ipar = 1. / (3. - par);
   const double hx2 = 1. / (2. * dx), hx12 = 1. / (12. * dx), hy2 = 1. / (2. * dy), hy12 = 1. / (12. * dy),
                hz2 = 1. / (2. * dz), hz12 = 1. / (12. * dz);
   const double wyz = in ? simp_w(j, d.ny) * simp_w(k, d.nz) : 0.;
   double mu = 0., en = 0.;
   const int c = (ty + 2) * PZ + tz + 2;
   const long long sx = (long long) d.ny * d.nz;
   const R *ph = phi + (long long) x0 * sx + (long long) (in ? j : 0) * d.nz + (in ? k : 0);
   for (int x = x0 - 2; x < x0 + 2; x++) {
      load(x);
      keep(x);
   }
   load(x0 + 2);
   R f = *ph;
   for (int x = x0; x < x1; x++) {
      keep(x + 2);
      __syncthreads();  // the slot this fills was last read two iterations ago (six planes, five in use)
      load(x + 3);
      const double fx = (double) f;
      if (x + 1 < x1) f = ph[(x + 1 - x0) * sx];
      if (in) {
         const double *r = ring[x % kMuRing];
         auto rx = [&](int q) { return ring[(x + q + kMuRing) % kMuRing][c]; };
         const double ddx = fd4(rx(-2), rx(-1), rx(1), rx(2), x, d.nx, hx2, hx12);
         const double ddy = fd4(r[c - 2 * PZ], r[c - PZ], r[c + PZ], r[c + 2 * PZ], j, d.ny, hy2, hy12);
         const double ddz = fd4(r[c - 2], r[c - 1], r[c + 1], r[c + 2], k, d.nz, hz2, hz12);
         const double dpsi = (ddx * ddx + ddy * ddy + ddz * ddz) * ipar;
         const double psi2 = r[c] * r[c];
         const double lin = psi2 * g + (fx * invN) * gd;
         const double v = trap.v(x, j, k), w = simp_w(x, d.nx) * wyz;
         mu = fma(w, fma(v + lin, psi2, dpsi), mu);
         en = fma(w, fma(v + 0.5 * lin, psi2, dpsi), en);
      }
   }
   for (int o = 16; o; o >>= 1) {
      mu += __shfl_xor_sync(0xffffffffu, mu, o);
      en += __shfl_xor_sync(0xffffffffu, en, o);
   }
   if (threadIdx.x % 32 == 0) {
      red[threadIdx.x / 32] = mu;
      red[NT / 32 + threadIdx.x / 32] = en;
   }
   __syncthreads();
   if (threadIdx.x < 2) {
      double s = 0.;
      for (int w = 0; w < NT / 32; w++) s += red[threadIdx.x * (NT / 32) + w];
      const long long cta = ((long long) blockIdx.z * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x;
      part[2 * cta + threadIdx.x] = s;
   }
}

// out[0] and out[1]: scaled sums of n pairs, in a fixed order (one CTA).
static __global__ void __launch_bounds__(256) k_sum2(const double *__restrict__ part, int n, double scale,
                                                    double *__restrict__ out) {
   __shared__ double red[2][256];
   double a = 0., b = 0.;
   for (int e = threadIdx.x; e < n; e += 256) {
      const double2 v = ((const double2 *) part)[e];
      a += v.x;
      b += v.y;
   }
   red[0][threadIdx.x] = a;
   red[1][threadIdx.x] = b;
   __syncthreads();
   for (int h = 128; h; h >>= 1) {
      if (threadIdx.x < h) {
         red[0][threadIdx.x] += red[0][threadIdx.x + h];
         red[1][threadIdx.x] += red[1][threadIdx.x + h];
      }
      __syncthreads();
   }
   if (threadIdx.x < 2) out[threadIdx.x] = red[threadIdx.x][0] * scale;
}

// ---- density outputs -------------------------------------------------------
// Line integral of |psi|^2 along `axis` for every line; out is indexed by the
// two remaining axes in (x, y, z) order.
template <class R, bool CPLX>
__global__ void k_lineint_psi(const typename Tr<R, CPLX>::P *__restrict__ psi, Dims d, int axis, double h,
                              double *__restrict__ out) {
   const int n[3] = {d.nx, d.ny, d.nz};
   const long long s[3] = {(long long) d.ny * d.nz, d.nz, 1};
   const int a1 = axis == 0 ? 1 : 0, a2 = axis == 2 ? 1 : 2;
   const long long nl = (long long) n[a1] * n[a2];
   const long long l = (long long) blockIdx.x * blockDim.x + threadIdx.x;
   if (l >= nl) return;
   const long long u = l / n[a2], v = l - u * n[a2];
   const auto *p = psi + u * s[a1] + v * s[a2];
   Simpson sp;
   sp.init(n[axis]);
   for (int c = 0; c < n[axis]; c++) sp.add(c, (double) dens2(p[(long long) c * s[axis]]));
   out[l] = sp.finish(h);
}

// out[u] = Simpson along axis `ax` (0 rows, 1 columns) of a [n0][n1] array.
static __global__ void k_lineint_arr(const double *__restrict__ a, int n0, int n1, int ax, double h, double *__restrict__ out) {
   const int l = blockIdx.x * blockDim.x + threadIdx.x;
   if (ax == 1) {
      if (l < n0) out[l] = simpint_arr(h, a + (long long) l * n1, n1, 1);
   } else {
      if (l < n1) out[l] = simpint_arr(h, a + l, n0, n1);
   }
}

// |psi|^2 gathered on a strided sub-grid of a box (3D cuts and raw density).
template <class R, bool CPLX>
__global__ void k_gather_dens(const typename Tr<R, CPLX>::P *__restrict__ psi, Dims d, int i0, int i1, int si,
                              int j0, int j1, int sj, int k0, int k1, int sk, double *__restrict__ out) {
   const long long ni = (i1 - i0 + si - 1) / si, nj = (j1 - j0 + sj - 1) / sj, nk = (k1 - k0 + sk - 1) / sk;
   const long long tot = ni * nj * nk;
   for (long long e = blockIdx.x * (long long) blockDim.x + threadIdx.x; e < tot; e += (long long) gridDim.x * blockDim.x) {
      const long long a = e / (nj * nk), r = e - a * nj * nk, b = r / nk, c = r - b * nk;
      const long long i = i0 + a * si, j = j0 + b * sj, k = k0 + c * sk;
      out[e] = (double) dens2(psi[(i * d.ny + j) * d.nz + k]);
   }
}

// n elements of one type to the other (psi and phi of mixed-precision handles
// on their way to and from the caller's FP64 arrays).
template <class D, class S> __global__ void k_convert(D *__restrict__ dst, const S *__restrict__ src, long long n) {
   for (long long q = blockIdx.x * (long long) blockDim.x + threadIdx.x; q < n; q += (long long) gridDim.x * blockDim.x)
      dst[q] = (D) src[q];
}

template <class R, bool CPLX>
__global__ void k_init_density(typename Tr<R, CPLX>::P *__restrict__ psi, const double *__restrict__ rho, long long n) {
   using P = typename Tr<R, CPLX>::P;
   for (long long q = blockIdx.x * (long long) blockDim.x + threadIdx.x; q < n; q += (long long) gridDim.x * blockDim.x) {
      const double a = sqrt(rho[q]);
      P v = zero_of<P>();
      if constexpr (CPLX) v.x = (R) a; else v = (R) a;
      psi[q] = v;
   }
}

}  // namespace gpe
