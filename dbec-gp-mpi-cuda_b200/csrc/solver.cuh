// solver.cuh -- the solver handle and the operators on it, per real type and
// mode: declared here for the planning and the C ABI (solver.cu), defined in
// impl.cuh and compiled in impl_*.cu and conv_*.cu, one translation unit each.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <complex>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "batch_kernels.cuh"
#include "gpe.h"
#include "internal.h"
#include "step_kernels.cuh"
#include "sweep_kernels.cuh"

using namespace gpe;

gpe_status fail(gpe_status st, const std::string &msg);

// On failure the runtime's last-error slot is cleared so that a non-sticky
// error is reported once, by the call that caused it.
#define CK(call)                                                                                   \
   do {                                                                                           \
      cudaError_t e_ = (call);                                                                    \
      if (e_ != cudaSuccess) {                                                                    \
         (void) cudaGetLastError();                                                               \
         return fail(e_ == cudaErrorMemoryAllocation ? GPE_ERR_OOM : GPE_ERR_CUDA,                \
                     std::string(#call) + ": " + cudaGetErrorString(e_));                          \
      }                                                                                           \
   } while (0)

#define CKL()                                                                                      \
   do {                                                                                           \
      cudaError_t e_ = cudaGetLastError();                                                        \
      if (e_ != cudaSuccess) return fail(GPE_ERR_CUDA, std::string("launch: ") + cudaGetErrorString(e_)); \
   } while (0)

#define CKS(expr)                                                                                  \
   do {                                                                                           \
      gpe_status s_ = (expr);                                                                     \
      if (s_ != GPE_OK) return s_;                                                                \
   } while (0)

struct gpe_solver {
   gpe_params p;
   int dev = 0;
   cudaStream_t st = nullptr;
   bool own_stream = false;
   bool cplx = false, fp32 = false;
   Dims d{};
   double par = 1.;
   FftPlan px{}, pxi{}, py{}, ph{};  // x lines forward and inverse, y lines and half-length z lines
   // x, y, z passes: 1 a compile-time length of the common set, 2 one of the
   // sets for one solve, 0 the run-time pass
   int fastx = 0, fasty = 0, fastz = 0;
   int LSr = 0, LSo = 0;                  // shared row strides of the z passes
   CUtensorMap tm_spec_y{}, tm_spec_x{};  // spectrum tiles of the y and x passes
   CUtensorMap tm_udd{};                  // Udd columns of the x pass's tiles
   int boxy = 0, nboxy = 1, boxx = 0, nboxx = 1;
   int Ly = 8, Lx = 8;  // kz columns per tile of the y and x passes
   gpe_tuning tune{};   // requested tile configuration (0 = default heuristic)
   // bumped whenever the tiles are planned again (their tables reallocated):
   // batches built over this handle rebuild their descriptors when it moves
   unsigned long long plan_gen = 0;
   size_t esz_psi = 8, esz_c = 16, esz_r = 8;
   void *psi = nullptr, *spec = nullptr, *phi = nullptr;
   void *twx = nullptr, *twy = nullptr, *twz = nullptr;
   double *udd = nullptr;
   std::vector<std::complex<double>> alpha[3], gamma[3];  // the Thomas coefficients (gencoef)
   double2 A[3];
   double *x2 = nullptr, *y2 = nullptr, *z2 = nullptr;
   float *x2f = nullptr, *y2f = nullptr, *z2f = nullptr;  // FP32 copies (mixed precision)
   void *lin[3] = {nullptr, nullptr, nullptr};  // per-axis trap factors of calcnu, imag (LinPhase)
   double *rowA = nullptr, *rowB = nullptr, *tmp = nullptr, *obs = nullptr;
   double *rms_buf = nullptr;  // rms samples of gpe_run, kRmsSlots x 4 doubles

   long long row_cap = 0;  // doubles in rowA / rowB: the largest of nx*ny, nx*nz, ny*nz
   State *state = nullptr;
   std::vector<double> hx, hy, hz, hx2, hy2, hz2;
   std::vector<unsigned char> nu_x;  // calcnu's table along x as the sweeps hold it
   long long launches = 0;
   // sweep configuration per axis (x, y: TMA tensor tiles; z: bulk rows)
   struct Sweep {
      int TW = 8, MSEG = 8, boxn = 0, nbox = 1, LS = 0, S = 2, ctas = 1;
      size_t smem = 0;
      CUtensorMap tm_psi{}, tm_phi{};
      SegTab tab{};
      // block of coefficient tables (FP64, or rounded once to FP32 in mixed
      // precision): sweep_tab_bytes
      void *tabs = nullptr;
   } sw[3];
   double *wz = nullptr;      // Simpson weights along z (norm partials)
   double *wz2 = nullptr;     // wz[k] * z[k]^2 (rms partials)
   int nsm = 148;             // streaming multiprocessors of the device
   uint32_t *err = nullptr;   // device status word (bounded waits)
   mutable RoomyKernels roomy;  // launched with more dynamic shared memory than the default
   // per-kernel profiling: when prof_ev is set, mark() records an event
   // after every kernel of a step
   cudaEvent_t *prof_ev = nullptr;
   int prof_i = 0, prof_cap = 0;
};

// rms samples gpe_run keeps on the device before copying them out (a run with
// more samples copies every full batch of slots while it continues)
constexpr long kRmsSlots = 256;

// zero entries before index 0 of the tables the sweeps index from the rows
// below a line (at least the longest segment)
constexpr int kTabPad = 32;

// Doubles the spectrum buffer holds: scratch for copies to and from the host
// (its contents live only inside one convolution).
inline size_t spec_doubles(const gpe_solver *s) {
   return s->esz_c * (size_t) s->d.nzp * (size_t) s->d.nxy / sizeof(double);
}

inline void mark(gpe_solver *s) {
   if (s->prof_ev && s->prof_i < s->prof_cap) cudaEventRecord(s->prof_ev[s->prof_i++], s->st);
}

// 3D tensor map over a [nx][ny][w * nz] array of `esz`-byte scalars with box
// {bw, by, bx} (innermost first).  Rows are `pitch` elements apart (pitch =
// w_nz when 0).
gpe_status make_tmap(CUtensorMap *m, void *base, size_t esz, long w_nz, long ny, long nx, int bw, int by, int bx,
                     long pitch = 0);

// Tensor map of Udd's columns for x tiles of L kz columns (rows padded to an
// even pitch: TMA strides are multiples of 16 bytes).
inline int udd_pitch(int nzh) { return (nzh + 1) & ~1; }
inline gpe_status make_udd_tmap(const gpe_solver *s, CUtensorMap *m, int L) {
   return make_tmap(m, s->udd, 8, s->d.nzh, s->d.ny / 2 + 1, s->d.nx / 2 + 1, L, 1, udd_box(s->d.nx, L).rows,
                    udd_pitch(s->d.nzh));
}

// Bytes of one pipeline stage of the x or y sweep.
inline size_t sweep_stage(const gpe_solver *s, int ax, int rows, int TW, int skip) {
   if (s->fp32)
      return s->cplx ? (ax == 0 ? xy_stage<float, true, true>(rows, TW, skip) : xy_stage<float, true, false>(rows, TW, skip)).bytes
                     : (ax == 0 ? xy_stage<float, false, true>(rows, TW, skip) : xy_stage<float, false, false>(rows, TW, skip)).bytes;
   return s->cplx ? (ax == 0 ? xy_stage<double, true, true>(rows, TW, skip) : xy_stage<double, true, false>(rows, TW, skip)).bytes
                  : (ax == 0 ? xy_stage<double, false, true>(rows, TW, skip) : xy_stage<double, false, false>(rows, TW, skip)).bytes;
}

// Operators of a handle (impl.cuh).
template <class R, bool CPLX> struct Ops {
   static gpe_status psidd2(gpe_solver *s);
   static gpe_status xsweep(gpe_solver *s, bool nu, double g, double gd);
   static gpe_status ysweep(gpe_solver *s);
   static gpe_status zsweep(gpe_solver *s, int mom);
   static gpe_status apply_scale(gpe_solver *s);
   static gpe_status calcnorm(gpe_solver *s, bool renorm);
   static gpe_status calcnu(gpe_solver *s, double g, double gd);
   static gpe_status rms(gpe_solver *s, double *dev_out);
   static gpe_status rms_final(gpe_solver *s, double *dev_out);
   static gpe_status muen(gpe_solver *s, double g, double gd, double *dev_out);
   static gpe_status step(gpe_solver *s, double g, double gd, double *dev_norm, bool rms_rows = false);
   static gpe_status density(gpe_solver *s, int kind, long sx, long sy, long sz, double *out, long cap, long *count);
   static gpe_status geom(gpe_solver *s, int Ly, int Lx, BatchGeom *g);
   static gpe_status desc(gpe_solver *s, int Ly, int Lx, double g, double gd, BatchDesc *D);
};
