// fedg_kernels.cuh -- launcher declarations shared by the translation units.
#pragma once
#include "fedg_common.cuh"

namespace fedg {

struct F5 { double* v[5]; };
struct F5c { const double* v[5]; };

// column-solve controls
struct ViArgs {
  double impl_fac, dt, tol;
  int max_iter;
  double cref;  // velocity scale of the MOMZ convergence test [m/s]
};

// host: 1D exponential modal filter matrix (row-major N1 x N1) of order N
void modal_filter_1d(int N, double etac, double alpha, int ord, double* F);
// host: the N+1 LGL nodes on [-1, 1]
void lgl_nodes_1d(int N, double* x);

int launch_tend_fp64(const Ops& op, const Prof& pf, const F5c& q, const double* dpres, const F5& t, int Ne,
                     int hevi, cudaStream_t s);
// A whole SSP-RK3 stage of the HEVE equations: qn = A q0 + B q + C tend(q), the modal filter if `filter`, and
// DPRES of qn into dpn unless NULL.  q0 may be qn's buffers; q and dpres, which neighbours read, may not.
struct SspArgs {
  F5c q0;
  F5 qn;
  double* dpn;
  double A, B, C;
  int filter;
};
int launch_ssp_stage_fp64(const Ops& op, const Prof& pf, const F5c& q, const double* dpres, const SspArgs& x, int Ne,
                          cudaStream_t s);
int launch_filter_fp64(const Ops& op, const F5& q, int Ne, cudaStream_t s);
int launch_drhot2pres(const Ops& op, const Prof& pf, const double* drhot, double* pres, double* dpres, size_t n,
                      cudaStream_t s);

// Vertical-implicit column solve (cal_vi).  qin: stage input q*, z: guess/var0 (also the
// state alph is frozen at).  tout: tendency (Q - q*)/impl_fac, or A(z) when impl_fac == 0.
// status[ncol]: solves used, -1 not converged, -2 non-finite.  gsc: scratch of at least
// vi_fp64_scratch_doubles(op) doubles (0 when the column does not fit in shared memory).
size_t vi_fp64_scratch_doubles(const Ops& op);
int launch_vi_fp64(const Ops& op, const Prof& pf, const F5c& qin, const F5c& z, const F5& tout, int* status,
                   const ViArgs& a, double* gsc, size_t gsc_doubles, cudaStream_t s);

// Its first pass, by iterative refinement (fedg_vi64.cu): columns it leaves get status VI_REDO and are
// solved by block LU.  Returns -1, nothing launched, if the columns are too tall for its shared memory or block LU serves
// the call better alone.
constexpr int VI_REDO = -100;
// The sweeps of both first passes (fedg_sweep.cuh, fedg_viseries.cu) contract by a factor that depends on the order and on
// the face dissipation's diagonal entry d = (impl_fac/2) Lift(0, bottom) Fscale_z c, c the base state's largest sound
// speed.  Above vi_courant_max, d of the spectral radius 0.58 (of (1 - w) I - w K, computed for columns of 1 to 16
// elements without gravity), the first pass is not launched: few columns would come out of it.  First pass and block
// LU, a step of 24x24x16 elements in float pairs at p = 7 in ms: d = 0.65 4.5 and 6.8, d = 0.9 5.7 and 6.8; 16x16x8 in
// FP64 d = 0.65 5.6 and 18.0; p = 3 in float pairs d = 0.65 0.59 and 0.64, d = 0.81 0.87 and 0.64.
inline double vi_courant(const Ops& op, double impl_fac) { return 0.5 * impl_fac * op.Lb[0] * op.FSz * op.cs_max; }
inline double vi_courant_max(int N1) {
  return N1 == 2 ? 0.40 : N1 == 3 ? 0.53 : N1 == 4 ? 0.65 : N1 == 5 ? 0.72 : N1 == 6 ? 0.78 : N1 == 7 ? 0.83 : 0.90;
}
size_t vi64_scratch_doubles(const Ops& op);
int launch_vi64(const Ops& op, const Prof& pf, const F5c& qin, const F5c& z, const F5& tout, int* status, const ViArgs& a,
                double* gsc, size_t gsc_doubles, cudaStream_t s);

}  // namespace fedg
