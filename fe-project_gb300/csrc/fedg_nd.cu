// fedg_nd.cu -- numerical diffusion (FElib's hyperdiffusion filter) and the sponge layer, FP64.
//
// Numerical diffusion: each prognostic variable q gets q += dt (-1)^(n+1) coef nabla^(2n) q after
// the dynamics step, the Laplacian built from one-sided LDG fluxes (the gradient takes the exterior
// value on faces with a negative normal, the divergence on faces with a positive one), with
// horizontal and vertical coefficients, density weighting of all variables but DDENS, and the lid
// values of FElib's boundary routines (centred fluxes there).
//   FElib/src/fluid_dyn_solver/scale_atm_dyn_dgm_nonhydro3d_numdiff.F90
//     Apply / apply_numfilter :214-376; numdiff_tend :379-440; cal_del_flux_lap_with_coef :443-500
//     numdiff_cal_laplacian :505-558; cal_del_flux_lap :561-601; numdiff_cal_flx :606-665
//     cal_del_gradDiffVar :668-721
//   lid values  ..._dgm_bnd.F90:370-508 (ApplyBC_numdiff_odd_lc / _even_lc), slip + adiabatic lids
// Sponge layer: Rayleigh damping of MOMZ (and optionally MOMX, MOMY) added to the explicit tendency,
// coefficient 0.25/tau (1 + sign(z - h)) (1 - cos(pi (z - h)/(z_top - h)))
//   ..._dgm_spongelayer.F90:134-219
//
// One thread block per element (EPB elements for p <= 3), one launch per pass and variable.  On the
// axis-aligned faces of the flat cube only the normal component of each face flux is nonzero, so
// each face node carries one value.
#include <cmath>
#include <cstring>
#include <vector>

#include "fedg_ctx.cuh"

namespace fedg {
namespace {

// Tables of a pass.  An interior face's flux is nonzero only on one of its two sides (the gradient takes the
// lower neighbour, the divergence the upper), so an element computes three faces, with Lift lf, and at the lid on the
// other side a fourth with Lift lo; the signs are in lf and lo.  E of each
// direction holds the pass's coefficient; Escale and Fscale are the same 2/dx.
struct NdOps {
  double E[3], lf[FEDG_MAXN1], lo[FEDG_MAXN1];
};

struct ElemIdx {
  long ke;
  int p, le, i, j, k, ex, ey, ez, nxy;
  bool valid;
};
template <int N1, int EPB>
__device__ __forceinline__ ElemIdx elem_idx(const Ops& op, int Ne) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1;
  ElemIdx e;
  const int tid = threadIdx.x;
  e.le = tid / Np;
  e.p = tid - e.le * Np;
  e.ke = (long)blockIdx.x * EPB + e.le;
  e.valid = e.ke < Ne;
  e.i = e.p % N1;
  e.j = (e.p / N1) % N1;
  e.k = e.p / NF;
  e.nxy = op.NeX * op.NeY;
  e.ez = e.valid ? (int)(e.ke / e.nxy) : 0;
  e.ey = e.valid ? (int)((e.ke - (long)e.ez * e.nxy) / op.NeX) : 0;
  e.ex = e.valid ? (int)(e.ke - (long)e.ez * e.nxy - (long)e.ey * op.NeX) : 0;
  return e;
}
// the exterior node of face node ab on the lower (up = 0) or upper face of direction dir, -1 at a lid, and its level
template <int N1>
__device__ __forceinline__ long nd_exterior(const Ops& op, const ElemIdx& e, int dir, int up, int ab, int& lev) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1;
  const int a = ab % N1, b = ab / N1, w = up ? 0 : N1 - 1;
  long kn = e.ke;
  if (dir == 0) kn += up ? (e.ex < op.NeX - 1 ? 1 : -(op.NeX - 1)) : (e.ex > 0 ? -1 : op.NeX - 1);
  else if (dir == 1) kn += up ? (e.ey < op.NeY - 1 ? op.NeX : -(long)(op.NeY - 1) * op.NeX) : (e.ey > 0 ? -op.NeX : (long)(op.NeY - 1) * op.NeX);
  else {
    if (up ? e.ez == op.NeZ - 1 : e.ez == 0) return -1;
    kn += up ? e.nxy : -e.nxy;
  }
  lev = dir == 2 ? (e.ez + (up ? 1 : -1)) * N1 + w : e.ez * N1 + b;
  return kn * Np + (dir == 0 ? w + N1 * ab : (dir == 1 ? a + N1 * w + NF * b : ab + NF * w));
}
// the element's own node of face node ab
template <int N1>
__device__ __forceinline__ int nd_own(int dir, int up, int ab) {
  constexpr int NF = N1 * N1;
  const int a = ab % N1, b = ab / N1, w = up ? N1 - 1 : 0;
  return dir == 0 ? w + N1 * ab : (dir == 1 ? a + N1 * w + NF * b : ab + NF * w);
}
// contraction along direction dir and the Lift of its faces; D: the block's copy of the operator
template <int N1>
__device__ __forceinline__ double nd_dir(const NdOps& nd, const double* D, const double* u, const double* df, int dir,
                                         const ElemIdx& e, bool lid) {
  constexpr int NF = N1 * N1;
  const int row = dir == 0 ? e.i : (dir == 1 ? e.j : e.k), stp = dir == 0 ? 1 : (dir == 1 ? N1 : NF);
  const int ab = dir == 0 ? e.j + N1 * e.k : (dir == 1 ? e.i + N1 * e.k : e.i + N1 * e.j);
  double s = 0.0;
  u += e.p - row * stp;
#pragma unroll
  for (int l = 0; l < N1; ++l) s = fma(D[row * N1 + l], u[l * stp], s);
  s = fma(nd.lf[row], df[dir * NF + ab], s);
  return dir == 2 && lid ? fma(nd.lo[row], df[3 * NF + ab], s) : s;
}

// numdiff_cal_flx: G = (d/dx Vh, d/dy Vh, d/dz Vv) (each divided by the density when dens_div).  refl: at the
// lids the even routine's exterior of Vv reflects it (the wall-normal momentum); otherwise no jump there.
//
// What bounds it: the FP64 pipe, about 47 instructions per node (one quotient for the node and a reciprocal for each
// side of a computed face node).  16x16x8 elements at p = 7: 128 -> 88 us.
template <int N1, int EPB>
__global__ void __launch_bounds__(EPB* N1* N1* N1)
    k_nd_grad(const __grid_constant__ Ops op, const __grid_constant__ NdOps nd, const double* __restrict__ dens_prof,
              const double* __restrict__ Vh, const double* __restrict__ Vv, const double* __restrict__ ddens, int dens_div,
              int refl, double* __restrict__ Gx, double* __restrict__ Gy, double* __restrict__ Gz, int Ne) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1;
  extern __shared__ double sm[];
  const ElemIdx e = elem_idx<N1, EPB>(op, Ne);
  double* D = sm;
  double* vh = sm + NF + e.le * (2 * Np + 4 * NF);
  double* vv = Vh == Vv ? vh : vh + Np;
  double* df = vh + 2 * Np;
  const size_t g = (size_t)e.ke * Np + e.p;
  for (int c = threadIdx.x; c < NF; c += EPB * Np) D[c] = op.D[c];
  const bool top = e.ez == op.NeZ - 1;
  if (e.valid) {
    // quotients, not a reciprocal's products: dens * const gives back the constant, whose derivative vanishes
    const double dens = dens_div ? __ldg(ddens + g) + __ldg(dens_prof + e.ez * N1 + e.k) : 1.0;
    vh[e.p] = dens_div ? __ldg(Vh + g) / dens : __ldg(Vh + g);
    if (vv != vh) vv[e.p] = dens_div ? __ldg(Vv + g) / dens : __ldg(Vv + g);
    // jumps of the lower faces of x, y, z, then the upper lid's, where half counts.  Of a uniform flow nothing is left but
    // the products' rounding, by one formula on every face as in FElib's flux.
    for (int fi = e.p; fi < (top ? 4 : 3) * NF; fi += Np) {
      const int f = fi / NF, dir = f < 2 ? f : 2, ab = fi - f * NF, pM = nd_own<N1>(dir, f == 3, ab);
      const size_t gM = (size_t)e.ke * Np + pM;
      const double* V = dir == 2 ? Vv : Vh;
      double wM = 1.0, wP = 1.0;
      if (dens_div) wM = 1.0 / (__ldg(ddens + gM) + __ldg(dens_prof + e.ez * N1 + pM / NF));
      const double vM = __ldg(V + gM);
      int lev;
      const long gP = f == 3 ? -1 : nd_exterior<N1>(op, e, dir, 0, ab, lev);
      if (gP < 0) {
        df[fi] = 0.5 * fma(refl ? -vM : vM, wM, -(vM * wM));
        continue;
      }
      if (dens_div) wP = 1.0 / (__ldg(ddens + gP) + __ldg(dens_prof + lev));
      df[fi] = fma(__ldg(V + gP), wP, -(vM * wM));
    }
  }
  __syncthreads();
  if (!e.valid) return;
  Gx[g] = nd.E[0] * nd_dir<N1>(nd, D, vh, df, 0, e, false);
  Gy[g] = nd.E[1] * nd_dir<N1>(nd, D, vh, df, 1, e, false);
  Gz[g] = nd.E[2] * nd_dir<N1>(nd, D, vv, df, 2, e, top);
}

// divergence of G (times the density when mul_dens).  At the lids the odd routine's exterior of G reflects it, but
// for the wall-normal momentum (keep: no jump).  TEND: numdiff_tend and V += its sum (nd.E holds dt and the
// coefficients); otherwise numdiff_cal_laplacian's horizontal and vertical parts.
//
// What bounds it: the FP64 pipe, about 38 instructions per node.  16x16x8 elements at p = 7: 102 -> 74 us.
template <int N1, int EPB, bool TEND>
__global__ void __launch_bounds__(EPB* N1* N1* N1)
    k_nd_div(const __grid_constant__ Ops op, const __grid_constant__ NdOps nd, const double* __restrict__ dens_prof,
             const double* __restrict__ Gx, const double* __restrict__ Gy, const double* __restrict__ Gz,
             const double* ddens, int mul_dens, int keep, double* __restrict__ lh, double* __restrict__ lv, double* V, int Ne) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1;
  extern __shared__ double sm[];
  const ElemIdx e = elem_idx<N1, EPB>(op, Ne);
  double* D = sm;
  double* fl = sm + NF + e.le * (3 * Np + 4 * NF);
  double* df = fl + 3 * Np;
  const size_t g = (size_t)e.ke * Np + e.p;
  for (int c = threadIdx.x; c < NF; c += EPB * Np) D[c] = op.D[c];
  const bool bot = !keep && e.ez == 0;
  if (e.valid) {
    // DDENS is read only when it weights the variable (for DDENS itself V aliases it)
    const double dens = mul_dens ? __ldg(dens_prof + e.ez * N1 + e.k) + __ldg(ddens + g) : 1.0;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double x = __ldg((d == 0 ? Gx : (d == 1 ? Gy : Gz)) + g);
      fl[d * Np + e.p] = mul_dens ? dens * x : x;
    }
    for (int fi = e.p; fi < 3 * NF; fi += Np) {
      const int dir = fi / NF;
      int lev;
      const long gP = nd_exterior<N1>(op, e, dir, 1, fi - dir * NF, lev);
      if (gP < 0) continue;
      const double x = __ldg((dir == 0 ? Gx : (dir == 1 ? Gy : Gz)) + gP);
      df[fi] = mul_dens ? (__ldg(dens_prof + lev) + __ldg(ddens + gP)) * x : x;
    }
  }
  __syncthreads();
  if (e.valid) {
    for (int fi = e.p; fi < (bot ? 4 : 3) * NF; fi += Np) {
      const int f = fi / NF, dir = f < 2 ? f : 2;
      const double own = fl[dir * Np + nd_own<N1>(dir, f != 3, fi - f * NF)];
      if (f == 3 || (f == 2 && e.ez == op.NeZ - 1)) df[fi] = keep ? 0.0 : -own;
      else df[fi] -= own;
    }
  }
  __syncthreads();
  if (!e.valid) return;
  const double h = fma(nd.E[0], nd_dir<N1>(nd, D, fl, df, 0, e, false), nd.E[1] * nd_dir<N1>(nd, D, fl + Np, df, 1, e, false));
  const double z = nd_dir<N1>(nd, D, fl + 2 * Np, df, 2, e, bot);
  if (TEND) {
    V[g] += fma(nd.E[2], z, h);
  } else {
    lh[g] = h;
    lv[g] = nd.E[2] * z;
  }
}

// sponge layer: tend -= c(z) (s MOMX, s MOMY, MOMZ), c per level
__global__ void k_sponge(const double* __restrict__ coef, double* __restrict__ tx, double* __restrict__ ty,
                         double* __restrict__ tz, const double* __restrict__ mx, const double* __restrict__ my,
                         const double* __restrict__ mz, double s, int N1, int Np, size_t nxy, size_t n) {
  const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  const size_t ke = g / Np;
  const int lev = (int)(ke / nxy) * N1 + (int)(g - ke * Np) / (N1 * N1);
  const double c = __ldg(coef + lev);
  tx[g] = tx[g] - s * c * __ldg(mx + g);
  ty[g] = ty[g] - s * c * __ldg(my + g);
  tz[g] = tz[g] - c * __ldg(mz + g);
}

template <int N1>
constexpr int nd_epb() { return N1 <= 4 ? (N1 <= 2 ? 16 : (N1 == 3 ? 8 : 4)) : 1; }

NdOps nd_ops(const Ops& d, double ch, double cv, bool lower) {
  NdOps n;
  std::memset(&n, 0, sizeof(n));
  n.E[0] = ch * d.E11;
  n.E[1] = ch * d.E22;
  n.E[2] = cv * d.E33;
  for (int i = 0; i < d.N1; ++i) {
    n.lf[i] = lower ? -d.Lb[i] : d.Lt[i];
    n.lo[i] = lower ? d.Lt[i] : -d.Lb[i];
  }
  return n;
}

struct NdPass {
  int pass;  // 0 gradient, 1 Laplacian, 2 update
  const double *a, *b;  // gradient: the fields of the horizontal and of the vertical derivative
  const double* ddens;
  int dens, wall;  // density division / weight; the lid's reflection (gradient), or none at it (divergence)
  double *G[3], *lh, *lv, *V;
};

template <int N1>
int nd_pass_n(const NdPass& P, const Ops& op, const NdOps& nd, const double* dp, int Ne, cudaStream_t s) {
  constexpr int EPB = nd_epb<N1>(), Np = N1 * N1 * N1, NF = N1 * N1;
  const size_t sm = sizeof(double) * (NF + EPB * ((P.pass == 0 ? 2 : 3) * Np + 4 * NF));
  auto go = [&](auto kf, auto... args) {
    cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    kf<<<(Ne + EPB - 1) / EPB, EPB * Np, sm, s>>>(op, nd, dp, args..., Ne);
    return (int)cudaGetLastError();
  };
  const double *gx = P.G[0], *gy = P.G[1], *gz = P.G[2];
  if (P.pass == 0) return go(k_nd_grad<N1, EPB>, P.a, P.b, P.ddens, P.dens, P.wall, P.G[0], P.G[1], P.G[2]);
  return P.pass == 1 ? go(k_nd_div<N1, EPB, false>, gx, gy, gz, P.ddens, P.dens, P.wall, P.lh, P.lv, P.V)
                     : go(k_nd_div<N1, EPB, true>, gx, gy, gz, P.ddens, P.dens, P.wall, P.lh, P.lv, P.V);
}

int nd_pass(const NdPass& P, const Ops& op, const NdOps& nd, const double* dp, int Ne, cudaStream_t s) {
  switch (op.N1) {
    case 2: return nd_pass_n<2>(P, op, nd, dp, Ne, s);
    case 3: return nd_pass_n<3>(P, op, nd, dp, Ne, s);
    case 4: return nd_pass_n<4>(P, op, nd, dp, Ne, s);
    case 5: return nd_pass_n<5>(P, op, nd, dp, Ne, s);
    case 6: return nd_pass_n<6>(P, op, nd, dp, Ne, s);
    case 7: return nd_pass_n<7>(P, op, nd, dp, Ne, s);
    case 8: return nd_pass_n<8>(P, op, nd, dp, Ne, s);
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace
}  // namespace fedg

namespace fedg {
void sponge_coef_host(const fedg_ctx* c, double tau, double height, double* coef) {
  std::vector<double> xs(c->N1);
  lgl_nodes_1d(c->N1 - 1, xs.data());
  const double dz = (c->d.zmax - c->d.zmin) / c->d.NeZ, rt = 1.0 / tau, ztop = c->d.zmax;
  for (int l = 0; l < c->L; ++l) {
    const int ez = l / c->N1, k = l - ez * c->N1;
    const double z = c->d.zmin + (ez + 0.5 * (xs[k] + 1.0)) * dz;
    coef[l] = 0.25 * rt * (1.0 + (std::signbit(z - height) ? -1.0 : 1.0)) *
              (1.0 - std::cos(M_PI * (z - height) / (ztop - height)));
  }
}
}  // namespace fedg

extern "C" {

int fedg_numdiff_apply(fedg_ctx* c, double* const q[5], int nlap, double coef_h, double coef_v, double dt) {
  return fedg_numdiff_apply_prec(c, q, nlap, coef_h, coef_v, dt, FEDG_PREC_FP64);
}

int fedg_numdiff_apply_prec(fedg_ctx* c, double* const q[5], int nlap, double coef_h, double coef_v, double dt,
                            int prec) {
  if (!c || !q) return api_fail("fedg_numdiff_apply: null argument");
  if (fedg::slab(c)) return api_fail("fedg_numdiff_apply: not available on a part of a decomposed mesh (periodic_x/y = FEDG_HALO)");
  if (prec != FEDG_PREC_FP64 && prec != FEDG_PREC_PAIR)
    return api_fail("fedg_numdiff_apply: prec must be FEDG_PREC_FP64 or FEDG_PREC_PAIR");
  for (int v = 0; v < 5; ++v)
    if (!q[v]) return api_fail("fedg_numdiff_apply: null field");
  if (nlap < 1) return api_fail("fedg_numdiff_apply: ND_LAPLACIAN_NUM must be >= 1");
  if (!c->base_set) return api_fail("fedg_numdiff_apply: the base state is not registered (fedg_set_base_state)");
  cudaSetDevice(c->d.device);
  const size_t n = c->n;
  if (!c->nd_buf) {
    if (cudaMalloc(&c->nd_buf, sizeof(double) * 5 * n) != cudaSuccess) {
      c->nd_buf = nullptr;
      return api_fail("fedg_numdiff_apply: out of device memory (5 fields of scratch)");
    }
  }
  if (prec == FEDG_PREC_PAIR) return numdiff_apply_pair(c, q, nlap, coef_h, coef_v, dt, c->nd_buf);
  double* Gx = c->nd_buf;
  double* Gy = Gx + n;
  double* Gz = Gy + n;
  double* lh = Gz + n;
  double* lv = lh + n;
  const double sgn = ((nlap + 1) % 2 == 0) ? 1.0 : -1.0;  // (-1)^mod(n+1, 2)
  const int order[5] = {VRT, VMZ, VMX, VMY, VD};         // apply_numfilter's order: DDENS changes last
  const NdOps grad = nd_ops(c->op, 1.0, 1.0, true), lap = nd_ops(c->op, 1.0, 1.0, false),
              upd = nd_ops(c->op, dt * (sgn * coef_h), dt * (sgn * coef_v), false);
  for (int vi = 0; vi < 5; ++vi) {
    const int var = order[vi];
    const int dw = var != VD, wall = var == VMZ;
    auto pass = [&](int kind, const double* a, const double* b, int dens, int wl, double* V) {
      const NdPass P{kind, a, b, q[VD], dens, wl, {Gx, Gy, Gz}, lh, lv, V};
      return tracked(c, FEDG_K_ND, [&] {
        return nd_pass(P, c->op, kind == 0 ? grad : (kind == 1 ? lap : upd), c->d_prof, c->Ne, c->stream);
      });
    };
    int r = pass(0, q[var], q[var], dw, wall, nullptr);
    for (int it = 1; it < nlap && !r; ++it) {
      r = pass(1, nullptr, nullptr, 0, wall, nullptr);
      if (!r) r = pass(0, lh, lv, 0, 0, nullptr);
    }
    if (!r) r = pass(2, nullptr, nullptr, dw, wall, q[var]);
    if (r) return api_cuda_fail((cudaError_t)r, "fedg_numdiff_apply");
  }
  return 0;
}

int fedg_sponge_add_tend(fedg_ctx* c, double* const tend[3], const double* const mom[3], double tau, double height,
                         int hveldamp) {
  if (!c || !tend || !mom) return api_fail("fedg_sponge_add_tend: null argument");
  for (int d = 0; d < 3; ++d)
    if (!tend[d] || !mom[d]) return api_fail("fedg_sponge_add_tend: null field");
  if (!(tau > 0.0)) return api_fail("fedg_sponge_add_tend: tau must be positive");
  if (!(height < c->d.zmax)) return api_fail("fedg_sponge_add_tend: the damping height must be below the top");
  cudaSetDevice(c->d.device);
  std::vector<double> coef(c->L);
  sponge_coef_host(c, tau, height, coef.data());
  if (!c->sponge_coef && cudaMalloc(&c->sponge_coef, sizeof(double) * c->L) != cudaSuccess) {
    c->sponge_coef = nullptr;
    return api_fail("fedg_sponge_add_tend: out of device memory");
  }
  const bool upload = !(c->sponge_key[0] == tau && c->sponge_key[1] == height);
  if (upload) {  // the profile is uploaded only when (tau, height) change
    if (cudaMemcpyAsync(c->sponge_coef, coef.data(), sizeof(double) * c->L, cudaMemcpyHostToDevice, c->stream) !=
        cudaSuccess)
      return api_fail("fedg_sponge_add_tend: coefficient upload");
    c->sponge_key[0] = tau;
    c->sponge_key[1] = height;
  }
  const int r = tracked(c, FEDG_K_ND, [&] {
    k_sponge<<<(unsigned)((c->n + 255) / 256), 256, 0, c->stream>>>(c->sponge_coef, tend[0], tend[1], tend[2], mom[0],
                                                                   mom[1], mom[2], hveldamp ? 1.0 : 0.0, c->N1, c->Np,
                                                                   c->nxy, c->n);
    return (int)cudaGetLastError();
  });
  if (r) return api_cuda_fail((cudaError_t)r, "fedg_sponge_add_tend");
  // the host coefficient array must outlive the asynchronous copy
  if (upload && cudaStreamSynchronize(c->stream) != cudaSuccess) return api_fail("fedg_sponge_add_tend: synchronise");
  return 0;
}

}  // extern "C"
