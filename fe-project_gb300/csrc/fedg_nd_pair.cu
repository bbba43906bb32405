// fedg_nd_pair.cu -- the numerical diffusion of fedg_nd.cu in float pairs (FEDG_PREC_PAIR).
//
// Same passes, fluxes and lid values as the FP64 kernels (FElib's nonhydro3d_numdiff.F90:214-721,
// ..._dgm_bnd.F90:370-508), with every intermediate an unevaluated float pair (fedg_f2.cuh): the
// FP64 fields are split with integer instructions on load, the gradient and Laplacian fields stay
// pairs between passes, contractions and Lift are compensated sums of exact products, divisions are
// pair reciprocals.  The update adds the pair increment dt*tend to the FP64 field in FP64 (two
// adds), so the field keeps all of its bits.
// Why: the FP64 passes keep GB300's FP64 pipe ~87 % busy; the FP32 pipe issues 64x faster.
//
// Layout: one thread carries the same node of two consecutive elements in the packed pair arithmetic of
// fedg_p2.cuh, so operator tables, indices along a line and the kernels of odd orders are shared by both.
// An interior face's flux is nonzero only on one of its two sides (the gradient takes the lower neighbour,
// the divergence the upper), so an element computes three faces, and a lid face only where the
// reflection leaves a jump.  Coefficients and dt are multiplied into E on the host.
//
// On large p = 7 meshes a thread owns NPT = 2 nodes (k and k + N1/2), which share the loads of the x and y tables.
//
// What bounds it: the latency of the loads and the barriers between them, the faces and the sums (FP32 pipe 40 %
// busy with two blocks of 512 threads per SM), so the blocks are small and many.  Update of five fields, 32x32x16
// elements, p = 7: six blocks of 256 threads per SM (40 registers) 1.59 ms, five 1.62; in an earlier form of the
// sums six 1.51, four of 256 (64 registers) 1.78, three of 512 threads with one node each 1.97, eight of 128 with
// four nodes each 1.77.  With one element and scalar pairs per thread, six faces and 512 threads it took 3.47 ms.
// The neighbours' face values are loaded with the element's own.
#include <cmath>
#include <cstring>

#include "fedg_ctx.cuh"
#include "fedg_two.cuh"

namespace fedg {
namespace {

// operator tables, [l][i]: D(i, l); the Lift of the face an interior element takes its flux from (lf) and of the
// opposite face, a lid (lo), with the face flux's sign; E of each direction, the pass's factor multiplied in
struct NdOpsP {
  float2 D[FEDG_MAXN1 * FEDG_MAXN1];
  float2 E[3], lf[FEDG_MAXN1], lo[FEDG_MAXN1];
  int NeX, NeY, NeZ;
};
template <int N1>
struct NdTab {
  p2m D[N1 * N1], lf[N1], lo[N1];
};
template <int N1>
__device__ __forceinline__ void nd_tables(const NdOpsP& op, NdTab<N1>& T) {
  for (int c = threadIdx.x; c < N1 * N1; c += blockDim.x) {
    st(T.D[c], p2_dup(op.D[c]));
    if (c < N1) {
      st(T.lf[c], p2_dup(op.lf[c]));
      st(T.lo[c], p2_dup(op.lo[c]));
    }
  }
}

// a field read either as FP64 (the prognostic variable) or as pairs (an intermediate)
struct Src {
  const double* d;
  const float2* p;
  __device__ __forceinline__ f2 at(size_t g) const { return d ? f2_split(__ldg(d + g)) : f2_of(__ldg(p + g)); }
};
__device__ __forceinline__ p2 nd_dens(const double* __restrict__ prof, const double* __restrict__ dd, const int (&lev)[2],
                                      const size_t (&g)[2]) {
  return p2_split(__ldg(dd + g[0]), __ldg(dd + g[1])) + p2_split(__ldg(prof + lev[0]), __ldg(prof + lev[1]));
}

// E times (the contraction along direction dir + the Lift of its faces): Fscale and Escale are the same 2/dx, and
// one factor keeps its rounding common to both terms, which cancel to a large part.  Each direction has a sum of
// its own: the rounding of a compensated sum's error term grows with the number of terms (the update's 27 in one
// sum: an error of 1.05e-14 of the change at p = 7; as here 6.2e-15)
template <int N1, int NPT>
__device__ __forceinline__ void nd_dir(p2 (&r)[NPT], const NdTab<N1>& T, p2 E, const p2m* u, const p2m* df, int dir, int i,
                                       int j, int k, bool lid) {
  constexpr int NF = N1 * N1, KH = N1 / NPT;
  const int row = dir == 0 ? i : j;
  p2acc s[NPT];
#pragma unroll
  for (int l = 0; l < N1; ++l) {
    p2 d, v;
    if (dir < 2) d = ld(T.D[l * N1 + row]);
    else v = ld(u[two_at<N1>(i, j + N1 * l)]);
#pragma unroll
    for (int h = 0; h < NPT; ++h) {
      const int kh = k + h * KH;
      if (dir < 2) v = ld(u[dir == 0 ? two_at<N1>(l, j + N1 * kh) : two_at<N1>(i, l + N1 * kh)]);
      else d = ld(T.D[l * N1 + kh]);
      s[h].add(d, v);
    }
  }
#pragma unroll
  for (int h = 0; h < NPT; ++h) {
    const int kh = k + h * KH, rw = dir == 2 ? kh : row;
    const int ab = dir == 0 ? j + N1 * kh : (dir == 1 ? i + N1 * kh : i + N1 * j);
    s[h].add(ld(T.lf[rw]), ld(df[dir * NF + ab]));
    if (dir == 2 && lid) s[h].add(ld(T.lo[rw]), ld(df[3 * NF + ab]));
    r[h] = E * s[h].get();
  }
}

// gradient pass: G = (d/dx Vh, d/dy Vh, d/dz Vv), divided by the density when dens_div; at a lid the even
// routine's exterior of Vv (when bc_v), which leaves a jump only for the wall-normal momentum.
// ONE: Vh and Vv are the same field.
template <int N1, int PPB, int NPT, bool ONE>
__global__ void __launch_bounds__(PPB* N1* N1* N1 / NPT, two_minb(PPB * N1 * N1 * N1 / NPT, 1536))
    k_nd_grad_p(const __grid_constant__ NdOpsP op, const double* __restrict__ dens_prof, const Src Vh, const Src Vv,
                const double* __restrict__ ddens, int dens_div, int refl, float2* __restrict__ Gx,
                float2* __restrict__ Gy, float2* __restrict__ Gz, int Ne) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1, NT = Np / NPT, KH = N1 / NPT;
  extern __shared__ p2m smp[];
  NdTab<N1>& T = *reinterpret_cast<NdTab<N1>*>(smp);
  int pair;
  const TwoIdx x = two_idx<N1, PPB, NT>(op, Ne, pair);
  p2m* vh = smp + sizeof(NdTab<N1>) / sizeof(p2m) + pair * ((ONE ? 1 : 2) * Np + 4 * NF);
  p2m* vv = ONE ? vh : vh + Np;
  p2m* df = vv + Np;
  const size_t g[2] = {(size_t)x.e[0] * Np + x.p, (size_t)x.e[1] * Np + x.p};
  nd_tables<N1>(op, T);
  if (x.valid) {
#pragma unroll
    for (int h = 0; h < NPT; ++h) {
      const size_t gh[2] = {g[0] + h * NT, g[1] + h * NT};
      p2 a = p2_of(Vh.at(gh[0]), Vh.at(gh[1])), b = ONE ? a : p2_of(Vv.at(gh[0]), Vv.at(gh[1]));
      if (dens_div) {
        const int lev[2] = {x.ez[0] * N1 + x.k + h * KH, x.ez[1] * N1 + x.k + h * KH};
        const p2 rd = p2_recip(nd_dens(dens_prof, ddens, lev, gh));
        a = a * rd;
        if (!ONE) b = b * rd;
      }
      const int at = two_at<N1>(x.i, x.j + N1 * (x.k + h * KH));
      st(vh[at], a);
      if (!ONE) st(vv[at], b);
    }
  }
  const bool top = refl && (x.ez[0] == op.NeZ - 1 || x.ez[1] == op.NeZ - 1);
  if (x.valid) {
    for (int fi = x.p; fi < 3 * NF; fi += NT) {
      const int dir = fi / NF, ab = fi - dir * NF;
      int iP, rP;
      two_face_node<N1>(dir, 1, ab, iP, rP);
      size_t gP[2];
      int lev[2];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int kn = two_nbr(op, x, m, dir, 0);
        gP[m] = (size_t)(kn < 0 ? x.e[m] : kn) * Np + rP * N1 + iP;
        lev[m] = (dir == 2 && kn >= 0 ? x.ez[m] - 1 : x.ez[m]) * N1 + rP / N1;
      }
      const Src& S = dir == 2 ? Vv : Vh;
      p2 sP = p2_of(S.at(gP[0]), S.at(gP[1]));
      if (dens_div) sP = sP * p2_recip(nd_dens(dens_prof, ddens, lev, gP));
      st(df[fi], sP);
    }
  }
  __syncthreads();
  // jumps of the lower faces of x, y, z, then the upper lid's
  if (x.valid) {
    for (int fi = x.p; fi < (top ? 4 : 3) * NF; fi += NT) {
      const int f = fi / NF, ab = fi - f * NF, dir = f < 2 ? f : 2;
      int iM, rM;
      two_face_node<N1>(dir, f == 3, ab, iM, rM);
      const p2 own = ld((dir == 2 ? vv : vh)[two_at<N1>(iM, rM)]);
      const int lz = f == 3 ? op.NeZ - 1 : 0;  // lid layer; -2 v there against the coefficient's 1/2
      const bool la = f >= 2 && x.ez[0] == lz, lb = f >= 2 && x.ez[1] == lz;
      p2 d = f == 3 ? p2_zero() : ld(df[fi]) - own;
      if (la || lb) {
        const p2 r = refl ? p2_neg(own) : p2_zero();
        d = p2_of(la ? p2_a(r) : p2_a(d), lb ? p2_b(r) : p2_b(d));
      }
      st(df[fi], d);
    }
  }
  __syncthreads();
  if (!x.valid) return;
#pragma unroll
  for (int dir = 0; dir < 3; ++dir) {
    p2 r[NPT];
    nd_dir<N1, NPT>(r, T, p2_dup(op.E[dir]), dir == 2 ? vv : vh, df, dir, x.i, x.j, x.k, top);
    float2* G = dir == 0 ? Gx : (dir == 1 ? Gy : Gz);
#pragma unroll
    for (int h = 0; h < NPT; ++h) {
      G[g[0] + h * NT] = f2_pack(p2_a(r[h]));
      if (x.both) G[g[1] + h * NT] = f2_pack(p2_b(r[h]));
    }
  }
}

// divergence of the gradient (times the density when mul_dens), with the odd routine's lid exterior of
// it, which leaves a jump except for the wall-normal momentum (keep).  TEND: V += the sum, whose
// tables hold dt and the coefficients (the increment in pairs, added to the FP64 field in FP64); else the Laplacian's
// horizontal and vertical parts.
template <int N1, int PPB, int NPT, bool TEND>
__global__ void __launch_bounds__(PPB* N1* N1* N1 / NPT, two_minb(PPB * N1 * N1 * N1 / NPT, 1536))
    k_nd_div_p(const __grid_constant__ NdOpsP op, const double* __restrict__ dens_prof, const float2* __restrict__ Gx,
               const float2* __restrict__ Gy, const float2* __restrict__ Gz, const double* ddens, int mul_dens, int keep,
               float2* __restrict__ lh, float2* __restrict__ lv, double* V, int Ne) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1, NT = Np / NPT, KH = N1 / NPT;
  extern __shared__ p2m smp[];
  NdTab<N1>& T = *reinterpret_cast<NdTab<N1>*>(smp);
  int pair;
  const TwoIdx x = two_idx<N1, PPB, NT>(op, Ne, pair);
  p2m* fl = smp + sizeof(NdTab<N1>) / sizeof(p2m) + pair * (3 * Np + 4 * NF);
  p2m* df = fl + 3 * Np;
  const size_t g[2] = {(size_t)x.e[0] * Np + x.p, (size_t)x.e[1] * Np + x.p};
  nd_tables<N1>(op, T);
  if (x.valid) {
#pragma unroll
    for (int h = 0; h < NPT; ++h) {
      const size_t gh[2] = {g[0] + h * NT, g[1] + h * NT};
      p2 v[3];
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const float2* G = d == 0 ? Gx : (d == 1 ? Gy : Gz);
        v[d] = p2_of(__ldg(G + gh[0]), __ldg(G + gh[1]));
      }
      if (mul_dens) {  // DDENS is read only when it weights the variable (for DDENS itself V aliases it)
        const int lev[2] = {x.ez[0] * N1 + x.k + h * KH, x.ez[1] * N1 + x.k + h * KH};
        const p2 dens = nd_dens(dens_prof, ddens, lev, gh);
#pragma unroll
        for (int d = 0; d < 3; ++d) v[d] = dens * v[d];
      }
#pragma unroll
      for (int d = 0; d < 3; ++d) st(fl[d * Np + two_at<N1>(x.i, x.j + N1 * (x.k + h * KH))], v[d]);
    }
  }
  const bool bot = !keep && (x.ez[0] == 0 || x.ez[1] == 0);
  if (x.valid) {
    for (int fi = x.p; fi < 3 * NF; fi += NT) {
      const int dir = fi / NF, ab = fi - dir * NF;
      int iP, rP;
      two_face_node<N1>(dir, 0, ab, iP, rP);
      size_t gP[2];
      int lev[2];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const int kn = two_nbr(op, x, m, dir, 1);
        gP[m] = (size_t)(kn < 0 ? x.e[m] : kn) * Np + rP * N1 + iP;
        lev[m] = (dir == 2 && kn >= 0 ? x.ez[m] + 1 : x.ez[m]) * N1 + rP / N1;
      }
      const float2* G = dir == 0 ? Gx : (dir == 1 ? Gy : Gz);
      p2 sP = p2_of(__ldg(G + gP[0]), __ldg(G + gP[1]));
      if (mul_dens) sP = nd_dens(dens_prof, ddens, lev, gP) * sP;
      st(df[fi], sP);
    }
  }
  __syncthreads();
  // jumps of the upper faces of x, y, z, then the lower lid's
  if (x.valid) {
    for (int fi = x.p; fi < (bot ? 4 : 3) * NF; fi += NT) {
      const int f = fi / NF, ab = fi - f * NF, dir = f < 2 ? f : 2;
      int iM, rM;
      two_face_node<N1>(dir, f != 3, ab, iM, rM);
      const p2 own = ld(fl[dir * Np + two_at<N1>(iM, rM)]);
      const int lz = f == 3 ? 0 : op.NeZ - 1;
      const bool la = f >= 2 && x.ez[0] == lz, lb = f >= 2 && x.ez[1] == lz;
      p2 d = f == 3 ? p2_zero() : ld(df[fi]) - own;
      if (la || lb) {
        const p2 r = keep ? p2_zero() : p2_neg(own);
        d = p2_of(la ? p2_a(r) : p2_a(d), lb ? p2_b(r) : p2_b(d));
      }
      st(df[fi], d);
    }
  }
  __syncthreads();
  if (!x.valid) return;
  p2 r[NPT], t[NPT];
  nd_dir<N1, NPT>(r, T, p2_dup(op.E[0]), fl, df, 0, x.i, x.j, x.k, false);
  nd_dir<N1, NPT>(t, T, p2_dup(op.E[1]), fl + Np, df, 1, x.i, x.j, x.k, false);
#pragma unroll
  for (int h = 0; h < NPT; ++h) {
    r[h] = r[h] + t[h];
    if (!TEND) {
      lh[g[0] + h * NT] = f2_pack(p2_a(r[h]));
      if (x.both) lh[g[1] + h * NT] = f2_pack(p2_b(r[h]));
    }
  }
  nd_dir<N1, NPT>(t, T, p2_dup(op.E[2]), fl + 2 * Np, df, 2, x.i, x.j, x.k, bot);
#pragma unroll
  for (int h = 0; h < NPT; ++h) {
    if (TEND) t[h] = r[h] + t[h];
    const f2 a = p2_a(t[h]), b = p2_b(t[h]);
    const size_t ga = g[0] + h * NT, gb = g[1] + h * NT;
    if (TEND) {
      V[ga] = (V[ga] + (double)a.h) + (double)a.l;
      if (x.both) V[gb] = (V[gb] + (double)b.h) + (double)b.l;
    } else {
      lv[ga] = f2_pack(a);
      if (x.both) lv[gb] = f2_pack(b);
    }
  }
}

float2 hsplit_nd(double x) {
  const float h = (float)x;
  return make_float2(h, (float)(x - (double)h));
}

// tables of a pass: factors of the three directions, and which side interior elements take their flux from
NdOpsP nd_ops(const Ops& d, const double (&fac)[3], bool lower) {
  NdOpsP op;
  std::memset(&op, 0, sizeof(op));
  const int N1 = d.N1;
  const double E[3] = {d.E11, d.E22, d.E33};
  for (int c = 0; c < 3; ++c) op.E[c] = hsplit_nd(fac[c] * E[c]);
  for (int i = 0; i < N1; ++i) {
    for (int l = 0; l < N1; ++l) op.D[l * N1 + i] = hsplit_nd(d.D[i * N1 + l]);
    op.lf[i] = hsplit_nd(lower ? -d.Lb[i] : d.Lt[i]);
    op.lo[i] = hsplit_nd(lower ? d.Lt[i] : -d.Lb[i]);
  }
  op.NeX = d.NeX;
  op.NeY = d.NeY;
  op.NeZ = d.NeZ;
  return op;
}

// pairs of elements per block: 108 to 512 threads
template <int N1>
constexpr int nd_ppb() { return N1 <= 4 ? (N1 == 2 ? 16 : (N1 == 3 ? 4 : 2)) : 1; }

struct NdPass {
  int pass;  // 0 gradient, 1 Laplacian, 2 update
  Src a, b;  // gradient: the fields of the horizontal and of the vertical derivative
  const double* ddens;
  int dens, wall;  // density division / weight; the lid's reflection (gradient), or none at it (divergence)
  float2 *G[3], *lh, *lv;
  double* V;
};

template <int N1, int NPT>
int nd_pass_n(const NdPass& P, const NdOpsP& op, const double* dp, int Ne, cudaStream_t s) {
  constexpr int PPB = nd_ppb<N1>(), Np = N1 * N1 * N1, NF = N1 * N1;
  const int grid = ((Ne + 1) / 2 + PPB - 1) / PPB;
  const bool one = P.pass == 0 && P.a.d == P.b.d && P.a.p == P.b.p;
  const size_t sm = sizeof(NdTab<N1>) + sizeof(p2m) * PPB * ((P.pass == 0 ? (one ? 1 : 2) : 3) * Np + 4 * NF);
  auto go = [&](auto kf, auto... args) {
    cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    kf<<<grid, PPB * Np / NPT, sm, s>>>(op, dp, args..., Ne);
    return (int)cudaGetLastError();
  };
  if (P.pass == 0)
    return one ? go(k_nd_grad_p<N1, PPB, NPT, true>, P.a, P.b, P.ddens, P.dens, P.wall, P.G[0], P.G[1], P.G[2])
               : go(k_nd_grad_p<N1, PPB, NPT, false>, P.a, P.b, P.ddens, P.dens, P.wall, P.G[0], P.G[1], P.G[2]);
  const float2 *gx = P.G[0], *gy = P.G[1], *gz = P.G[2];
  return P.pass == 1 ? go(k_nd_div_p<N1, PPB, NPT, false>, gx, gy, gz, P.ddens, P.dens, P.wall, P.lh, P.lv, P.V)
                     : go(k_nd_div_p<N1, PPB, NPT, true>, gx, gy, gz, P.ddens, P.dens, P.wall, P.lh, P.lv, P.V);
}

int nd_pass_p(int N1, int nsm, const NdPass& P, const NdOpsP& op, const double* dp, int Ne, cudaStream_t s) {
  switch (N1) {
    case 2: return nd_pass_n<2, 1>(P, op, dp, Ne, s);
    case 3: return nd_pass_n<3, 1>(P, op, dp, Ne, s);
    case 4: return nd_pass_n<4, 1>(P, op, dp, Ne, s);
    case 5: return nd_pass_n<5, 1>(P, op, dp, Ne, s);
    case 6: return nd_pass_n<6, 1>(P, op, dp, Ne, s);
    case 7: return nd_pass_n<7, 1>(P, op, dp, Ne, s);
    case 8:
      // Two nodes per thread once the pairs are more than the SMs hold as three blocks of 512 threads.  Gradient +
      // divergence in us, one / two nodes: 20 pairs 16.8 / 21.5, 320 pairs 28.6 / 30.4, 640 pairs
      // 44.5 / 40.8, 1280 pairs 73 / 64.  At p = 3 one node is as good at 10,240 pairs (59) and better at 162 (13 / 20).
      return (Ne + 1) / 2 > 3 * nsm ? nd_pass_n<8, 2>(P, op, dp, Ne, s) : nd_pass_n<8, 1>(P, op, dp, Ne, s);
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace

// fedg_numdiff_apply_prec with prec == FEDG_PREC_PAIR; scratch = 5 Np*Ne doubles reused as pairs
int numdiff_apply_pair(fedg_ctx* c, double* const q[5], int nlap, double coef_h, double coef_v, double dt,
                       double* scratch) {
  const double sgn = ((nlap + 1) % 2 == 0) ? 1.0 : -1.0;
  const NdOpsP grad = nd_ops(c->op, {1.0, 1.0, 1.0}, true), lap = nd_ops(c->op, {1.0, 1.0, 1.0}, false),
               upd = nd_ops(c->op, {dt * (sgn * coef_h), dt * (sgn * coef_h), dt * (sgn * coef_v)}, false);
  const size_t n = c->n;
  float2* Gx = reinterpret_cast<float2*>(scratch);
  float2 *Gy = Gx + n, *Gz = Gy + n, *lh = Gz + n, *lv = lh + n;
  const int order[5] = {VRT, VMZ, VMX, VMY, VD};
  for (int vi = 0; vi < 5; ++vi) {
    const int var = order[vi];
    const int dw = var != VD, wall = var == VMZ;
    auto pass = [&](int kind, Src a, Src b, int dens, int wl, double* V) {
      const NdPass P{kind, a, b, q[VD], dens, wl, {Gx, Gy, Gz}, lh, lv, V};
      return tracked(c, FEDG_K_ND, [&] {
        return nd_pass_p(c->N1, c->op.nsm, P, kind == 0 ? grad : (kind == 1 ? lap : upd), c->d_prof, c->Ne, c->stream);
      });
    };
    const Src qv{q[var], nullptr}, L0{nullptr, lh}, L1{nullptr, lv};
    int r = pass(0, qv, qv, dw, wall, nullptr);
    for (int it = 1; it < nlap && !r; ++it) {
      r = pass(1, Src{}, Src{}, 0, wall, nullptr);
      if (!r) r = pass(0, L0, L1, 0, 0, nullptr);
    }
    if (!r) r = pass(2, Src{}, Src{}, dw, wall, q[var]);
    if (r) return api_cuda_fail((cudaError_t)r, "fedg_numdiff_apply (pair)");
  }
  return 0;
}

}  // namespace fedg
