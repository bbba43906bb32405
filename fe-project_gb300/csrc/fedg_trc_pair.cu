// fedg_trc_pair.cu -- the tracer step of fedg_trc_update in float pairs (FEDG_PREC_PAIR).
//
// Same algorithm as the FP64 kernels of fedg_trc.cu (FElib's trcadvect3d_heve.F90 FCT coefficient :234-306,
// cal_tend :149-231, TMAR :311-340, the tracer filter ..._dgm_modalfilter.F90:232-270 and
// rk_advance_trcvar_low_storage2D, scale_timeint_rk.F90:1390-1498), with every value carried as an
// unevaluated float pair (hi + lo, about 48 bits; fedg_f2.cuh):
//   - FP64 inputs are split with integer instructions on load; the stage fields stay pairs between
//     launches; the final QTRC is converted back to FP64;
//   - the face and element integrals are pair sums, the D_x/D_y/D_z contractions and the Lift are
//     compensated sums of exact products, divisions are pair reciprocals;
//   - sums of two or three FP64 inputs (densities, mass flux and Rusanov coefficient) are taken in FP64, whose
//     pipe is otherwise idle here, and split once.
// Why: the FP64 kernels keep GB300's FP64 pipe 77 % (coefficient) and 90 % (stage) busy at 30 and 64 to 84 FP64
// instructions per node and launch; the FP32 pipe has 64x its issue rate.  The pair path is FP64-class (relative rounding
// ~1e-14), not bit-identical: the reciprocal replaces FP64 division, and the FCT face selection
// 0.5 (R+ + R- - (R+ - R-) sign) is taken exactly as R- or R+.
//
// Layout: one thread carries the same node of two consecutive elements in the packed pair arithmetic of
// fedg_p2.cuh, and two nodes (k and k + N1/2) for even N1.  With the limiter, the coefficient kernel of a stage
// leaves the face fluxes and the sign of each face's integral for the stage kernel, which needs
// neither again.  q^n dens^n and varTmp = q^n dens^n / 3 (SSP-RK3) come from QTRC, which the last stage overwrites.
//
// What bounds it: issue slots and load latency together (p = 7: 52-64 % of the slots, FP32 pipe 31-54 %, ALU pipe with
// the integer splits 36-54 %).  Step of three stages with limiter, 32x32x16 elements, p = 7: 2.10 -> 1.23 ms
// (coefficient 185 -> 150 us, stages 460-557 -> 223-303 us) against one element and scalar pairs per thread, the face
// fluxes formed in both kernels.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "fedg_ctx.cuh"
#include "fedg_two.cuh"

namespace fedg {
namespace {

__device__ __forceinline__ f2 operator+(f2 a, f2 b) { return f2_add(a, b); }
__device__ __forceinline__ f2 operator*(f2 a, f2 b) { return f2_mul(a, b); }
__device__ __forceinline__ f2 zero2() { return f2{0.f, 0.f}; }

__device__ __forceinline__ f2 ldp(const float2* p, size_t g) { return f2_of(__ldg(p + g)); }
__device__ __forceinline__ f2 pos_part(f2 x) { return x.h > 0.f ? x : zero2(); }
__device__ __forceinline__ f2 clamp01(f2 x) {
  if (!(x.h > 0.f)) return zero2();
  if (x.h > 1.f || (x.h == 1.f && x.l > 0.f)) return f2{1.f, 0.f};
  return x;
}

struct TrcOpsP {
  float2 D[FEDG_MAXN1 * FEDG_MAXN1], Fh[FEDG_MAXN1 * FEDG_MAXN1], Fv[FEDG_MAXN1 * FEDG_MAXN1];  // [l][i]
  float2 w2[FEDG_MAXN1 * FEDG_MAXN1];  // w_a w_b
  float2 Lb[FEDG_MAXN1], Lt[FEDG_MAXN1], w[FEDG_MAXN1];
  float2 E[3];   // -Escale (= -Fscale)
  float2 J, JF[3];
  int NeX, NeY, NeZ;
};

struct InP {
  const double* Q64;   // stage input as FP64 (first stage: QTRC) ...
  const float2* Qp;    // ... or as pairs (later stages)
  const double* mf[3];
  const double* aM;
  const double* aP;
  const double* rhoq;
  const double* ddens;
  const double* ddens0;
  __device__ __forceinline__ p2 q(const size_t (&g)[2]) const {
    return Qp ? p2_of(__ldg(Qp + g[0]), __ldg(Qp + g[1])) : p2_split(__ldg(Q64 + g[0]), __ldg(Q64 + g[1]));
  }
};

struct StageP {
  int c_ssm1, c_ss;  // twice the stage's time fraction and the next one's
  float2 sig_ss, one_m_sig, gam_ss, sig_N1, rdt_fct;
  int first, last, filter, tmar, keep0;  // keep0: one_m_sig != 0
  float2* fct;     // per element (limiter)
  unsigned* sgn;   // per element: bit f set where face f's flux integral is negative (limiter)
  float2* nf;      // face fluxes (limiter)
  float2* q_out;
  const double* ddens_fin;
  double* qtrc;
};

// DENS_hyd + (1 - c) DDENS0 + c DDENS for c = h/2
__device__ __forceinline__ double stage_dens(double dh, double dd0, double dd, int h) {
  if (h == 1) return fma(0.5, dd - dd0, dh + dd0);
  return dh + (h ? dd : dd0);
}

// Rusanov flux 0.5 (q+ m+ + q- m- - alpha+ q+ + alpha- q-) of face node fi (face fi / NF) of both elements, m the
// mass flux along the outward normal
template <int N1>
__device__ __forceinline__ p2 face_flux_p(const TrcOpsP& op, const InP& in, const TwoIdx& x, int fi) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1;
  const int f = fi / NF, ab = fi - f * NF, dir = f >= 4 ? 2 : (f & 1 ? 0 : 1), up = f == 1 || f == 2 || f == 5;
  int iM, rM, iP, rP;
  two_face_node<N1>(dir, up, ab, iM, rM);
  two_face_node<N1>(dir, !up, ab, iP, rP);
  size_t gM[2], gP[2];
  double cM[2], cP[2];
#pragma unroll
  for (int m = 0; m < 2; ++m) {
    const int kn = two_nbr(op, x, m, dir, up);
    gM[m] = (size_t)x.e[m] * Np + rM * N1 + iM;
    gP[m] = kn < 0 ? gM[m] : (size_t)kn * Np + rP * N1 + iP;
    const double* mf = dir == 0 ? in.mf[0] : (dir == 1 ? in.mf[1] : in.mf[2]);
    const double mM = __ldg(mf + gM[m]), mP = __ldg(mf + gP[m]);
    const size_t fa = (size_t)x.e[m] * 6 * NF + fi;
    cM[m] = (up ? mM : -mM) + __ldg(in.aM + fa);
    cP[m] = (up != (kn < 0) ? mP : -mP) - __ldg(in.aP + fa);  // the exterior of a slip lid is reflected
  }
  return p2_scale(in.q(gP) * p2_split_n(cP[0], cP[1]) + in.q(gM) * p2_split_n(cM[0], cM[1]), pk1(0.5f));
}

__device__ __forceinline__ p2 shfl_xor(p2 v, int o) {
  return {__shfl_xor_sync(0xffffffffu, v.h, o), __shfl_xor_sync(0xffffffffu, v.l, o)};
}

// sums over the NT threads of each pair in a fixed order into the first C entries of red, 16 C + C (warps) or
// C (NT + 1) entries per pair, which the first warp (thread) of the pair writes: the caller synchronises.  Begins with a
// barrier.
template <int C, int NT, int PPB>
__device__ __forceinline__ void pair_sums(p2 (&v)[C], p2m* red, int p) {
  constexpr int NW = NT / 32;
  __syncthreads();
  if constexpr (NT % 32 == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = v[c] + shfl_xor(v[c], o);
    p2m* part = red + C;
    if constexpr (NW > 1) {
#pragma unroll
      for (int c = 0; c < C; ++c)
        if ((p & 31) == 0) st(part[c * NW + (p >> 5)], v[c]);
      __syncthreads();
      if (p < 32) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          v[c] = p < NW ? ld(part[c * NW + p]) : p2_zero();
#pragma unroll
          for (int o = NW / 2; o > 0; o >>= 1) v[c] = v[c] + shfl_xor(v[c], o);
        }
      }
    }
#pragma unroll
    for (int c = 0; c < C; ++c)
      if (p == 0) st(red[c], v[c]);
  } else {
    p2m* part = red + C;
#pragma unroll
    for (int c = 0; c < C; ++c) st(part[c * NT + p], v[c]);
    __syncthreads();
    if (PPB == 1 && NT >= 32) {
      if (p < 32) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          p2 s = ld(part[c * NT + p]);
          for (int q = p + 32; q < NT; q += 32) s = s + ld(part[c * NT + q]);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) s = s + shfl_xor(s, o);
          if (p == 0) st(red[c], s);
        }
      }
    } else if (p < C) {
      p2 s = p2_zero();
      for (int q = 0; q < NT; ++q) s = s + ld(part[p * NT + q]);
      st(red[p], s);
    }
  }
}

template <int N1>
struct FctTab {
  p2m w2[N1 * N1], w[N1];
};

// FCT coefficient of the lowest mode, the face fluxes and the signs of their integrals
// how many elements: MANY; FEW, at most a block per SM; SOLO, so few that a block takes one element, not two
enum TrcMesh { MANY, FEW, SOLO };

template <int N1, int PPB, int NPT, TrcMesh MESH>
__global__ void __launch_bounds__(PPB* N1* N1* N1 / NPT, two_minb(PPB * N1 * N1 * N1 / NPT, MESH != MANY ? 512 : 1536))
    k_trc_fct_p(const __grid_constant__ TrcOpsP op, const double* __restrict__ dens_prof, const InP in, const StageP sp, int Ne) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1, NT = Np / NPT, KH = N1 / NPT;
  extern __shared__ p2m smp[];
  FctTab<N1>& T = *reinterpret_cast<FctTab<N1>*>(smp);
  int pair;
  const TwoIdx x = two_idx<N1, PPB, NT, MESH == SOLO>(op, Ne, pair);
  p2m* sf = smp + sizeof(FctTab<N1>) / sizeof(p2m) + pair * (6 * NF + 8);
  p2m* out = sf + 6 * NF;
  p2m* red = smp + sizeof(FctTab<N1>) / sizeof(p2m) + PPB * (6 * NF + 8) + pair * (NT + 1);
  for (int c = threadIdx.x; c < NF; c += PPB * NT) {
    st(T.w2[c], p2_dup(op.w2[c]));
    if (c < N1) st(T.w[c], p2_dup(op.w[c]));
  }
  p2 v[1] = {p2_zero()};
  p2 m[NPT];
  if (x.valid) {
    for (int fi = x.p; fi < 6 * NF; fi += NT) {
      const p2 nf = face_flux_p<N1>(op, in, x, fi);
      st(sf[fi], nf);
      sp.nf[(size_t)x.e[0] * 6 * NF + fi] = f2_pack(p2_a(nf));
      if (x.both) sp.nf[(size_t)x.e[1] * 6 * NF + fi] = f2_pack(p2_b(nf));
    }
#pragma unroll
    for (int h = 0; h < NPT; ++h) {
      const size_t g[2] = {(size_t)x.e[0] * Np + x.p + h * NT, (size_t)x.e[1] * Np + x.p + h * NT};
      double d[2];
#pragma unroll
      for (int e = 0; e < 2; ++e)
        d[e] = stage_dens(__ldg(dens_prof + x.ez[e] * N1 + x.k + h * KH), __ldg(in.ddens0 + g[e]), __ldg(in.ddens + g[e]), sp.c_ssm1);
      m[h] = p2_split_n(d[0], d[1]) * in.q(g) * p2_dup(sp.rdt_fct);
      if (in.rhoq) m[h] = m[h] + p2_split(__ldg(in.rhoq + g[0]), __ldg(in.rhoq + g[1]));
    }
  }
  __syncthreads();
  if (x.valid) {
#pragma unroll
    for (int h = 0; h < NPT; ++h) v[0] = v[0] + (ld(T.w2[x.i + N1 * x.j]) * ld(T.w[x.k + h * KH])) * m[h];
  }
  pair_sums<1, NT, PPB>(v, red, x.p);
  if constexpr (NT >= 7 * 32) {  // a warp per face beside the first one, else a thread
    const int f = (x.p >> 5) - 1, lane = x.p & 31;
    if (f >= 0 && f < 6) {
      p2 s = p2_zero();
      for (int q = lane; q < NF; q += 32) s = s + ld(T.w2[q]) * ld(sf[f * NF + q]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s = s + shfl_xor(s, o);
      if (lane == 0) st(out[f], s);
    }
  } else {
    for (int f = x.p; f < 6 && x.valid; f += NT) {
      p2 s = p2_zero();
      for (int q = 0; q < NF; ++q) s = s + ld(T.w2[q]) * ld(sf[f * NF + q]);
      st(out[f], s);
    }
  }
  __syncthreads();
  if (x.p < (x.both ? 2 : (x.valid ? 1 : 0))) {  // one element of the pair each
    f2 net = zero2();
    unsigned sg = 0;
#pragma unroll
    for (int f = 0; f < 6; ++f) {
      const p2 o = ld(out[f]);
      const f2 s = x.p ? p2_b(o) : p2_a(o);
      net = net + pos_part(f2_of(op.JF[f >= 4 ? 2 : (f & 1 ? 0 : 1)]) * s);
      sg |= (unsigned)(signbit(s.h) != 0) << f;
    }
    net = f2_add_f(net, 1.0e-10f);
    const p2 sum = ld(red[0]);
    const f2 qe = f2_of(op.J) * (x.p ? p2_b(sum) : p2_a(sum));
    const int e = x.p ? x.e[1] : x.e[0];
    sp.fct[e] = f2_pack(clamp01(qe * f2_recip(net)));
    sp.sgn[e] = sg;
  }
}

template <int N1>
struct StageTab {
  p2m D[N1 * N1], Lb[N1], Lt[N1];
};
template <int N1>
struct LastTab {  // filter and TMAR, last stage
  p2m Fh[N1 * N1], Fv[N1 * N1], w2[N1 * N1], w[N1];
};

// one direction's contraction for the NPT nodes of a thread
template <int N1, int NPT>
__device__ __forceinline__ void contract(p2acc (&s)[NPT], const p2m* D, const p2m* u, int dir, int i, int j, int k) {
  constexpr int KH = N1 / NPT;
#pragma unroll
  for (int l = 0; l < N1; ++l) {
    p2 d, v;
    if (dir < 2) d = ld(D[l * N1 + (dir == 0 ? i : j)]);
    else v = ld(u[two_at<N1>(i, j + N1 * l)]);
#pragma unroll
    for (int h = 0; h < NPT; ++h) {
      const int kh = k + h * KH;
      if (dir < 2) v = ld(u[dir == 0 ? two_at<N1>(l, j + N1 * kh) : two_at<N1>(i, l + N1 * kh)]);
      else d = ld(D[l * N1 + kh]);
      s[h].add(d, v);
    }
  }
}

// tendency and Runge-Kutta stage; LIM: with the coefficient kernel's outputs
template <int N1, int PPB, int NPT, TrcMesh MESH, bool LIM, bool LAST>
__global__ void __launch_bounds__(PPB* N1* N1* N1 / NPT, two_minb(PPB * N1 * N1 * N1 / NPT, MESH != MANY ? 512 : 1280))
    k_trc_stage_p(const __grid_constant__ TrcOpsP op, const double* __restrict__ dens_prof, const InP in, const StageP sp, int Ne) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1, NT = Np / NPT, KH = N1 / NPT;
  extern __shared__ p2m smp[];
  StageTab<N1>& T = *reinterpret_cast<StageTab<N1>*>(smp);
  LastTab<N1>& TL = *reinterpret_cast<LastTab<N1>*>(smp + sizeof(StageTab<N1>) / sizeof(p2m));
  constexpr int NTAB = (sizeof(StageTab<N1>) + (LAST ? sizeof(LastTab<N1>) : 0)) / sizeof(p2m);
  int pair;
  const TwoIdx x = two_idx<N1, PPB, NT, MESH == SOLO>(op, Ne, pair);
  p2m* fl = smp + NTAB + pair * (3 * Np + 6 * NF);
  p2m* df = fl + 3 * Np;
  for (int c = threadIdx.x; c < NF; c += PPB * NT) {
    st(T.D[c], p2_dup(op.D[c]));
    if (c < N1) {
      st(T.Lb[c], p2_dup(op.Lb[c]));
      st(T.Lt[c], p2_dup(op.Lt[c]));
    }
    if (LAST) {
      st(TL.Fh[c], p2_dup(op.Fh[c]));
      st(TL.Fv[c], p2_dup(op.Fv[c]));
      st(TL.w2[c], p2_dup(op.w2[c]));
      if (c < N1) st(TL.w[c], p2_dup(op.w[c]));
    }
  }
  const size_t g0[2] = {(size_t)x.e[0] * Np + x.p, (size_t)x.e[1] * Np + x.p};
  p2 q[NPT];
  if (x.valid) {
#pragma unroll
    for (int h = 0; h < NPT; ++h) {
      const size_t g[2] = {g0[0] + h * NT, g0[1] + h * NT};
      q[h] = in.q(g);
      const int at = two_at<N1>(x.i, x.j + N1 * (x.k + h * KH));
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        const double* mf = d == 0 ? in.mf[0] : (d == 1 ? in.mf[1] : in.mf[2]);
        st(fl[d * Np + at], p2_split(__ldg(mf + g[0]), __ldg(mf + g[1])) * q[h]);
      }
    }
    if (LIM) {  // numflux R, R = R- on outflow faces, R+ on inflow faces
      const f2 ownA = ldp(sp.fct, x.e[0]), ownB = ldp(sp.fct, x.e[1]);
      const unsigned sgA = __ldg(sp.sgn + x.e[0]), sgB = __ldg(sp.sgn + x.e[1]);
      for (int fi = x.p; fi < 6 * NF; fi += NT) {
        const int f = fi / NF, dir = f >= 4 ? 2 : (f & 1 ? 0 : 1), up = f == 1 || f == 2 || f == 5;
        const int ka = two_nbr(op, x, 0, dir, up), kb = two_nbr(op, x, 1, dir, up);
        const f2 ra = (sgA >> f & 1) && ka >= 0 ? ldp(sp.fct, ka) : ownA, rb = (sgB >> f & 1) && kb >= 0 ? ldp(sp.fct, kb) : ownB;
        const p2 nf = p2_of(__ldg(sp.nf + (size_t)x.e[0] * 6 * NF + fi), __ldg(sp.nf + (size_t)x.e[1] * 6 * NF + fi));
        st(df[fi], nf * p2_of(ra, rb));
      }
    } else {
      for (int fi = x.p; fi < 6 * NF; fi += NT) st(df[fi], face_flux_p<N1>(op, in, x, fi));
    }
  }
  __syncthreads();
  if (x.valid) {  // numflux R - q- m-
    for (int fi = x.p; fi < 6 * NF; fi += NT) {
      const int f = fi / NF, dir = f >= 4 ? 2 : (f & 1 ? 0 : 1), up = f == 1 || f == 2 || f == 5;
      int iM, rM;
      two_face_node<N1>(dir, up, fi - f * NF, iM, rM);
      const p2 own = ld(fl[dir * Np + two_at<N1>(iM, rM)]), nf = ld(df[fi]);
      st(df[fi], up ? nf - own : nf + own);
    }
  }
  __syncthreads();

  p2 qn[NPT];
  double wgt[NPT][2];
  if (x.valid) {
    p2 t[NPT];
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {  // Escale (= Fscale) times (D F + Lift del_flux)
      const int fb = dir == 0 ? 3 : (dir == 1 ? 0 : 4), ft = dir == 0 ? 1 : (dir == 1 ? 2 : 5);
      p2acc s[NPT];
      contract<N1, NPT>(s, T.D, fl + dir * Np, dir, x.i, x.j, x.k);
#pragma unroll
      for (int h = 0; h < NPT; ++h) {
        const int kh = x.k + h * KH, rw = dir == 0 ? x.i : (dir == 1 ? x.j : kh);
        const int ab = dir == 0 ? x.j + N1 * kh : (dir == 1 ? x.i + N1 * kh : x.i + N1 * x.j);
        s[h].add(ld(T.Lb[rw]), ld(df[fb * NF + ab]));
        s[h].add(ld(T.Lt[rw]), ld(df[ft * NF + ab]));
        const p2 r = p2_dup(op.E[dir]) * s[h].get();
        t[h] = dir == 0 ? r : t[h] + r;
      }
    }
    // rk_advance_trcvar_low_storage in pairs
#pragma unroll
    for (int h = 0; h < NPT; ++h) {
      const size_t g[2] = {g0[0] + h * NT, g0[1] + h * NT};
      if (in.rhoq) t[h] = t[h] + p2_split(__ldg(in.rhoq + g[0]), __ldg(in.rhoq + g[1]));
      double d0[2], dm[2], ds[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double dh = __ldg(dens_prof + x.ez[e] * N1 + x.k + h * KH), dd0 = __ldg(in.ddens0 + g[e]), dd = __ldg(in.ddens + g[e]);
        d0[e] = dh + dd0;
        dm[e] = stage_dens(dh, dd0, dd, sp.c_ssm1);
        ds[e] = LAST ? dh + dd : stage_dens(dh, dd0, dd, sp.c_ss);
        wgt[h][e] = ds[e];
      }
      p2 r = p2_dup(sp.sig_ss) * (q[h] * p2_split_n(dm[0], dm[1])) + p2_dup(sp.gam_ss) * t[h];
      if (LAST || sp.keep0) {
        const p2 v0 = (sp.first ? q[h] : p2_split(sp.qtrc[g[0]], sp.qtrc[g[1]])) * p2_split_n(d0[0], d0[1]);
        r = r + p2_dup(LAST ? sp.sig_N1 : sp.one_m_sig) * v0;
      }
      qn[h] = r * p2_recip(p2_split_n(ds[0], ds[1]));
      if (!LAST) {
        sp.q_out[g[0]] = f2_pack(p2_a(qn[h]));
        if (x.both) sp.q_out[g[1]] = f2_pack(p2_b(qn[h]));
      }
    }
  }
  if constexpr (LAST) {  // tracer filter of dens q, TMAR, rescale (FP64 output)
    if (sp.filter) {
      p2m *a = fl, *b = fl + Np;  // the flux arrays are free after the contractions above
      p2 s[NPT];
      __syncthreads();
#pragma unroll
      for (int h = 0; h < NPT; ++h) s[h] = x.valid ? p2_split_n(wgt[h][0], wgt[h][1]) * qn[h] : p2_zero();
#pragma unroll
      for (int dir = 0; dir < 3; ++dir) {  // b, written for z, was last read before the barrier of the y pass
        p2m* u = dir == 1 ? a : b;
#pragma unroll
        for (int h = 0; h < NPT; ++h) st(u[two_at<N1>(x.i, x.j + N1 * (x.k + h * KH))], s[h]);
        __syncthreads();
        p2acc c[NPT];
        contract<N1, NPT>(c, dir == 2 ? TL.Fv : TL.Fh, u, dir, x.i, x.j, x.k);
#pragma unroll
        for (int h = 0; h < NPT; ++h) s[h] = c[h].get();
      }
#pragma unroll
      for (int h = 0; h < NPT; ++h)
        if (x.valid) qn[h] = s[h] * p2_recip(p2_split_n(wgt[h][0], wgt[h][1]));
    }
    if (sp.tmar) {
      p2 v[2] = {p2_zero(), p2_zero()}, qp[NPT];
#pragma unroll
      for (int h = 0; h < NPT; ++h) {
        if (!x.valid) continue;
        const p2 wd = (ld(TL.w2[x.i + N1 * x.j]) * ld(TL.w[x.k + h * KH])) * p2_split_n(wgt[h][0], wgt[h][1]);
        qp[h] = p2_of(pos_part(p2_a(qn[h])), pos_part(p2_b(qn[h])));
        v[0] = v[0] + wd * qn[h];
        v[1] = v[1] + wd * qp[h];
      }
      pair_sums<2, NT, PPB>(v, fl, x.p);  // over the flux arrays
      __syncthreads();
      const p2 J = p2_dup(op.J);
      const p2 r = (J * ld(fl[0])) * p2_recip(p2_add_x(J * ld(fl[1]), pk1(1.0e-32f)));
#pragma unroll
      for (int h = 0; h < NPT; ++h)
        if (x.valid) qn[h] = r * qp[h];
    }
    if (!x.valid) return;
#pragma unroll
    for (int h = 0; h < NPT; ++h) {
      const size_t g[2] = {g0[0] + h * NT, g0[1] + h * NT};
      if (sp.ddens_fin) {
        double df_[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) df_[e] = __ldg(dens_prof + x.ez[e] * N1 + x.k + h * KH) + __ldg(sp.ddens_fin + g[e]);
        qn[h] = p2_split_n(wgt[h][0], wgt[h][1]) * p2_recip(p2_split_n(df_[0], df_[1])) * qn[h];
      }
      const f2 a = p2_a(qn[h]), b = p2_b(qn[h]);
      sp.qtrc[g[0]] = (double)a.h + (double)a.l;
      if (x.both) sp.qtrc[g[1]] = (double)b.h + (double)b.l;
    }
  }
}

float2 hsplit(double x) {
  const float h = (float)x;
  return make_float2(h, (float)(x - (double)h));
}

// pairs of elements per block: 108 to 343 threads
template <int N1>
constexpr int ppb_t() { return N1 <= 4 ? (N1 == 2 ? 16 : (N1 == 3 ? 4 : 2)) : 1; }

template <int N1, int NPF, int NPS, TrcMesh MESH>
int launch_pair_n(bool fct, const TrcOpsP& op, const double* dp, const InP& in, const StageP& st, int Ne, cudaStream_t s) {
  constexpr int PPB = ppb_t<N1>(), Np = N1 * N1 * N1, NF = N1 * N1;
  const int grid = ((MESH == SOLO ? Ne : (Ne + 1) / 2) + PPB - 1) / PPB;
  auto go = [&](auto kf, int nt, size_t sm) {
    cudaFuncSetAttribute(kf, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    kf<<<grid, PPB * nt, sm, s>>>(op, dp, in, st, Ne);
    return (int)cudaGetLastError();
  };
  if (fct) return go(k_trc_fct_p<N1, PPB, NPF, MESH>, Np / NPF, sizeof(FctTab<N1>) + sizeof(p2m) * PPB * (6 * NF + 8 + Np / NPF + 1));
  const size_t sm = sizeof(StageTab<N1>) + (st.last ? sizeof(LastTab<N1>) : 0) + sizeof(p2m) * PPB * (3 * Np + 6 * NF);
  static_assert(3 * Np + 6 * NF >= 2 * (Np + 1), "the sums' workspace");
  if (st.fct)
    return st.last ? go(k_trc_stage_p<N1, PPB, NPS, MESH, true, true>, Np / NPS, sm)
                   : go(k_trc_stage_p<N1, PPB, NPS, MESH, true, false>, Np / NPS, sm);
  return st.last ? go(k_trc_stage_p<N1, PPB, NPS, MESH, false, true>, Np / NPS, sm)
                 : go(k_trc_stage_p<N1, PPB, NPS, MESH, false, false>, Np / NPS, sm);
}

int launch_pair(int N1, int nsm, bool fct, const TrcOpsP& op, const double* dp, const InP& in, const StageP& st, int Ne,
                cudaStream_t s) {
  // FEW: at most a block per SM, which gets the registers of one: coefficient kernel of 20 pairs at p = 7 8.0 us
  // against 9.0, of 162 pairs at p = 3 9.6 against 12.4.  More at p = 7: two nodes per thread in the stage (three
  // stages of 1280 pairs 151 us, one node 181; 320 pairs 71 either way); in the coefficient kernel only
  // from some thousand pairs on (a whole step with one node / two: 1280 pairs 257 / 266 us, 3072 542 / 542,
  // 4224 708 / 697, 8192 1284 / 1252).  SOLO: half the FP64 sums per SM; a step of 64 elements at p = 7 76.1 us with
  // pairs, 73.4 with single elements, of 125 and 150 the same either way.
  const bool few = (Ne + 1) / 2 <= nsm * (N1 == 4 ? ppb_t<4>() : 1);
#define FEDG_T(n, f, g, w) launch_pair_n<n, f, g, w>(fct, op, dp, in, st, Ne, s)
  switch (N1) {
    case 2: return FEDG_T(2, 1, 1, MANY);
    case 3: return FEDG_T(3, 1, 1, MANY);
    case 4: return few ? FEDG_T(4, 1, 1, FEW) : FEDG_T(4, 1, 1, MANY);
    case 5: return FEDG_T(5, 1, 1, MANY);
    case 6: return FEDG_T(6, 1, 1, MANY);
    case 7: return FEDG_T(7, 1, 1, MANY);
    case 8:
      if (2 * Ne <= nsm) return FEDG_T(8, 1, 1, SOLO);
      if (few) return FEDG_T(8, 1, 1, FEW);
      return (Ne + 1) / 2 <= 4096 ? FEDG_T(8, 1, 2, MANY) : FEDG_T(8, 2, 2, MANY);
  }
#undef FEDG_T
  return (int)cudaErrorInvalidValue;
}

}  // namespace

// the fused tracer step in float pairs (fedg_trc_update with opts->prec == FEDG_PREC_PAIR); buffers
// are the FP64 path's scratch reinterpreted as pairs
int trc_update_pair(fedg_ctx* c, double* QTRC, const double* const mflx[3], const double* aM, const double* aP,
                    const double* ddens_trc, const double* ddens0_trc, const double* ddens, const double* rhoq,
                    const fedg_trc_opts* o, double* scratch) {
  const Ops& d = c->op;
  TrcOpsP op;
  std::memset(&op, 0, sizeof(op));
  const int N1 = c->N1;
  std::vector<double> Fh(N1 * N1), Fv(N1 * N1);
  if (o->filter) {
    modal_filter_1d(N1 - 1, o->mf_etac_h, o->mf_alpha_h, o->mf_order_h, Fh.data());
    modal_filter_1d(N1 - 1, o->mf_etac_v, o->mf_alpha_v, o->mf_order_v, Fv.data());
  }
  for (int i = 0; i < N1; ++i) {
    for (int l = 0; l < N1; ++l) {
      op.D[l * N1 + i] = hsplit(d.D[i * N1 + l]);
      op.Fh[l * N1 + i] = hsplit(Fh[i * N1 + l]);
      op.Fv[l * N1 + i] = hsplit(Fv[i * N1 + l]);
      op.w2[l * N1 + i] = hsplit(d.w[l] * d.w[i]);
    }
    op.Lb[i] = hsplit(d.Lb[i]);
    op.Lt[i] = hsplit(d.Lt[i]);
    op.w[i] = hsplit(d.w[i]);
  }
  const double E[3] = {d.E11, d.E22, d.E33}, FS[3] = {d.FSx, d.FSy, d.FSz};
  for (int c = 0; c < 3; ++c) {
    op.E[c] = hsplit(-E[c]);
    op.JF[c] = hsplit(d.Jac * FS[c]);
  }
  op.J = hsplit(d.Jac);
  op.NeX = d.NeX;
  op.NeY = d.NeY;
  op.NeZ = d.NeZ;
  const size_t n = c->n;
  float2* bufA = reinterpret_cast<float2*>(scratch);
  float2* bufB = bufA + n;
  float2* nf = bufB + n;
  float2* fct = nf + std::max(2 * n, (size_t)6 * N1 * N1 * c->Ne);
  unsigned* sgn = reinterpret_cast<unsigned*>(fct + c->Ne);
  constexpr int ns = 3;  // ERK_SSP_3s3o (scale_timeint_rk_butcher_tab.F90:200-210)
  const double sig[4][3] = {{0, 0, 0}, {1, 0, 0}, {0.75, 0.25, 0}, {1.0 / 3.0, 0, 2.0 / 3.0}};
  const double gam[4][3] = {{0, 0, 0}, {1, 0, 0}, {0, 0.25, 0}, {0, 0, 2.0 / 3.0}};
  const int cn2[3] = {0, 2, 1};
  for (int step = 0; step < o->nsteps; ++step) {
    const float2* qsp = nullptr;
    for (int s = 1; s <= ns; ++s) {
      InP in{s == 1 ? QTRC : nullptr, qsp, {mflx[0], mflx[1], mflx[2]}, aM, aP, rhoq, ddens_trc, ddens0_trc};
      StageP st;
      std::memset(&st, 0, sizeof(st));
      // varTmp collects the last stage's terms of the earlier stages: here sig(3,1) q^n dens^n alone
      const double sig_ss = sig[s][s - 1], gam_ss = gam[s][s - 1];
      st.c_ssm1 = cn2[s - 1];
      st.c_ss = s < ns ? cn2[s] : 0;
      st.sig_ss = hsplit(sig_ss);
      st.one_m_sig = hsplit(1.0 - sig_ss);
      st.keep0 = sig_ss != 1.0;
      st.gam_ss = hsplit(o->dt * gam_ss);
      st.sig_N1 = hsplit(sig[ns][0]);
      st.rdt_fct = hsplit(sig_ss / (o->dt * gam_ss));
      st.first = s == 1;
      st.last = s == ns;
      st.filter = o->filter != 0;
      st.tmar = o->limiter && o->tmar;
      st.fct = o->limiter ? fct : nullptr;
      st.sgn = sgn;
      st.nf = nf;
      st.q_out = (s & 1) ? bufA : bufB;
      st.ddens_fin = ddens;
      st.qtrc = QTRC;
      int r = 0;
      if (o->limiter)
        r = tracked(c, FEDG_K_TRC_FCT, [&] { return launch_pair(N1, d.nsm, true, op, c->d_prof, in, st, c->Ne, c->stream); });
      if (!r)
        r = tracked(c, FEDG_K_TRC_TEND, [&] { return launch_pair(N1, d.nsm, false, op, c->d_prof, in, st, c->Ne, c->stream); });
      if (r) return api_cuda_fail((cudaError_t)r, "fedg_trc_update (pair)");
      qsp = st.q_out;
    }
  }
  return 0;
}

}  // namespace fedg
