// fedg_viseries.cu -- HEVI column Newton solve of the float-pair mode by a fixed-point series, a warp
// per two columns.
//
// Same problem, residual and convergence test as k_vi_cols (fedg_vicol.cu; FElib's cal_vi,
// scale_atm_dyn_dgm_nonhydro3d_rhot_hevi.F90:772-965, hevi_common_2.F90): Q - q* - impl_fac A(Q) = 0 for
// the vertical operator A with the Rusanov speed frozen at var0, accepted only on the float-pair
// residual.  What differs is how a correction J delta = b, J = I + K, is solved: on elements about as tall as
// wide, whose step the explicit horizontal terms set, ||K|| is well below one (about 0.26 on the
// 128x128x16 p = 7 mesh at dt 0.005 s), and the fixed point x <- (1 - w) x + w (b - K x) reaches FP32
// accuracy in about ten products K x, none of which needs the block-Thomas history, the element LU or
// its shuffles.  w = 1 / (1 + d), d the face dissipation's diagonal entry: K's spectrum is the
// dissipation's [0, 2 d] plus an almost imaginary acoustic part, and w centres it.  On flat elements d grows; above
// vi_courant_max the kernel is not launched.  A warp whose iteration does not contract, or whose Newton does not
// converge within the caller's limit, leaves a mark in `status`; k_vi_cols, launched after this kernel, solves the
// marked columns by block LU from the start.  From the second correction on such a warp has stored outputs already
// (`emitted`); block LU overwrites them, and no output overlaps an input.
//
// MOMX/MOMY: E = Q - q* is a combination of the two interface jumps of each element,
// E_ek = -beta_ek J_e + tau_ek J_{e+1}, and the jumps solve a scalar tridiagonal system with the jumps
// of q* on the right (see k_vi_cols): one Thomas sweep in float pairs per component, no iteration.
//
// Layout: a warp per pair of columns (i, i + 1), in the packed pair arithmetic of fedg_p2.cuh, all
// elements of the pair at once: lane l owns the nodes l, l + 32, ... of the NeZ*N1 levels.  Every sweep and
// every residual is then one or two passes over independent nodes instead of a walk along the column.  Shared
// memory (128 bytes per level) holds the iterate's float pairs and x with the products the derivative along
// z is taken of, in two copies (a sweep reads one and writes the other); b and the Jacobian's level
// quantities (48 bytes), which only their own lane reads, are there too or, for tall columns, in global
// scratch that stays in L2 and is discarded from it at the end.  The warps of a block hold neighbouring pairs,
// which share the sectors of their global accesses.
//
// What bounds it (p = 7, 32x32x8 elements, 715 us per launch): the load/store path at 71 % -- half of its
// wavefronts are the broadcast reads of the derivative, half the global accesses, where each lane's level is
// on a line of its own -- with the issue slots at 50 % and the FMA pipe at 42 %.  With b and the Jacobian in global
// scratch (32x32x16, 1381 us) 69, 41 and 39 %, and the load latency with three blocks per SM.  A walk along the columns
// (one lane per node of an element, the element loop serial) took 760 us there and 100 instead of 24 us
// for 8x8x8 elements of p = 3, where it is one warp's dependent chain.
#include <algorithm>

#include "fedg_ctx.cuh"
#include "fedg_mixed.cuh"
#include "fedg_p2.cuh"

namespace fedg {
namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr u64x SG = 0x8000000080000000ull;  // both sign bits
constexpr float SWEEP_RATE = 0.55f;  // of the sweeps' envelope

// shared memory of one pair (bytes)
struct SLayout {
  int oB, oX, oA, stride;  // P at 0; b and the Jacobian at oB unless glb; x copies at oX and oX + 40 L
  __host__ __device__ SLayout(int N1, int NeZ, bool glb) {
    const int L = N1 * NeZ;
    oB = 48 * L;
    oX = oB + (glb ? 0 : 48 * L);
    oA = oX + 80 * L;
    stride = (oA + 8 * (NeZ + 1) + 15) / 16 * 16;
  }
};

// bytes of one pair's global scratch (glb): b and the Jacobian's level quantities, whole 128-byte lines
__host__ __device__ inline size_t pair_scratch(int L) { return ((size_t)48 * L + 127) / 128 * 128; }

struct SerArgs {
  MixViArgs v;
  // as pairs, impl_fac multiplied in: E33 D, FSz/2 times the Lift, and grav times VPOrdM1 in the form
  // I - tv tw^T (it removes one mode)
  float2 cD[FEDG_MAXN1 * FEDG_MAXN1], cLb[FEDG_MAXN1], cLt[FEDG_MAXN1], tv[FEDG_MAXN1], tw[FEDG_MAXN1], cg;
  float c1, c2;                             // weights of MOMZ and RHOT in the sweep's change
  float dmin;                               // smallest DENS_hyd of the column (residual scale)
};

__device__ __forceinline__ unsigned long long l2_evict_first() {
  unsigned long long p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ p2 ld_pair(const float2* a) {  // two nodes
  const float4 v = __ldg(reinterpret_cast<const float4*>(a));
  return {pk(v.x, v.z), pk(v.y, v.w)};
}
__device__ __forceinline__ void st_once(float2* a, p2 v, unsigned long long pol) {
  const float2 h = unpk(v.h), l = unpk(v.l);
  asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(a), "f"(h.x), "f"(l.x), "f"(h.y),
               "f"(l.y), "l"(pol)
               : "memory");
}
__device__ __noinline__ f2 dev_pow(float rh, float rl, double kap64) {
  return f2_split(pow(1.0 + ((double)rh + (double)rl), kap64) - 1.0);
}
__device__ __forceinline__ float warp_max_bits(float e) {  // e >= 0 or NaN (which wins)
  return __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(e) & 0x7fffffffu));
}
__device__ __forceinline__ p2 shfl(p2 v, int src) {
  return {__shfl_sync(FULL, v.h, src), __shfl_sync(FULL, v.l, src)};
}

// Place of level n in the arrays that a warp reads element-wise (every lane the same node of its element,
// 32/N1 elements at once): the nodes of an element are permuted by an element-dependent XOR, so that the
// lanes' 16-byte reads fall on different banks.  place(n0, e) ^ m is the place of node m of element e.
template <int N1>
__device__ __forceinline__ int place(int n0, int e) {
  return n0 | (N1 == 8 ? (e & 7) : ((e >> 1) & 3));
}

// one pair's shared memory; n: level, i: its place
struct Pair {
  p2m* P;            // iterate [3][L], by place
  ulonglong2* B01;   // b of DENS and MOMZ [L]
  u64x* B2;          // b of RHOT [L]
  ulonglong2* J01;   // pot = RHOT/DENS, wt = MOMZ/DENS [L]
  u64x* J2;          // dpd = dP/dRHOT [L]
  unsigned char* X;  // two copies of x: (DENS, MOMZ) [L] and (dpd RHOT, heat flux) [L] by place, RHOT [L]
  u64x* A;           // wave speed of face e (0 .. NeZ)
  int NeZ, L, lane;
  __device__ ulonglong2* x01(int c) const { return reinterpret_cast<ulonglong2*>(X + c * 40 * L); }
  __device__ ulonglong2* xpt(int c) const { return x01(c) + L; }
  __device__ u64x* x2(int c) const { return reinterpret_cast<u64x*>(xpt(c) + L); }
  // x at level n, place i, into copy c, with its products p = dpd RHOT and t = pot (MOMZ - wt DENS) + wt RHOT
  __device__ void put(int c, int n, int i, ulonglong2 j, u64x j2, u64x r, u64x m, u64x h) const {
    x01(c)[i] = make_ulonglong2(r, m);
    xpt(c)[i] = make_ulonglong2(xmul(j2, h), xfma(j.x, xfma(j.y, r ^ SG, m), xmul(j.y, h)));
    x2(c)[n] = h;
  }
};

// FP32 rows of K for the lane's node k
template <int N1>
struct KRow {
  u64x D[N1], T[N1], fB, fT;
  __device__ __forceinline__ KRow(const Ops& op, double impl_fac, int k) {
    const float fi = (float)impl_fac, fd = (float)op.E33 * fi;
#pragma unroll
    for (int m = 0; m < N1; ++m) {
      D[m] = pk1(fd * (float)op.D[k * N1 + m]);
      T[m] = pk1(fi * (float)op.grav * (float)op.T[k * N1 + m]);
    }
    fB = pk1(0.5f * fi * (float)op.Lb[k] * (float)op.FSz);
    fT = pk1(0.5f * fi * (float)op.Lt[k] * (float)op.FSz);
  }
};

// One sweep x <- (1 - w) x + w (b - K x) from copy c into the other one; returns the lane's largest
// weighted change.  (A NaN can drop out of the change; the certifying residual looks at every node.)
template <int N1>
__device__ __forceinline__ float sweep(const Pair& s, const KRow<N1>& K, int c, u64x w, u64x w1, float c1, float c2) {
  constexpr int N = N1 - 1;
  const ulonglong2 *x01 = s.x01(c), *xpt = s.xpt(c);
  const u64x* x2 = s.x2(c);
  float dmax = 0.f;
#pragma unroll 1
  for (int n = s.lane; n < s.L; n += 32) {
    const int e = n / N1, n0 = e * N1, p0 = place<N1>(n0, e);
    const ulonglong2 bb = s.B01[n], j = s.J01[n];  // from L2, while the derivatives are formed
    const u64x b2 = s.B2[n], j2 = s.J2[n];
    u64x y0 = 0, y1 = 0, y2 = 0, z1 = 0;
    ulonglong2 a0, b0, aN, bN;
#pragma unroll
    for (int m = 0; m < N1; ++m) {
      const ulonglong2 a = x01[p0 ^ m], b = xpt[p0 ^ m];
      y0 = xfma(K.D[m], a.y, y0);
      z1 = xfma(K.T[m], a.x, z1);
      y1 = xfma(K.D[m], b.x, y1);
      y2 = xfma(K.D[m], b.y, y2);
      if (m == 0) { a0 = a; b0 = b; }
      if (m == N) { aN = a; bN = b; }
    }
    {  // bottom face (nz = -1); a slip lid reflects MOMZ and the heat flux
      u64x dr = 0, dm, dp = 0, dt, dh = 0;
      if (e > 0) {
        const int i = place<N1>(n0 - N1, e - 1) ^ N;
        const ulonglong2 a = x01[i], b = xpt[i];
        dr = xsub(a0.x, a.x); dm = xsub(a0.y, a.y); dp = xsub(b0.x, b.x); dt = xsub(b0.y, b.y);
        dh = xsub(x2[n0], x2[n0 - 1]);
      } else {
        dm = xadd(a0.y, a0.y);
        dt = xadd(b0.y, b0.y);
      }
      const u64x al = s.A[e];
      y0 = xfma(K.fB, xfma(al, dr, dm), y0);
      y1 = xfma(K.fB, xfma(al, dm, dp), y1);
      y2 = xfma(K.fB, xfma(al, dh, dt), y2);
    }
    {  // top face (nz = +1)
      u64x dr = 0, dm, dp = 0, dt, dh = 0;
      if (e + 1 < s.NeZ) {
        const int i = place<N1>(n0 + N1, e + 1);
        const ulonglong2 a = x01[i], b = xpt[i];
        dr = xsub(aN.x, a.x); dm = xsub(a.y, aN.y); dp = xsub(b.x, bN.x); dt = xsub(b.y, bN.y);
        dh = xsub(x2[n0 + N], x2[n0 + N1]);
      } else {
        dm = xadd(aN.y, aN.y) ^ SG;
        dt = xadd(bN.y, bN.y) ^ SG;
      }
      const u64x al = s.A[e + 1];
      y0 = xfma(K.fT, xfma(al, dr, dm), y0);
      y1 = xfma(K.fT, xfma(al, dm ^ SG, dp), y1);
      y2 = xfma(K.fT, xfma(al, dh, dt), y2);
    }
    const int i = p0 ^ (n - n0);
    const ulonglong2 o = x01[i];
    const u64x oh = x2[n];
    const u64x nr = xfma(w, xsub(bb.x, y0), xmul(w1, o.x));
    const u64x nm = xfma(w, xsub(bb.y, xadd(y1, z1)), xmul(w1, o.y));
    const u64x nh = xfma(w, xsub(b2, y2), xmul(w1, oh));
    s.put(1 - c, n, i, j, j2, nr, nm, nh);
    const float2 da = unpk(xsub(nr, o.x)), db = unpk(xsub(nm, o.y)), dd = unpk(xsub(nh, oh));
    const float ma = fmaxf(fmaxf(fabsf(da.x), c1 * fabsf(db.x)), c2 * fabsf(dd.x));
    const float mb = fmaxf(fmaxf(fabsf(da.y), c1 * fabsf(db.y)), c2 * fabsf(dd.y));
    dmax = fmaxf(dmax, fmaxf(ma, mb));
  }
  __syncwarp();
  return dmax;
}

// The certifying residual b = impl_fac A(P) + q* - P in float pairs (col_residual of fedg_vicol.cu) of P + x
// (x in copy c), which becomes the iterate; the two copies of x are scratch.  errA, errB: the two columns'
// max |b| / scale (NaN if not finite).  emit: the outputs are stored too, for the case that this residual
// is accepted (they are stored again otherwise).
template <int N1>
__device__ __forceinline__ void residual(const OpsX& ox, const SerArgs& args, const Pair& s, int c, const ProfX& px,
                                         const X5& qin, size_t gb, size_t gs, void* const* qsf, void* const* tout,
                                         unsigned long long once, bool emit, float& errA, float& errB) {
  constexpr int N = N1 - 1, NF = N1 * N1;
  const int k = s.lane % N1, L = s.L;
  const int gv[3] = {VD, VMZ, VRT};
  p2m* fm = reinterpret_cast<p2m*>(s.X + (1 - c) * 40 * L);  // pressure deviation [L]
  p2m* fr = fm + L;                                          // heat flux [L]
  p2m* del = reinterpret_cast<p2m*>(s.X + c * 40 * L);       // face fluxes [NeZ][2][3]
  for (int n = s.lane; n < L; n += 32) {
    const int i = place<N1>(n - k, n / N1) ^ k;
    const ulonglong2 x = s.x01(c)[i];
    const p2 Pd = p2_add_x(ld(s.P[i]), x.x), Pm = p2_add_x(ld(s.P[L + i]), x.y), Pr = p2_add_x(ld(s.P[2 * L + i]), s.x2(c)[n]);
    st(s.P[i], Pd);
    st(s.P[L + i], Pm);
    st(s.P[2 * L + i], Pr);
    const p2 dens = p2_dup(__ldg(px.dh + n)) + Pd;
    const p2 rhot = p2_dup(__ldg(px.rh + n)) + Pr;
    const p2 pot = rhot * p2_recip(dens);
    const p2 rr = Pr * p2_dup(__ldg(px.rhinv + n));
    u64x tl = pk1(ox.cb[11]);
#pragma unroll
    for (int m = 10; m >= 1; --m) tl = xfma(tl, rr.h, pk1(ox.cb[m]));
    p2 S = p2_add_x(p2_dup(ox.kap) * rr, xmul(xmul(rr.h, rr.h), tl));
    const float2 rh = unpk(rr.h);
    if (!(fabsf(rh.x) <= ox.rmax && fabsf(rh.y) <= ox.rmax)) {
      const float2 rl = unpk(rr.l);
      f2 a = p2_a(S), b = p2_b(S);
      if (!(fabsf(rh.x) <= ox.rmax)) a = dev_pow(rh.x, rl.x, ox.kap64);
      if (!(fabsf(rh.y) <= ox.rmax)) b = dev_pow(rh.y, rl.y, ox.kap64);
      S = p2_of(a, b);
    }
    st(fm[i], p2_dup(__ldg(px.ph + n)) * S);
    st(fr[i], pot * Pm);
  }
  __syncwarp();
  // vertical-face fluxes of every element: a lane per (element, side, variable)
  for (int t = s.lane; t < 6 * s.NeZ; t += 32) {
    const int e = t / 6, r = t - 6 * e, sd = r / 3, v = r - 3 * sd;
    const bool lid = sd == 0 ? (e == 0) : (e == s.NeZ - 1);
    const int nM = place<N1>(e * N1, e) ^ (sd == 0 ? 0 : N);
    const int eP = sd == 0 ? e - 1 : e + 1, nP = lid ? nM : place<N1>(eP * N1, eP) ^ (sd == 0 ? N : 0);
    const u64x al = s.A[e + sd];
    // v = 0: MOMZ jump (flux) and DDENS jump; 1: pressure and MOMZ; 2: heat flux and RHOT.  A slip lid
    // reflects MOMZ and the heat flux and leaves the rest without a jump
    const p2m* qf = v == 0 ? s.P + L : (v == 1 ? fm : fr);
    const p2m* qd = s.P + (v == 0 ? 0 : (v == 1 ? L : 2 * L));
    const p2 fM = ld(qf[nM]), dM = ld(qd[nM]);
    p2 fP = ld(qf[nP]), dP = ld(qd[nP]);
    if (lid) {
      if (v != 1) fP = p2_neg(fP);
      else dP = p2_neg(dP);
    }
    const p2 f = sd == 0 ? fM - fP : fP - fM;
    st(del[t], f - p2_mul_x(dP - dM, al));
  }
  __syncwarp();
  p2 Dk[N1];
#pragma unroll
  for (int m = 0; m < N1; ++m) Dk[m] = p2_dup(args.cD[k * N1 + m]);
  const p2 lbk = p2_dup(args.cLb[k]), ltk = p2_dup(args.cLt[k]);
  const p2 tv = p2_neg(p2_dup(args.tv[k])), tw = p2_dup(args.tw[k]);
  const p2 cg = p2_dup(args.cg), iimpl = p2_dup(args.v.inv_impl2);
  const float cref = (float)args.v.cref;
  errA = errB = 0.f;
  bool badA = false, badB = false;
  for (int nb = 0; nb < L; nb += 32) {  // every lane takes part in the shuffles of the last, partly empty pass
    const int n = nb + s.lane < L ? nb + s.lane : nb + k, n0 = n - k, e = n0 / N1;
    const int p0 = place<N1>(n0, e), i = p0 ^ k;
    const bool act = nb + s.lane < L;
    const size_t g = gb + (size_t)e * gs + (size_t)NF * k;
    const p2 q0 = ld_pair(qin.v[VD] + g), q1 = ld_pair(qin.v[VMZ] + g), q2 = ld_pair(qin.v[VRT] + g);
    const p2 dd = ld(s.P[i]);
    p2 mode = tw * dd;  // the mode that VPOrdM1 removes: summed over the element's nodes
#pragma unroll
    for (int o = N1 / 2; o > 0; o >>= 1)
      mode = mode + p2{__shfl_xor_sync(FULL, mode.h, o), __shfl_xor_sync(FULL, mode.l, o)};
    p2acc sd, sm, sr;
#pragma unroll
    for (int m = 0; m < N1; ++m) {
      sd.add(Dk[m], ld(s.P[L + (p0 ^ m)]));
      sm.add(Dk[m], ld(fm[p0 ^ m]));
      sr.add(Dk[m], ld(fr[p0 ^ m]));
    }
    const p2m* d = del + 6 * e;
    sm.add(cg, dd);
    sm.add(tv, mode);
    sd.add(lbk, ld(d[0]));
    sm.add(lbk, ld(d[1]));
    sr.add(lbk, ld(d[2]));
    sd.add(ltk, ld(d[3]));
    sm.add(ltk, ld(d[4]));
    sr.add(ltk, ld(d[5]));
    const float dhf = __ldg(px.dhf + n);
    const float isc[3] = {1.f / dhf, 1.f / (dhf * cref), 1.f / __ldg(px.rhf + n)};
    u64x b[3];
    auto row = [&](int v, p2 qs, p2 Pl, p2 A) {  // A holds -impl_fac A: b = (q* - P) - (-impl_fac A)
      const p2 x = (qs - Pl) - A;
      b[v] = xadd(x.h, x.l);
      const float2 f = unpk(b[v]);
      errA = fmaxf(errA, fabsf(f.x) * isc[v]);
      errB = fmaxf(errB, fabsf(f.y) * isc[v]);
      badA = badA || !(fabsf(f.x) < 3.0e38f);
      badB = badB || !(fabsf(f.y) < 3.0e38f);
      if (emit && act) {
        st_once(static_cast<float2*>(qsf[gv[v]]) + g, Pl, once);
        st_once(static_cast<float2*>(tout[gv[v]]) + g, (Pl - qs) * iimpl, once);
      }
    };
    row(0, q0, dd, sd.get());
    row(1, q1, ld(s.P[L + i]), sm.get());
    row(2, q2, ld(s.P[2 * L + i]), sr.get());
    if (act) {
      s.B01[n] = make_ulonglong2(b[0], b[1]);
      s.B2[n] = b[2];
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    errA = fmaxf(errA, __shfl_xor_sync(FULL, errA, o));
    errB = fmaxf(errB, __shfl_xor_sync(FULL, errB, o));
  }
  if (__any_sync(FULL, badA)) errA = __int_as_float(0x7fc00000);
  if (__any_sync(FULL, badB)) errB = __int_as_float(0x7fc00000);
}

template <int N1, bool GLB>
__global__ void __launch_bounds__(128, GLB ? 3 : 4)
    k_vi_series(const __grid_constant__ Ops op, const __grid_constant__ OpsX ox, const ProfX px, const X5 qin, const F5c z,
                const A3 a0, void* const* qsf, void* const* tout, float* gsc, int* status, unsigned long long* cnt,
                const __grid_constant__ SerArgs args, int ncol) {
  constexpr int N = N1 - 1, NF = N1 * N1, Np = NF * N1;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int cp = blockIdx.x * (blockDim.x >> 5) + wib, ncp = ncol / 2;
  if (cp >= ncp) return;  // no block barriers
  const int NeZ = op.NeZ, L = op.L, k = lane % N1;
  const SLayout lay(N1, NeZ, GLB);
  unsigned char* base = smraw + (size_t)wib * lay.stride;
  Pair s;
  s.P = reinterpret_cast<p2m*>(base);
  unsigned char* gl = GLB ? reinterpret_cast<unsigned char*>(gsc) + (size_t)cp * pair_scratch(L) : base + lay.oB;
  s.B01 = reinterpret_cast<ulonglong2*>(gl);
  s.J01 = s.B01 + L;
  s.B2 = reinterpret_cast<u64x*>(s.J01 + L);
  s.J2 = s.B2 + L;
  s.X = base + lay.oX;
  s.A = reinterpret_cast<u64x*>(base + lay.oA);
  s.NeZ = NeZ; s.L = L; s.lane = lane;
  const size_t gs = (size_t)op.NeX * op.NeY * Np;
  const size_t gb = (size_t)(2 * cp / NF) * Np + 2 * cp % NF;  // node (0, 0) of the first column
  const MixViArgs& va = args.v;
  const float kapf = ox.kap.x;
  const unsigned long long once = l2_evict_first();
  const int gv[3] = {VD, VMZ, VRT};

  // ---- the iterate P = var0, the first residual b = (q* - var0) + impl_fac A(var0) from the stage-1 kernel's
  // A(var0), the Jacobian's level quantities ----
  float bmax = 0.f;  // largest weighted |b|
  {
    const p2 impl = p2_dup(va.impl2);
#pragma unroll 1
    for (int n = lane; n < L; n += 32) {
      const size_t g = gb + (size_t)(n / N1) * gs + (size_t)NF * k;
      p2 P[3], q[3], a[3];
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        P[v] = p2_split(__ldg(z.v[gv[v]] + g), __ldg(z.v[gv[v]] + g + 1));
        q[v] = ld_pair(qin.v[gv[v]] + g);
        a[v] = ld_pair(a0.v[v] + g);
      }
      u64x b[3];
      float mx[3];
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        st(s.P[v * L + (place<N1>(n - k, n / N1) ^ k)], P[v]);
        const p2 x = (q[v] - P[v]) + impl * a[v];
        b[v] = xadd(x.h, x.l);
        mx[v] = fmaxf(fabsf(unpk(b[v]).x), fabsf(unpk(b[v]).y));
      }
      s.B01[n] = make_ulonglong2(b[0], b[1]);
      s.B2[n] = b[2];
      bmax = fmaxf(bmax, fmaxf(mx[0], fmaxf(args.c1 * mx[1], args.c2 * mx[2])));
      // pot = RHOT/DENS, wt = MOMZ/DENS, dpd = kappa PRES/RHOT (FP32, the correction's accuracy)
      const float2 d = unpk(P[0].h), m = unpk(P[1].h), x = unpk(P[2].h);
      const float dh = __ldg(px.dhf + n), rh = __ldg(px.rhf + n), pf = __ldg(px.phf + n), rt = __ldg(px.rthf + n);
      const float iA = __fdividef(1.f, dh + d.x), iB = __fdividef(1.f, dh + d.y);
      const float tA = rh + x.x, tB = rh + x.y;
      s.J01[n] = make_ulonglong2(pk(tA * iA, tB * iB), pk(m.x * iA, m.y * iB));
      s.J2[n] = pk(__fdividef(kapf * pf * __powf(1.f + x.x * rt, kapf), tA),
                   __fdividef(kapf * pf * __powf(1.f + x.y * rt, kapf), tB));
    }
    __syncwarp();
    // frozen wave speed |w| + c at the face nodes (hevi_common_2.F90:1149-1155), a lane per element and side
    u64x* sp = reinterpret_cast<u64x*>(s.X);  // [2 NeZ]
    for (int t = lane; t < 2 * NeZ; t += 32) {
      const int e = t >> 1, kf = (t & 1) ? N : 0, n = e * N1 + kf, i = place<N1>(e * N1, e) ^ kf;
      const float dh = __ldg(px.dhf + n), pf = __ldg(px.phf + n), rt = __ldg(px.rthf + n);
      const float2 d = unpk(s.P[i].h), m = unpk(s.P[L + i].h), x = unpk(s.P[2 * L + i].h);
      auto speed = [&](float dd0, float mz0, float dr0) {
        const float rdens0 = 1.f / (dh + dd0);
        const float wt0 = mz0 * rdens0;
        const float pres0 = pf * (1.f + expm1f(kapf * log1pf(dr0 * rt)));
        return fabsf(wt0) + sqrtf(kapf * pres0 * rdens0);
      };
      sp[t] = pk(speed(d.x, m.x, x.x), speed(d.y, m.y, x.y));
    }
    __syncwarp();
    for (int e = lane; e <= NeZ; e += 32) {
      const float2 lo = unpk(sp[e > 0 ? 2 * e - 1 : 0]), up = unpk(sp[e < NeZ ? 2 * e : 2 * NeZ - 1]);
      s.A[e] = pk(fmaxf(lo.x, up.x), fmaxf(lo.y, up.y));
    }
    __syncwarp();
  }

  // ---- DENS/MOMZ/RHOT Newton ----
  int nsolve = 0, stA = 0, stB = 0;
  bool give_up = false, emitted = false;
  {
    // relaxation: the face dissipation's diagonal entry with the wave speed of the lowest face
    const float2 af = unpk(s.A[0]);
    const float wr = 1.f / (1.f + 0.5f * (float)va.impl_fac * (float)op.Lb[0] * (float)op.FSz * fmaxf(af.x, af.y));
    const u64x w = pk1(wr), w1 = pk1(1.f - wr);
    const float ctol = 0.02f * (float)va.tol * args.dmin;
    while (true) {
      // Sweeps from x = w b until the change that the next one would make (the last change times the
      // observed contraction) is below 2e-6 of the first one, which FP32 resolves to 1e-7 (a later
      // correction goes on from the pair residual), or 2 % of the tolerance, so that what is accepted lies
      // well inside, as after the LU kernel's corrections.  The change falls in beats (K's spectrum is complex), so it
      // is held against a geometric envelope: what falls slower is left to the LU kernel, unless it is FP32's floor.
      int c = 0;
      bool ok = false;
      {
        const KRow<N1> K(op, va.impl_fac, k);
        for (int n = lane; n < L; n += 32) {
          const ulonglong2 b = s.B01[n];
          s.put(0, n, place<N1>(n - k, n / N1) ^ k, s.J01[n], s.J2[n], xmul(w, b.x), xmul(w, b.y), xmul(w, s.B2[n]));
        }
        __syncwarp();
        const float d0 = wr * warp_max_bits(bmax), stop = fmaxf(2.0e-6f * d0, ctol);
        float prev = d0, env = 4.f * d0;
        for (int it = 0; it < 24; ++it) {
          const float d = warp_max_bits(sweep<N1>(s, K, c, w, w1, args.c1, args.c2));
          c = 1 - c;
          const float r = __fdividef(d, prev);
          env *= SWEEP_RATE;
          if (d * r <= stop || (!(r <= 0.8f) && d <= 1.0e-4f * d0)) { ok = true; break; }
          if (!(d <= env)) break;
          prev = d;
        }
      }
      if (!ok) { give_up = true; break; }
      ++nsolve;
      emitted = nsolve >= 2;
      float eA, eB;
      residual<N1>(ox, args, s, c, px, qin, gb, gs, qsf, tout, once, emitted, eA, eB);
      bmax = fmaxf(eA, eB) * args.dmin;
      if (!stA && (double)eA <= va.tol) stA = nsolve;
      if (!stB && (double)eB <= va.tol) stB = nsolve;
      if ((double)eA <= va.tol && (double)eB <= va.tol) break;  // warp-uniform
      if (nsolve >= va.max_iter || eA != eA || eB != eB) { give_up = true; break; }
      __syncwarp();
    }
  }
  if (GLB) {  // the scratch lines are dead: drop them from L2 without a write-back
    __syncwarp();
    for (int t = lane; t < (int)(pair_scratch(L) / 128); t += 32)
      asm volatile("discard.global.L2 [%0], 128;" ::"l"(gl + 128 * t) : "memory");
  }
  if (give_up) {  // block LU for these columns, by the kernel that follows
    if (lane == 0) status[2 * cp] = status[2 * cp + 1] = VI_REDO;
    return;
  }
  // ---- DENS/MOMZ/RHOT out, if the accepted residual did not store it ----
  if (!emitted) {
    const p2 iimpl = p2_dup(va.inv_impl2);
    for (int n = lane; n < L; n += 32) {
      const size_t g = gb + (size_t)(n / N1) * gs + (size_t)NF * k;
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        const p2 q = ld_pair(qin.v[gv[v]] + g), p = ld(s.P[v * L + (place<N1>(n - k, n / N1) ^ k)]);
        st_once(static_cast<float2*>(qsf[gv[v]]) + g, p, once);
        st_once(static_cast<float2*>(tout[gv[v]]) + g, (p - q) * iimpl, once);
      }
    }
  }
  // ---- MOMX/MOMY: the interface jumps J_e (e = 1 .. NeZ - 1; zero at the lids) ----
  //   (1 + beta_e0 + tau_{e-1,N}) J_e - tau_e0 J_{e+1} - beta_{e-1,N} J_{e-1} = q*(e, 0) - q*(e-1, N)
  // beta_ek = cLb[k] A_e, tau_ek = cLt[k] A_{e+1}
  __syncwarp();
  p2m* Jm = reinterpret_cast<p2m*>(s.X);  // [2][NeZ + 1]
  const p2 diag = p2_dup(args.cLb[0]) + p2_dup(args.cLt[N]);
  const p2 lo = p2_dup(args.cLb[N]), up = p2_dup(args.cLt[0]);
  const p2 one = p2_dup(f2{1.f, 0.f});
  if (NeZ <= 16) {
    // cyclic reduction: half-warp m has component m, its lane i the row e = i + 1 (rows beyond NeZ - 1 are
    // the identity); a row is scaled to a unit diagonal and takes its neighbours at distance d out
    const int m = lane >> 4, e = (lane & 15) + 1;
    const bool row = e < NeZ;
    p2 a = p2_zero(), b = one, c = p2_zero(), r = p2_zero();
    if (row) {
      r = ld_pair(qin.v[VMX + m] + gb + (size_t)e * gs) - ld_pair(qin.v[VMX + m] + gb + (size_t)(e - 1) * gs + (size_t)NF * N);
      a = e > 1 ? p2_mul_x(lo, s.A[e - 1]) : p2_zero();  // minus the entries left and right of the diagonal
      c = e < NeZ - 1 ? p2_mul_x(up, s.A[e + 1]) : p2_zero();
      b = one + p2_mul_x(diag, s.A[e]);
    }
#pragma unroll 1
    for (int d = 1; d < NeZ; d *= 2) {
      const p2 ib = p2_recip(b);
      a = a * ib; c = c * ib; r = r * ib;
      const int i = lane & 15, h = lane & 16;
      const bool lf = i - d >= 0, rt = i + d < 16;
      const int sl = h + (lf ? i - d : i), sr = h + (rt ? i + d : i);
      const p2 al = shfl(a, sl), cl = shfl(c, sl), rl = shfl(r, sl);
      const p2 ar = shfl(a, sr), cr = shfl(c, sr), rr = shfl(r, sr);
      // J_e = r + a J_{e-d} + c J_{e+d}, J_{e-d} = rl + al J_{e-2d} + cl J_e, ...
      const p2 a0_ = lf ? a : p2_zero(), c0_ = rt ? c : p2_zero();
      b = (one - a0_ * cl) - c0_ * ar;
      r = (r + a0_ * rl) + c0_ * rr;
      a = a0_ * al;
      c = c0_ * cr;
    }
    r = r * p2_recip(b);
    if (e <= NeZ) st(Jm[m * (NeZ + 1) + e], row ? r : p2_zero());
    if ((lane & 15) == 0) st(Jm[m * (NeZ + 1)], p2_zero());
    __syncwarp();
  } else {  // a Thomas sweep per component
    p2m* Cp = Jm + 2 * (NeZ + 1);  // [NeZ + 1]
    for (int t = lane; t < 2 * (NeZ + 1); t += 32) {
      const int m = t & 1, e = t >> 1;
      p2 j = p2_zero();
      if (e > 0 && e < NeZ)
        j = ld_pair(qin.v[VMX + m] + gb + (size_t)e * gs) - ld_pair(qin.v[VMX + m] + gb + (size_t)(e - 1) * gs + (size_t)NF * N);
      st(Jm[m * (NeZ + 1) + e], j);
    }
    __syncwarp();
    if (lane < 2) {
      p2m* J = Jm + lane * (NeZ + 1);
      p2 cprev = p2_zero(), rprev = p2_zero();
      for (int e = 1; e < NeZ; ++e) {
        const p2 l = p2_mul_x(lo, e > 1 ? s.A[e - 1] : 0ull);
        const p2 ip = p2_recip((one + p2_mul_x(diag, s.A[e])) - l * cprev);
        cprev = p2_mul_x(up, e < NeZ - 1 ? s.A[e + 1] : 0ull) * ip;
        rprev = (ld(J[e]) + l * rprev) * ip;
        st(J[e], rprev);
        if (lane == 0) st(Cp[e], cprev);
      }
    }
    __syncwarp();
    if (lane < 2) {
      p2m* J = Jm + lane * (NeZ + 1);
      p2 x = p2_zero();
      for (int e = NeZ - 1; e >= 1; --e) {
        x = ld(J[e]) + ld(Cp[e]) * x;
        st(J[e], x);
      }
    }
    __syncwarp();
  }
  {
    const p2 iimpl = p2_dup(va.inv_impl2);
    const p2 U = p2_dup(ox.Uref), V = p2_dup(ox.Vref);
    const p2 lb = p2_dup(args.cLb[k]), lt = p2_dup(args.cLt[k]);
#pragma unroll 1
    for (int n = lane; n < L; n += 32) {
      const int e = n / N1;
      const size_t g = gb + (size_t)e * gs + (size_t)NF * k;
      const p2 be = p2_mul_x(lb, s.A[e]), ta = p2_mul_x(lt, s.A[e + 1]);
      const p2 dh = p2_dup(__ldg(px.dh + n));
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const p2m* J = Jm + m * (NeZ + 1) + e;
        const p2 q = ld_pair(qin.v[VMX + m] + g);
        const p2 E = ta * ld(J[1]) - be * ld(J[0]);
        st_once(static_cast<float2*>(qsf[VMX + m]) + g, (q - dh * (m == 0 ? U : V)) + E, once);
        st_once(static_cast<float2*>(tout[VMX + m]) + g, E * iimpl, once);
      }
    }
  }
  if (lane == 0) {
    status[2 * cp] = stA;
    status[2 * cp + 1] = stB;
    atomicAdd(cnt + 1, (unsigned long long)(stA + stB));
    atomicAdd(cnt + 2, 2ull);
  }
}

template <int N1, bool GLB>
int launch_n(const Ops& op, const OpsX& ox, const ProfX& px, const X5& qin, const F5c& z, const A3& a0,
             void* const* qsf, void* const* tout, float* gsc, int* status, unsigned long long* cnt, const SerArgs& a, cudaStream_t s) {
  if (vi_courant(op, a.v.impl_fac) > vi_courant_max(N1)) return -1;
  const SLayout lay(N1, op.NeZ, GLB);
  int wpb = 4;  // neighbouring pairs share 32-byte sectors; fewer where four would leave an SM one block
  while (wpb > 1 && (size_t)lay.stride * wpb > 113 * 1024) wpb /= 2;
  const size_t smem = (size_t)lay.stride * wpb;
  if (smem > 227 * 1024) return -1;
  const int ncol = op.NeX * op.NeY * N1 * N1, ncp = ncol / 2;
  auto kfn = k_vi_series<N1, GLB>;
  cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  kfn<<<(ncp + wpb - 1) / wpb, 32 * wpb, smem, s>>>(op, ox, px, qin, z, a0, qsf, tout, gsc, status, cnt, a, ncol);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_vi_series(int N1, const Ops& op, const OpsX& ox, const ProfX& px, const X5& qin, const F5c& z, const A3& a0,
                     void* const* qsf, void* const* tout, float* gsc, int* status, unsigned long long* cnt,
                     const MixViArgs& a, const float hyd[3], cudaStream_t s) {
  SerArgs sa;
  sa.v = a;
  auto split = [](double x) {
    const float h = (float)x;
    return make_float2(h, (float)(x - (double)h));
  };
  for (int i = 0; i < N1 * N1; ++i) sa.cD[i] = split(a.impl_fac * op.E33 * op.D[i]);
  // VPOrdM1 = I - R, R the projection on the highest mode, of rank one: R = R(:, 0) R(0, :) / R(0, 0)
  for (int k = 0; k < N1; ++k) {
    sa.cLb[k] = split(0.5 * a.impl_fac * op.FSz * op.Lb[k]);
    sa.cLt[k] = split(0.5 * a.impl_fac * op.FSz * op.Lt[k]);
    const double rk0 = (k == 0 ? 1.0 : 0.0) - op.T[k * N1], r0k = (k == 0 ? 1.0 : 0.0) - op.T[k];
    sa.tv[k] = split(a.impl_fac * op.grav * rk0 / (1.0 - op.T[0]));
    sa.tw[k] = split(r0k);
  }
  sa.cg = split(a.impl_fac * op.grav);
  sa.c1 = 1.f / (float)a.cref;
  sa.c2 = hyd[0] / hyd[1];
  sa.dmin = hyd[2];
  // All in shared memory as long as that leaves an SM three blocks of four warps (p = 7: NeZ <= 13).
  // Measured, p = 7, a step in ms with b and the Jacobian in shared memory / in global scratch: 32x32x8 elements
  // 3.44 / 3.56 (four blocks fit either way), 128x128x16 113 / 107 (two blocks against three).
  const bool glb = 3 * (4 * (size_t)SLayout(N1, op.NeZ, false).stride + 1024) > 228 * 1024;
#define FEDG_SER(n, g) return launch_n<n, g>(op, ox, px, qin, z, a0, qsf, tout, gsc, status, cnt, sa, s)
  if (N1 == 4) {
    if (glb) FEDG_SER(4, true);
    FEDG_SER(4, false);
  }
  if (N1 == 8) {
    if (glb) FEDG_SER(8, true);
    FEDG_SER(8, false);
  }
#undef FEDG_SER
  return (int)cudaErrorInvalidValue;
}

}  // namespace fedg
