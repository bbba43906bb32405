// fedg_viseries.cu -- HEVI column Newton solve of the float-pair mode by a fixed-point series, two
// columns per lane.
//
// Same problem, residual and convergence test as k_vi_cols (fedg_vicol.cu; FElib's cal_vi,
// scale_atm_dyn_dgm_nonhydro3d_rhot_hevi.F90:772-965, hevi_common_2.F90): Q - q* - impl_fac A(Q) = 0 for
// the vertical operator A with the Rusanov speed frozen at var0, accepted only on the float-pair
// residual.  What differs is how a correction J delta = b, J = I + K, is solved.  At the vertical
// Courant numbers the explicit horizontal terms allow, ||K|| is well below one (about 0.26 on the
// 128x128x16 p = 7 mesh at dt 0.005 s), and the fixed point x <- (1 - w) x + w (b - K x) reaches FP32
// accuracy in about ten products K x, none of which needs the block-Thomas history, the element LU or
// its shuffles.  w = 1 / (1 + d), d the face dissipation's diagonal entry: K's spectrum is the
// dissipation's [0, 2 d] plus an almost imaginary acoustic part, and w centres it.  A warp whose
// iteration does not contract, or whose Newton does not converge within the caller's limit, writes
// nothing but a mark in `status`; k_vi_cols, launched after this kernel, solves the marked columns by
// block LU from the start, so what it accepts or reports as failed is as before.
//
// MOMX/MOMY: E = Q - q* is a combination of the two interface jumps of each element,
// E_ek = -beta_ek J_e + tau_ek J_{e+1}, and the jumps solve a scalar tridiagonal system with the jumps
// of q* on the right (see k_vi_cols): one Thomas sweep in float pairs per component, no iteration.
//
// Layout: N1 lanes per pair of columns (i, i + 1), in the packed pair arithmetic of fedg_p2.cuh: 8
// columns per warp at p = 7 (one row of an element), 16 at p = 3.  Lane k owns node k of every element.
// x, b and the iterate are private to their lane; only the level quantities that the derivative along z
// needs go through a small exchange buffer per element.  The iterate's pairs and the Jacobian's three
// level quantities sit in global planes, L2-resident while the columns are in flight and discarded from
// L2 at the end; b and x are in shared memory.
//
// What bounds it: latency, at 8 warps per SM (shared memory; more columns in flight push the planes out
// of L2), with the FP32 pipe 30 % busy; of a warp's time the two residuals take 34 %, about eight sweeps
// 25 %, the streaming passes the rest.  Float-pair HEVI step against the LU kernel alone (both with the
// packed stage kernel): p = 7, 32x32x8 elements at dt 0.04 s 5.31 -> 3.54 ms, 128x128x16 at dt 0.005 s 170 ->
// 115 ms, p = 3, 8x8x8 0.307 -> 0.270 ms.  Two nodes of a column per lane (half the exchange's shared-memory
// traffic) needs twice the columns in flight and lost 6 % on 128x128x16.
#include <algorithm>

#include "fedg_ctx.cuh"
#include "fedg_mixed.cuh"
#include "fedg_p2.cuh"
#include "fedg_sweep.cuh"

namespace fedg {
namespace {

// shared memory of one column pair (bytes): two vectors [3][L], x and b (the residual adds x to the
// iterate, writes the new b over it and uses the old b's space for its ring of level quantities, then
// they change places); the sweep's exchange slots; the wave speed of every face.  The wave-speed pass and
// the MOMX/MOMY system use the vectors' space before and after.
struct SLayout {
  int oB, oE, oA, stride;
  __host__ __device__ SLayout(int N1, int NeZ) {
    const int L = N1 * NeZ;
    const int ring = 3 * 5 * 16 * N1 + 96;
    oB = 24 * L > ring ? 24 * L : ring;
    oE = 2 * oB;
    oA = oE + 2 * (32 * N1 + 16);
    int o = oA + 8 * (NeZ + 1);
    // the pairs of a half warp read 8 N1 consecutive bytes each: put them on different banks
    const int r = 8 * N1, m = 128;
    stride = ((o - r + m - 1) / m) * m + r;
  }
};

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
__device__ __forceinline__ double ld_once(const double* a, unsigned long long pol) {
  double v;
  asm("ld.global.nc.L2::cache_hint.f64 %0, [%1], %2;" : "=d"(v) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ p2 ld_once(const float2* a, unsigned long long pol) {  // two nodes
  float4 v;
  asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(a), "l"(pol));
  return {pk(v.x, v.z), pk(v.y, v.w)};
}
__device__ __forceinline__ p2 ld_pair(const float2* a) {
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
__device__ __forceinline__ float grp_max_nan(float e, int width) {
  for (int o = width / 2; o > 0; o >>= 1) {
    const float oe = __shfl_xor_sync(FULL, e, o);
    e = (e != e || oe != oe) ? __int_as_float(0x7fc00000) : fmaxf(e, oe);
  }
  return e;
}
template <int N1>
struct Pair : SweepCtx<N1, N1> {
  p2m* P;         // iterate: planes of the three variables, indexed like J
  size_t gb, gs;  // node index of the first column's node (0, 0) and the element-layer stride
  __device__ size_t g(int e, int k) const { return gb + (size_t)e * gs + (size_t)(N1 * N1) * k; }
};

// The certifying residual b = impl_fac A(P) + q* - P in float pairs (col_residual of fedg_vicol.cu) of
// P + x, which becomes the iterate; b goes over x and the two vectors change places.  errA, errB: the two
// columns' max |b| / scale (NaN if not finite).  emit: the outputs are stored too, for the case that this
// residual is accepted (they are stored again otherwise).
template <int N1>
__device__ __forceinline__ void residual(const OpsX& ox, const SerArgs& args, Pair<N1>& c, const ProfX& px,
                                         const X5& qin, void* const* qsf, void* const* tout, unsigned long long once,
                                         bool emit, float& errA, float& errB) {
  constexpr int N = N1 - 1;
  const int NeZ = c.NeZ, L = c.L;
  const float cref = (float)args.v.cref;
  p2m* r2 = reinterpret_cast<p2m*>(c.B);
  p2m* del = r2 + 3 * 5 * N1;
  auto ri = [](int s, int q, int m) { return (s * 5 + q) * N1 + m; };
  p2 Dk[N1], lbk, ltk, tv, tw;
  const int k = c.k;
#pragma unroll
  for (int m = 0; m < N1; ++m) Dk[m] = p2_dup(args.cD[k * N1 + m]);
  lbk = p2_dup(args.cLb[k]);
  ltk = p2_dup(args.cLt[k]);
  tv = p2_neg(p2_dup(args.tv[k]));
  tw = p2_dup(args.tw[k]);
  const p2 cg = p2_dup(args.cg), iimpl = p2_dup(args.v.inv_impl2);
  auto fill = [&](int e, int k, p2 Pd, p2 Pm, p2 Pr) {  // level quantities of node (e, k) into slot e % 3
    const int l = e * N1 + k, s = e % 3;
    const p2 dens = p2_dup(__ldg(px.dh + l)) + Pd;
    const p2 rhot = p2_dup(__ldg(px.rh + l)) + Pr;
    const p2 pot = rhot * p2_recip(dens);
    const p2 rr = Pr * p2_dup(__ldg(px.rhinv + l));
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
    st(r2[ri(s, 0, k)], Pm);
    st(r2[ri(s, 1, k)], Pd);
    st(r2[ri(s, 2, k)], p2_dup(__ldg(px.ph + l)) * S);
    st(r2[ri(s, 3, k)], pot * Pm);
    st(r2[ri(s, 4, k)], Pr);
  };
  errA = errB = 0.f;
  bool badA = false, badB = false;
  const int gv[3] = {VD, VMZ, VRT};
  p2 q[3], pn[3];  // q* of the element and the iterate of the element two ahead, loaded early
#pragma unroll
  for (int v = 0; v < 3; ++v) pn[v] = ld(c.P[c.pi(v, 0)]);
  for (int e = -2; e < NeZ; ++e) {
    if (e + 1 >= 0 && e + 1 < NeZ && e < 0) {
#pragma unroll
      for (int v = 0; v < 3; ++v) q[v] = ld_pair(qin.v[gv[v]] + c.g(0, c.k));
    }
    if (e >= 0) {
      const int sc = e % 3, sb = (e + 2) % 3, su = (e + 1) % 3;
      // vertical-face fluxes of element e: lanes over (side, variable)
      for (int t = c.k; t < 6; t += N1) {
        const int s = t / 3, v = t - 3 * s;
        const int nM = s == 0 ? 0 : N;
        const bool lid = s == 0 ? (e == 0) : (e == NeZ - 1);
        const int sP = lid ? sc : (s == 0 ? sb : su), nP = lid ? nM : (s == 0 ? N : 0);
        const u64x al = c.A[e + s];
        // v = 0: MOMZ jump (flux) and DDENS jump; 1: pressure and MOMZ; 2: heat flux and RHOT.  A slip
        // lid reflects MOMZ and the heat flux and leaves the rest without a jump
        const int qf = v == 0 ? 0 : (v == 1 ? 2 : 3), qd = v == 0 ? 1 : (v == 1 ? 0 : 4);
        const p2 fM = ld(r2[ri(sc, qf, nM)]), dM = ld(r2[ri(sc, qd, nM)]);
        p2 fP = ld(r2[ri(sP, qf, nP)]), dP = ld(r2[ri(sP, qd, nP)]);
        if (lid) {
          if (v != 1) fP = p2_neg(fP);
          else dP = p2_neg(dP);
        }
        const p2 f = s == 0 ? fM - fP : fP - fM;
        st(del[t], f - p2_mul_x(dP - dM, al));
      }
      __syncwarp();
      {
        const p2 dd = ld(r2[ri(sc, 1, c.k)]);
        p2 mode = tw * dd;  // the mode that VPOrdM1 removes: summed over the column's nodes
#pragma unroll
        for (int o = N1 / 2; o > 0; o >>= 1)
          mode = mode + p2{__shfl_xor_sync(FULL, mode.h, o), __shfl_xor_sync(FULL, mode.l, o)};
        p2acc sd, sm, sr;
#pragma unroll
        for (int m = 0; m < N1; ++m) {
          const p2 a = ld(r2[ri(sc, 0, m)]), b = ld(r2[ri(sc, 2, m)]), d = ld(r2[ri(sc, 3, m)]);
          sd.add(Dk[m], a);
          sm.add(Dk[m], b);
          sr.add(Dk[m], d);
        }
        const p2 d0 = ld(del[0]), d1 = ld(del[1]), d2 = ld(del[2]), d3 = ld(del[3]), d4 = ld(del[4]), d5 = ld(del[5]);
        sm.add(cg, dd);
        sm.add(tv, mode);
        sd.add(lbk, d0);
        sm.add(lbk, d1);
        sr.add(lbk, d2);
        sd.add(ltk, d3);
        sm.add(ltk, d4);
        sr.add(ltk, d5);
        const int l = e * N1 + c.k;
        const float dhf = __ldg(px.dhf + l);
        const float isc[3] = {1.f / dhf, 1.f / (dhf * cref), 1.f / __ldg(px.rhf + l)};
        auto row = [&](int v, p2 qs, p2 Pl, p2 A) {  // A holds -impl_fac A: b = (q* - P) - (-impl_fac A)
          const p2 x = (qs - Pl) - A;
          const u64x b = xadd(x.h, x.l);
          c.X[v * L + l] = b;
          if (emit) {
            const size_t g = c.g(e, c.k);
            st_once(static_cast<float2*>(qsf[gv[v]]) + g, Pl, once);
            st_once(static_cast<float2*>(tout[gv[v]]) + g, (Pl - qs) * iimpl, once);
          }
          const float2 f = unpk(b);
          errA = fmaxf(errA, fabsf(f.x) * isc[v]);
          errB = fmaxf(errB, fabsf(f.y) * isc[v]);
          badA = badA || !(fabsf(f.x) < 3.0e38f);
          badB = badB || !(fabsf(f.y) < 3.0e38f);
        };
        row(0, q[0], dd, sd.get());
        row(1, q[1], ld(r2[ri(sc, 0, c.k)]), sm.get());
        row(2, q[2], ld(r2[ri(sc, 4, c.k)]), sr.get());
      }
      if (e + 1 < NeZ) {
#pragma unroll
        for (int v = 0; v < 3; ++v) q[v] = ld_pair(qin.v[gv[v]] + c.g(e + 1, c.k));
      }
      __syncwarp();
    }
    if (e + 2 < NeZ) {
      p2 p[3];
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        p[v] = p2_add_x(pn[v], c.X[v * L + (e + 2) * N1 + c.k]);
        st(c.P[c.pi(v, e + 2)], p[v]);
      }
      fill(e + 2, c.k, p[0], p[1], p[2]);
      if (e + 3 < NeZ) {
#pragma unroll
        for (int v = 0; v < 3; ++v) pn[v] = ld(c.P[c.pi(v, e + 3)]);
      }
    }
    __syncwarp();
  }
  errA = grp_max_nan(badA ? __int_as_float(0x7fc00000) : errA, N1);
  errB = grp_max_nan(badB ? __int_as_float(0x7fc00000) : errB, N1);
  u64x* t = c.X;
  c.X = c.B;
  c.B = t;
}

template <int N1>
__global__ void __launch_bounds__(64, N1 == 8 ? 6 : 4)
    k_vi_series(const __grid_constant__ Ops op, const __grid_constant__ OpsX ox, const ProfX px, const X5 qin, const F5c z,
                const A3 a0, void* const* qsf, void* const* tout, float* gsc, int* status, unsigned long long* cnt,
                const __grid_constant__ SerArgs args, int ncol) {
  constexpr int N = N1 - 1, G = 32 / N1, NF = N1 * N1, Np = NF * N1;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int grp = lane / N1, k = lane % N1;
  const int pair0 = (blockIdx.x * 2 + wib) * G, ncp = ncol / 2;
  if (pair0 >= ncp) return;  // ncp is a multiple of G (checked at the launch); no block barriers
  const int cp = pair0 + grp;
  const int NeZ = op.NeZ, L = op.L;
  const SLayout lay(N1, NeZ);
  unsigned char* base = smraw + (size_t)(wib * G + grp) * lay.stride;
  Pair<N1> c;
  c.X = reinterpret_cast<u64x*>(base);
  c.B = reinterpret_cast<u64x*>(base + lay.oB);
  c.E = base + lay.oE;
  c.A = reinterpret_cast<u64x*>(base + lay.oA);
  c.k = k; c.act = true; c.NeZ = NeZ; c.L = L;
  c.pn = (size_t)ncp * L;
  c.P = reinterpret_cast<p2m*>(gsc);
  c.J = reinterpret_cast<u64x*>(gsc + 12 * c.pn);
  c.pb = (size_t)cp * N1 + k;
  c.ps = (size_t)ncp * N1;
  {
    const int col = 2 * cp, ij = col % NF, exy = col / NF;
    const size_t nxy = (size_t)op.NeX * op.NeY;
    c.gb = (size_t)exy * Np + ij;
    c.gs = nxy * Np;
  }
  const MixViArgs& va = args.v;
  const float kapf = ox.kap.x;
  const unsigned long long once = l2_evict_first();
  const int gv[3] = {VD, VMZ, VRT};

  // ---- one pass over the columns: the iterate P = var0, the first residual
  // b = (q* - var0) + impl_fac A(var0) from the stage-1 kernel's A(var0), the Jacobian's level
  // quantities, and the face nodes' values for the wave speed; the loads run two elements ahead ----
  float bmax = 0.f;  // largest weighted |b|
  {
    const p2 impl = p2_dup(va.impl2);
    u64x* face = c.X;  // [NeZ][2][3]
    double zA[2][3], zB[2][3];
    p2 qc[2][3], ac[2][3];
    auto load = [&](int t, int i) {  // node of element t
      if (t >= NeZ) return;
      const size_t g = c.g(t, c.k);
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        zA[i][v] = ld_once(z.v[gv[v]] + g, once);
        zB[i][v] = ld_once(z.v[gv[v]] + g + 1, once);
        qc[i][v] = ld_pair(qin.v[gv[v]] + g);
        ac[i][v] = ld_once(a0.v[v] + g, once);
      }
    };
    auto node = [&](int t, int i) {
      if (t >= NeZ) return;
      const int e = t;
      const int l = e * N1 + k;
      u64x ph[3];
      p2 P[3], q[3], a[3];
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        P[v] = p2_split(zA[i][v], zB[i][v]);
        q[v] = qc[i][v];
        a[v] = ac[i][v];
      }
      load(t + 2, i);
      float mx[3];
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        ph[v] = P[v].h;
        st(c.P[c.pi(v, e)], P[v]);
        const p2 b = (q[v] - P[v]) + impl * a[v];
        const u64x bf = xadd(b.h, b.l);
        c.B[v * L + l] = bf;
        mx[v] = fmaxf(fabsf(unpk(bf).x), fabsf(unpk(bf).y));
        if (k == 0) face[(2 * e) * 3 + v] = ph[v];
        if (k == N) face[(2 * e + 1) * 3 + v] = ph[v];
      }
      bmax = fmaxf(bmax, fmaxf(mx[0], fmaxf(args.c1 * mx[1], args.c2 * mx[2])));
      // pot = RHOT/DENS, wt = MOMZ/DENS, dpd = kappa PRES/RHOT (FP32, the correction's accuracy)
      const float2 d = unpk(ph[0]), m = unpk(ph[1]), x = unpk(ph[2]);
      const float dh = __ldg(px.dhf + l), rh = __ldg(px.rhf + l), pf = __ldg(px.phf + l), rt = __ldg(px.rthf + l);
      const float iA = __fdividef(1.f, dh + d.x), iB = __fdividef(1.f, dh + d.y);
      const float tA = rh + x.x, tB = rh + x.y;
      c.J[c.pi(0, e)] = pk(tA * iA, tB * iB);
      c.J[c.pi(1, e)] = pk(m.x * iA, m.y * iB);
      c.J[c.pi(2, e)] = pk(__fdividef(kapf * pf * __powf(1.f + x.x * rt, kapf), tA),
                              __fdividef(kapf * pf * __powf(1.f + x.y * rt, kapf), tB));
    };
    load(0, 0);
    load(1, 1);
    for (int t = 0; t < NeZ; t += 2) {
      node(t, 0);
      node(t + 1, 1);
    }
    __syncwarp();
    // frozen wave speed |w| + c at the face nodes (hevi_common_2.F90:1149-1155), a lane per element and side
    for (int t = k; t < 2 * NeZ; t += N1) {
      const int l = (t >> 1) * N1 + ((t & 1) ? N : 0);
      const float dh = __ldg(px.dhf + l), pf = __ldg(px.phf + l), rt = __ldg(px.rthf + l);
      const float2 d = unpk(face[3 * t]), m = unpk(face[3 * t + 1]), x = unpk(face[3 * t + 2]);
      auto speed = [&](float dd0, float mz0, float dr0) {
        const float rdens0 = 1.f / (dh + dd0);
        const float wt0 = mz0 * rdens0;
        const float pres0 = pf * (1.f + expm1f(kapf * log1pf(dr0 * rt)));
        return fabsf(wt0) + sqrtf(kapf * pres0 * rdens0);
      };
      face[3 * t] = pk(speed(d.x, m.x, x.x), speed(d.y, m.y, x.y));
    }
    __syncwarp();
    for (int e = k; e <= NeZ; e += N1) {
      const float2 lo = unpk(face[3 * (e > 0 ? 2 * e - 1 : 0)]), up = unpk(face[3 * (e < NeZ ? 2 * e : 2 * NeZ - 1)]);
      c.A[e] = pk(fmaxf(lo.x, up.x), fmaxf(lo.y, up.y));
    }
    __syncwarp();
  }

  // ---- DENS/MOMZ/RHOT Newton ----
  int nsolve = 0, stA = 0, stB = 0;
  bool give_up = false, emitted = false;
  {
    const SweepCoef<N1> sc(op, va.impl_fac, k, c.A[0]);
    const float ctol = 0.02f * (float)va.tol * args.dmin;
    while (true) {
      // to 2e-6 of the first change, which FP32 resolves to 1e-7 (a later correction goes on from the pair
      // residual), or 2 % of the tolerance, so that what is accepted lies well inside, as after the LU
      // kernel's corrections
      const bool ok = sweeps<N1, N1>(c, sc, op, va.impl_fac, warp_max_bits(bmax), 2.0e-6f, ctol, args.c1, args.c2);
      if (!ok) { give_up = true; break; }
      ++nsolve;
      __syncwarp();
      float eA, eB;
      emitted = nsolve >= 2;
      residual<N1>(ox, args, c, px, qin, qsf, tout, once, emitted, eA, eB);
      bmax = fmaxf(eA, eB) * args.dmin;
      if (!stA && (double)eA <= va.tol) stA = nsolve;
      if (!stB && (double)eB <= va.tol) stB = nsolve;
      if (__all_sync(FULL, (double)eA <= va.tol && (double)eB <= va.tol)) break;
      if (nsolve >= va.max_iter || __any_sync(FULL, eA != eA || eB != eB)) { give_up = true; break; }
    }
  }
  if (give_up) {  // warp-uniform: block LU for these columns, by the kernel that follows
    if (k == 0) status[2 * cp] = status[2 * cp + 1] = VI_REDO;
  } else {
    // ---- DENS/MOMZ/RHOT out, if the accepted residual did not store it ----
    if (!emitted) {
      const p2 iimpl = p2_dup(va.inv_impl2);
      for (int t0 = 0; t0 < NeZ; t0 += 2) {  // two elements' loads in flight
        p2 q[2][3], p[2][3];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int e = t0 + i;
          if (e < NeZ) {
#pragma unroll
            for (int v = 0; v < 3; ++v) {
              q[i][v] = ld_once(qin.v[gv[v]] + c.g(e, c.k), once);
              p[i][v] = ld(c.P[c.pi(v, e)]);
            }
          }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int e = t0 + i;
          if (e < NeZ) {
#pragma unroll
            for (int v = 0; v < 3; ++v) {
              const size_t g = c.g(e, c.k);
              st_once(static_cast<float2*>(qsf[gv[v]]) + g, p[i][v], once);
              st_once(static_cast<float2*>(tout[gv[v]]) + g, (p[i][v] - q[i][v]) * iimpl, once);
            }
          }
        }
      }
    }
    // ---- MOMX/MOMY: the interface jumps J_e (e = 1 .. NeZ - 1; zero at the lids) ----
    //   (1 + beta_e0 + tau_{e-1,N}) J_e - tau_e0 J_{e+1} - beta_{e-1,N} J_{e-1} = q*(e, 0) - q*(e-1, N)
    // beta_ek = cLb[k] A_e, tau_ek = cLt[k] A_{e+1}
    __syncwarp();
    p2m* Jm = reinterpret_cast<p2m*>(base);  // [2][NeZ + 1]
    p2m* Cp = Jm + 2 * (NeZ + 1);            // [NeZ + 1]
    for (int t = k; t < 2 * (NeZ + 1); t += N1) {
      const int m = t & 1, e = t >> 1;
      p2 j = p2_zero();
      if (e > 0 && e < NeZ) j = ld_pair(qin.v[VMX + m] + c.g(e, 0)) - ld_pair(qin.v[VMX + m] + c.g(e - 1, N));
      st(Jm[m * (NeZ + 1) + e], j);
    }
    __syncwarp();
    if (k < 2) {
      p2m* J = Jm + k * (NeZ + 1);
      const p2 diag = p2_dup(args.cLb[0]) + p2_dup(args.cLt[N]);
      const p2 lo = p2_dup(args.cLb[N]), up = p2_dup(args.cLt[0]);
      const p2 one = p2_dup(f2{1.f, 0.f});
      p2 cprev = p2_zero(), rprev = p2_zero();
      for (int e = 1; e < NeZ; ++e) {
        const p2 l = p2_mul_x(lo, e > 1 ? c.A[e - 1] : 0ull);
        const p2 ip = p2_recip((one + p2_mul_x(diag, c.A[e])) - l * cprev);
        cprev = p2_mul_x(up, e < NeZ - 1 ? c.A[e + 1] : 0ull) * ip;
        rprev = (ld(J[e]) + l * rprev) * ip;
        st(J[e], rprev);
        if (k == 0) st(Cp[e], cprev);
      }
    }
    __syncwarp();
    if (k < 2) {
      p2m* J = Jm + k * (NeZ + 1);
      p2 x = p2_zero();
      for (int e = NeZ - 1; e >= 1; --e) {
        x = ld(J[e]) + ld(Cp[e]) * x;
        st(J[e], x);
      }
    }
    __syncwarp();
    {
      const p2 iimpl = p2_dup(va.inv_impl2);
      const p2 U = p2_dup(ox.Uref), V = p2_dup(ox.Vref);
      for (int t0 = 0; t0 < NeZ; t0 += 8) {  // eight elements' loads in flight
        p2 q[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int e = t0 + i;
          if (e < NeZ) {
            q[i][0] = ld_once(qin.v[VMX] + c.g(e, c.k), once);
            q[i][1] = ld_once(qin.v[VMY] + c.g(e, c.k), once);
          }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int e = t0 + i;
          if (e < NeZ) {
            const size_t g = c.g(e, k);
            const p2 be = p2_mul_x(p2_dup(args.cLb[k]), c.A[e]), ta = p2_mul_x(p2_dup(args.cLt[k]), c.A[e + 1]);
            const p2 dh = p2_dup(__ldg(px.dh + e * N1 + k));
#pragma unroll
            for (int m = 0; m < 2; ++m) {
              const p2m* J = Jm + m * (NeZ + 1) + e;
              const p2 E = ta * ld(J[1]) - be * ld(J[0]);
              st_once(static_cast<float2*>(qsf[VMX + m]) + g, (q[i][m] - dh * (m == 0 ? U : V)) + E, once);
              st_once(static_cast<float2*>(tout[VMX + m]) + g, E * iimpl, once);
            }
          }
        }
      }
    }
    if (k == 0) {
      status[2 * cp] = stA;
      status[2 * cp + 1] = stB;
    }
    const unsigned nsol = __reduce_add_sync(FULL, k == 0 ? (unsigned)(stA + stB) : 0u);
    if (lane == 0) {
      atomicAdd(cnt + 1, (unsigned long long)nsol);
      atomicAdd(cnt + 2, (unsigned long long)(2 * G));
    }
  }
  // the planes' lines of this warp are dead: drop them from L2 without a write-back (per element,
  // four 128-byte lines of each plane of P and two of each plane of J)
  __syncwarp();
  for (int t = lane; t < 18 * NeZ; t += 32) {
    const int e = t / 18, r = t - 18 * e;
    const size_t n0 = (size_t)pair0 * N1 + (size_t)e * c.ps;
    const char* a = r < 12 ? reinterpret_cast<const char*>(c.P + (size_t)(r / 4) * c.pn + n0) + 128 * (r % 4)
                           : reinterpret_cast<const char*>(c.J + (size_t)((r - 12) / 2) * c.pn + n0) + 128 * ((r - 12) % 2);
    asm volatile("discard.global.L2 [%0], 128;" ::"l"(a) : "memory");
  }
}

template <int N1>
int launch_n(const Ops& op, const OpsX& ox, const ProfX& px, const X5& qin, const F5c& z, const A3& a0,
             void* const* qsf, void* const* tout, float* gsc, int* status, unsigned long long* cnt, const SerArgs& a,
             cudaStream_t s) {
  constexpr int G = 32 / N1;
  const SLayout lay(N1, op.NeZ);
  const size_t smem = (size_t)lay.stride * 2 * G;
  if (smem > 227 * 1024) return -1;
  const int ncol = op.NeX * op.NeY * N1 * N1, ncp = ncol / 2;
  auto kfn = k_vi_series<N1>;
  cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  kfn<<<(ncp + 2 * G - 1) / (2 * G), 64, smem, s>>>(op, ox, px, qin, z, a0, qsf, tout, gsc, status, cnt, a, ncol);
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
  switch (N1) {
    case 4: return launch_n<4>(op, ox, px, qin, z, a0, qsf, tout, gsc, status, cnt, sa, s);
    case 8: return launch_n<8>(op, ox, px, qin, z, a0, qsf, tout, gsc, status, cnt, sa, s);
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace fedg
