// fedg_vi64.cu -- FP64 vertical-implicit column solve (cal_vi) by iterative refinement: FP32 sweeps as the
// solver, FP64 residuals, two columns per lane.
//
// Same problem as k_vi_fp64 (fedg_vi.cu; FElib's cal_vi, scale_atm_dyn_dgm_nonhydro3d_rhot_hevi.F90:772-965,
// hevi_common_2.F90): Newton on P - q* - impl_fac A(P) = 0 from var0, each linear system J delta = b solved to
// FP64 roundoff, the nonlinear residual and its convergence test in FP64; one solve for max_iter = 1,
// A(var0) itself for impl_fac = 0.  k_vi_fp64 factors J (pivoted block LU): about 2400 FP64 operations per
// node, on a part that retires two per cycle and SM.  Here delta is built up in FP64 from FP32 solutions,
// delta += S (b - J delta), where S is a series of packed FP32 sweeps (fedg_sweep.cuh) that leaves about 1e-6
// of its right-hand side, and b - J delta is formed in FP64 from the FP64 delta: two such residuals take the
// linear system's error from 1e-6 over 1e-12 below 1e-16, where the next FP64 residual has nothing left
// to see; a system for which the residual does not say so is not taken as solved.  That costs 346 FP64 instructions per
// node for a launch with one solve and its nonlinear residuals.  The pressure
// deviation PRES_hyd ((1 + DRHOT/RHOT_hyd)^kappa - 1) is its binomial series up to 3 % (13 terms, to
// roundoff, no cancellation of totals) and pow() beyond.  A column whose sweeps do not contract, whose Newton
// does not converge in max_iter solves or whose residual is not finite stores nothing but a mark in
// `status`; k_vi_fp64, launched after this kernel, solves the marked columns from the start, and all of them where
// block_lu_alone says so.
//
// MOMX/MOMY: Q - q* from the interface jumps, one Thomas sweep per component (see fedg_viseries.cu), in FP64.
//
// Layout: GL = 2, 4 or 8 lanes per pair of neighbouring columns, lane k < N1 owns node k of every element.  Relaxation,
// stopping rules and counts are the column's own, so its result does not depend on which columns share its lanes or its
// warp: a decomposed mesh gives the bits of the whole one.
// FP64 fields of the columns in flight (the iterate, b, delta, the Jacobian's level quantities) sit in a
// global slice of the warp, 16 bytes per lane and entry, which a persistent grid keeps in L2; the FP32
// vectors and the exchange of level quantities are in shared memory.
//
// What bounds it: the FP64 pipe, 69 % busy (p = 7, 16x16x8 elements: 968 us per launch, A(var0) alone 254 us; block LU
// 4562 us); on small meshes the length of a warp's chain (93,000 instructions for 8 elements of p = 3).
#include <algorithm>

#include "fedg_kernels.cuh"
#include "fedg_sweep.cuh"

namespace fedg {
namespace {

struct S64Args {
  ViArgs v;
  double cD[FEDG_MAXN1 * FEDG_MAXN1], cLb[FEDG_MAXN1], cLt[FEDG_MAXN1], tv[FEDG_MAXN1], tw[FEDG_MAXN1], cg;
  double cb[13];     // binomial coefficients C(kappa, n), n = 1 .. 13
  double inv_impl;   // 1 / impl_fac
  float c1, c2;      // weights of MOMZ and RHOT in the sweeps' change
  float tol_lo, tol_hi;  // tol less and plus 1e-5 of it
};

// shared memory of one column pair (bytes): the FP32 vectors x and b, the sweeps' exchange slots, the
// wave speeds in FP64 and FP32.  x's space also holds the residuals' ring of level quantities and the
// face values of the wave-speed pass; the two vectors together the MOMX/MOMY system.
struct S64Layout {
  int oB, oE, oA, oAf, stride;
  __host__ __device__ S64Layout(int N1, int GL, int NeZ) {
    const int L = N1 * NeZ, ring = 3 * 5 * 16 * N1 + 96, uv = 24 * (NeZ + 1);
    oB = 24 * L;
    if (oB < ring) oB = ring;
    if (oB < uv) oB = uv;
    oB = (oB + 15) / 16 * 16;
    oE = 2 * oB;
    oA = oE + 2 * (32 * N1 + 16);
    oAf = oA + 16 * (NeZ + 1);
    const int o = oAf + 8 * (NeZ + 1);
    const int r = 8 * GL, m = 128;  // the pairs of a half warp on different banks
    stride = ((o - r + m - 1) / m) * m + r;
  }
};

// doubles of one warp's global slice: P, b, delta, pot/wt/dpd as (A, B) pairs, and the FP32 copy of the last
__host__ __device__ inline size_t s64_slice(int NeZ) { return (size_t)NeZ * 32 * (12 * 2 + 3); }

__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 operator*(double2 a, double2 b) { return make_double2(a.x * b.x, a.y * b.y); }
__device__ __forceinline__ double2 operator*(double a, double2 b) { return make_double2(a * b.x, a * b.y); }
__device__ __forceinline__ double2 fma2(double a, double2 b, double2 c) { return make_double2(fma(a, b.x, c.x), fma(a, b.y, c.y)); }
__device__ __forceinline__ double2 fma2(double2 a, double2 b, double2 c) { return make_double2(fma(a.x, b.x, c.x), fma(a.y, b.y, c.y)); }
__device__ __forceinline__ double2 neg2(double2 a) { return make_double2(-a.x, -a.y); }
__device__ __forceinline__ u64x to_f(double2 a) { return pk((float)a.x, (float)a.y); }
__device__ __forceinline__ double2 shx(double2 v, int o) {
  return make_double2(__shfl_xor_sync(FULL, v.x, o), __shfl_xor_sync(FULL, v.y, o));
}
constexpr double2 Z22{0.0, 0.0};

// (1 + r)^kappa - 1
__device__ __noinline__ double dev_pow64(double r, double kap) { return pow(1.0 + r, kap) - 1.0; }
__device__ __forceinline__ double dev64(const S64Args& a, double r, double kap) {
  if (!(fabs(r) <= 0.03)) return dev_pow64(r, kap);
  double s = a.cb[12];
#pragma unroll
  for (int m = 11; m >= 0; --m) s = fma(s, r, a.cb[m]);
  return s * r;
}

template <int N1, int GL>
struct Ctx64 : SweepCtx<N1, GL> {
  double2* W;       // the warp's slice: planes [12][NeZ][32]
  double2* A64;     // wave speed of face e
  int lane;
  size_t gA, gB, gs;  // node index of (0, 0) of the two columns, element-layer stride
  __device__ double2& w(int plane, int v, int e) const { return W[((size_t)(3 * plane + v) * this->NeZ + e) * 32 + lane]; }
  __device__ double2 ldg2(const double* q, int e, int k) const {
    const size_t o = (size_t)e * gs + (size_t)(N1 * N1) * k;
    return make_double2(__ldg(q + gA + o), __ldg(q + gB + o));
  }
};
enum { W_P = 0, W_B = 1, W_D = 2, W_J = 3 };

// One pass over the columns with the vertical operator: fill(e, q) gives the level quantities of the lane's
// node, q = (MOMZ, DENS, momentum flux, heat flux, RHOT), nonlinear or linearised; row(e, q, s) takes the
// operator s = f (E33 D flux + Lift faces + grav VPOrdM1 DENS), f = impl_fac (1 for impl_fac = 0).
template <int N1, int GL, class Fill, class Row>
__device__ __forceinline__ void pass64(const S64Args& args, const Ctx64<N1, GL>& c, Fill&& fill, Row&& row) {
  constexpr int N = N1 - 1;
  const int k = c.k, NeZ = c.NeZ;
  double2* r2 = reinterpret_cast<double2*>(c.X);
  double2* del = r2 + 3 * 5 * N1;
  auto ri = [](int s, int q, int m) { return (s * 5 + q) * N1 + m; };
  double Dk[N1];
#pragma unroll
  for (int m = 0; m < N1; ++m) Dk[m] = args.cD[k * N1 + m];
  const double lb = args.cLb[k], lt = args.cLt[k], tv = args.tv[k], tw = c.act ? args.tw[k] : 0.0;
  for (int e = -2; e < NeZ; ++e) {
    if (e >= 0) {
      const int sc = e % 3, sb = (e + 2) % 3, su = (e + 1) % 3;
      // vertical-face fluxes of element e: lanes over (side, variable)
      for (int t = c.lane % GL; t < 6; t += GL) {
        const int s = t / 3, v = t - 3 * s;
        const int nM = s == 0 ? 0 : N;
        const bool lid = s == 0 ? (e == 0) : (e == NeZ - 1);
        const int sP = lid ? sc : (s == 0 ? sb : su), nP = lid ? nM : (s == 0 ? N : 0);
        const double2 al = c.A64[e + s];
        // v = 0: MOMZ (flux) and DENS; 1: pressure and MOMZ; 2: heat flux and RHOT.  A slip lid reflects
        // MOMZ and the heat flux and leaves the rest without a jump
        const int qf = v == 0 ? 0 : (v == 1 ? 2 : 3), qd = v == 0 ? 1 : (v == 1 ? 0 : 4);
        const double2 fM = r2[ri(sc, qf, nM)], dM = r2[ri(sc, qd, nM)];
        double2 fP = r2[ri(sP, qf, nP)], dP = r2[ri(sP, qd, nP)];
        if (lid) {
          if (v != 1) fP = neg2(fP);
          else dP = neg2(dP);
        }
        del[t] = fma2(neg2(al), dP - dM, s == 0 ? fM - fP : fP - fM);
      }
      __syncwarp();
      {
        const double2 own[3] = {r2[ri(sc, 1, k)], r2[ri(sc, 0, k)], r2[ri(sc, 4, k)]};
        double2 mode = tw * own[0];  // the mode that VPOrdM1 removes: summed over the column's nodes
#pragma unroll
        for (int o = GL / 2; o > 0; o >>= 1) mode = mode + shx(mode, o);
        double2 s[3] = {Z22, fma2(args.cg, own[0], (-tv) * mode), Z22};
#pragma unroll
        for (int m = 0; m < N1; ++m) {
          s[0] = fma2(Dk[m], r2[ri(sc, 0, m)], s[0]);
          s[1] = fma2(Dk[m], r2[ri(sc, 2, m)], s[1]);
          s[2] = fma2(Dk[m], r2[ri(sc, 3, m)], s[2]);
        }
#pragma unroll
        for (int v = 0; v < 3; ++v) s[v] = fma2(lb, del[v], fma2(lt, del[3 + v], s[v]));
        row(e, own, s);
      }
      __syncwarp();
    }
    if (e + 2 < NeZ) {
      double2 q[5];
      fill(e + 2, q);
      if (GL == N1 || c.act) {
        const int s = (e + 2) % 3;
#pragma unroll
        for (int m = 0; m < 5; ++m) r2[ri(s, m, k)] = q[m];
      }
    }
    __syncwarp();
  }
}

// max |b| / scale of a pair's two columns from its planes of b (kept out of line: it hardly ever runs)
template <int GL>
__device__ __noinline__ double2 scaled_max(const Prof& pf, double cref, const double2* b, int k, int N1, int NeZ) {
  double2 x = Z22;
  for (int e = 0; e < NeZ; ++e) {
    const double dh = __ldg(pf.dens + e * N1 + k), scale[3] = {dh, dh * cref, __ldg(pf.rhyd + e * N1 + k)};
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      const double2 y = b[((size_t)v * NeZ + e) * 32];
      x = make_double2(fmax(x.x, fabs(y.x) / scale[v]), fmax(x.y, fabs(y.y) / scale[v]));
    }
  }
#pragma unroll
  for (int o = GL / 2; o > 0; o >>= 1) {
    const double2 y = shx(x, o);
    x = make_double2(fmax(x.x, y.x), fmax(x.y, y.y));
  }
  return x;
}

template <int N1, int GL>
__global__ void __launch_bounds__(64, 6)
    k_vi64(const __grid_constant__ Ops op, const Prof pf, const F5c qin, const F5c z, const F5 tout, int* status,
           const __grid_constant__ S64Args args, int ncol, double* gsc) {
  constexpr int N = N1 - 1, G = 32 / GL, NF = N1 * N1, Np = NF * N1;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int slot = blockIdx.x * wpb + wib, nslot = gridDim.x * wpb;
  const int grp = lane / GL, kl = lane % GL;
  const int NeZ = op.NeZ, L = op.L, ncp = (ncol + 1) / 2;
  const S64Layout lay(N1, GL, NeZ);
  unsigned char* base = smraw + (size_t)(wib * G + grp) * lay.stride;
  Ctx64<N1, GL> c;
  c.X = reinterpret_cast<u64x*>(base);
  c.B = reinterpret_cast<u64x*>(base + lay.oB);
  c.E = base + lay.oE;
  c.A64 = reinterpret_cast<double2*>(base + lay.oA);
  c.A = reinterpret_cast<u64x*>(base + lay.oAf);
  c.k = kl < N1 ? kl : N; c.act = kl < N1; c.NeZ = NeZ; c.L = L; c.lane = lane;
  c.W = reinterpret_cast<double2*>(gsc + (size_t)slot * s64_slice(NeZ));
  c.J = reinterpret_cast<u64x*>(c.W + (size_t)12 * NeZ * 32);
  c.pn = (size_t)NeZ * 32; c.pb = lane; c.ps = 32;
  const int k = c.k;
  const double impl = args.v.impl_fac, kap = op.kap;
  const int gv[3] = {VD, VMZ, VRT};

  for (int p0 = slot * G; p0 < ncp; p0 += nslot * G) {
    const int cp = min(p0 + grp, ncp - 1), colA = 2 * cp, colB = min(colA + 1, ncol - 1);
    bool liveA = p0 + grp < ncp && c.act, liveB = liveA && colB != colA;
    c.gA = (size_t)(colA / NF) * Np + colA % NF;
    c.gB = (size_t)(colB / NF) * Np + colB % NF;
    c.gs = (size_t)op.NeX * op.NeY * Np;
    auto store = [&](int v, int e, double2 x) {
      const size_t o = (size_t)e * c.gs + (size_t)NF * k;
      if (liveA) tout.v[v][c.gA + o] = x.x;
      if (liveB) tout.v[v][c.gB + o] = x.y;
    };

    // ---- the iterate P = var0; the frozen wave speed |w| + c of its face nodes (hevi_common_2.F90:1149-1155),
    // a lane per element and side ----
    {
      double2* face = reinterpret_cast<double2*>(c.X);  // [NeZ][2][3], then the speeds in [.][.][0]
      for (int e = 0; e < NeZ; ++e) {
#pragma unroll
        for (int v = 0; v < 3; ++v) {
          const double2 x = c.ldg2(z.v[gv[v]], e, k);
          c.w(W_P, v, e) = x;
          if (c.act && k == 0) face[(2 * e) * 3 + v] = x;
          if (c.act && k == N) face[(2 * e + 1) * 3 + v] = x;
        }
      }
      __syncwarp();
      for (int t = kl; t < 2 * NeZ; t += GL) {
        const int l = (t >> 1) * N1 + ((t & 1) ? N : 0);
        const double dh = __ldg(pf.dens + l), ph = __ldg(pf.pres + l), ri = __ldg(pf.rhinv + l);
        const double2 d = face[3 * t], m = face[3 * t + 1], r = face[3 * t + 2];
        auto speed = [&](double dd0, double mz0, double dr0) {
          const double rdens0 = 1.0 / (dh + dd0);
          const double pres0 = fma(ph, dev64(args, dr0 * ri, kap), ph);
          return fabs(mz0 * rdens0) + sqrt(kap * pres0 * rdens0);
        };
        face[3 * t] = make_double2(speed(d.x, m.x, r.x), speed(d.y, m.y, r.y));
      }
      __syncwarp();
      for (int e = kl; e <= NeZ; e += GL) {
        const double2 lo = face[3 * (e > 0 ? 2 * e - 1 : 0)], up = face[3 * (e < NeZ ? 2 * e : 2 * NeZ - 1)];
        const double2 a = make_double2(fmax(lo.x, up.x), fmax(lo.y, up.y));
        c.A64[e] = a;
        c.A[e] = to_f(a);
      }
      __syncwarp();
    }

    // nonlinear level quantities of the iterate (eval_Ax :236-295), and the Jacobian's
    auto fill = [&](int e, double2 (&q)[5]) {
      const int l = e * N1 + k;
      const double2 Pd = c.w(W_P, 0, e), Pm = c.w(W_P, 1, e), Pr = c.w(W_P, 2, e);
      const double dh = __ldg(pf.dens + l), rh = __ldg(pf.rhyd + l), ph = __ldg(pf.pres + l), ri = __ldg(pf.rhinv + l);
      const double2 rd = make_double2(1.0 / (dh + Pd.x), 1.0 / (dh + Pd.y));
      const double2 rt = make_double2(rh + Pr.x, rh + Pr.y);
      const double2 pot = rt * rd;
      const double2 S = make_double2(dev64(args, Pr.x * ri, kap), dev64(args, Pr.y * ri, kap));
      q[0] = Pm;
      q[1] = Pd;
      q[2] = ph * S;
      q[3] = pot * Pm;
      q[4] = Pr;
      if (impl != 0.0) {
        const double2 wt = Pm * rd;
        const double kp = kap * ph;
        const double2 dp = make_double2(fma(kp, S.x, kp) / rt.x, fma(kp, S.y, kp) / rt.y);
        c.w(W_J, 0, e) = pot;
        c.w(W_J, 1, e) = wt;
        c.w(W_J, 2, e) = dp;
        c.J[c.pi(0, e)] = to_f(pot);
        c.J[c.pi(1, e)] = to_f(wt);
        c.J[c.pi(2, e)] = to_f(dp);
      }
    };

    int stA = 0, stB = 0;
    if (impl == 0.0) {
      pass64<N1, GL>(args, c, fill, [&](int e, const double2 (&)[3], const double2 (&s)[3]) {
#pragma unroll
        for (int v = 0; v < 3; ++v) store(gv[v], e, neg2(s[v]));
      });
    } else {
      // ---- DENS/MOMZ/RHOT Newton.  Sets of columns: bit 0 is A, bit 1 is B, uniform over the pair's lanes ----
      const SweepCoef<N1> sc(op, impl, c.A[0]);
      int run = (p0 + grp < ncp ? 1 : 0) | (p0 + grp < ncp && colB != colA ? 2 : 0), give_up = 0;  // run: still iterating
      int nsolve = 0;
      while (true) {
        float errA = 0.f, errB = 0.f;
        unsigned bm[2] = {0u, 0u};
        pass64<N1, GL>(args, c, fill, [&](int e, const double2 (&own)[3], const double2 (&s)[3]) {
          const int l = e * N1 + k;
          const float dh = (float)__ldg(pf.dens + l), rh = (float)__ldg(pf.rhyd + l);
          const float isc[3] = {__fdividef(1.f, dh), __fdividef(1.f, dh * (float)args.v.cref), __fdividef(1.f, rh)};
          const float wt[3] = {1.f, args.c1, args.c2};
#pragma unroll
          for (int v = 0; v < 3; ++v) {
            const double2 b = (c.ldg2(qin.v[gv[v]], e, k) - own[v]) - s[v];
            c.w(W_B, v, e) = b;
            const u64x bf = to_f(b);
            if (c.act) c.B[v * L + l] = bf;
            const float2 f = unpk(bf);
            errA = fmaxf(errA, fabsf(f.x) * isc[v]);
            errB = fmaxf(errB, fabsf(f.y) * isc[v]);
            max_bits(bm[0], wt[v], f.x);
            max_bits(bm[1], wt[v], f.y);
          }
        });
        const float2 bmax = make_float2(pair_max_bits<GL>(bm[0]), pair_max_bits<GL>(bm[1]));
        const int bad = run & ((bmax.x < 3.0e38f ? 0 : 1) | (bmax.y < 3.0e38f ? 0 : 2));
        give_up |= bad;
        run &= ~bad;
        if (args.v.max_iter > 1) {
#pragma unroll
          for (int o = GL / 2; o > 0; o >>= 1) {
            errA = fmaxf(errA, __shfl_xor_sync(FULL, errA, o));
            errB = fmaxf(errB, __shfl_xor_sync(FULL, errB, o));
          }
          // The test is in FP64.  errA and errB are right to 1e-6 (above FP32's smallest numbers), so they decide it
          // outside 1e-5 of tol; the rest takes the FP64 residual that the pass left
          auto above = [&](float x) { return x > 1.0e-30f && x > args.tol_hi; };
          auto sure = [&](float x) { return above(x) || (args.tol_lo > 1.0e-30f && x < args.tol_lo); };
          int conv = (above(errA) ? 0 : 1) | (above(errB) ? 0 : 2);
          if (__any_sync(FULL, run & ((sure(errA) ? 0 : 1) | (sure(errB) ? 0 : 2)))) {
            const double2 x = scaled_max<GL>(pf, args.v.cref, c.W + (size_t)3 * W_B * NeZ * 32 + lane, k, N1, NeZ);
            conv = (x.x <= args.v.tol ? 1 : 0) | (x.y <= args.v.tol ? 2 : 0);
          }
          conv &= run;
          if (conv & 1) stA = nsolve;
          if (conv & 2) stB = nsolve;
          run &= ~conv;
          if (nsolve >= args.v.max_iter) {
            give_up |= run;
            run = 0;
          }
        }
        if (!__any_sync(FULL, run)) break;
        // ---- J delta = b by refinement: rho is the residual's size over b's.  Solved once what the last sweeps
        // left, or the residual itself, is below FP64's roundoff; anything else is left to block LU ----
        float2 rho = make_float2(1.f, 1.f), rmax = bmax;
        int open = run, solved = 0;  // open: still refining
        for (int it = 0; it < 6; ++it) {
          // the sweeps leave rel of their right-hand side; the last ones need not go below FP64's roundoff
          const float2 rel = make_float2(fminf(1.0e-3f, fmaxf(1.0e-6f, 1.0e-17f / rho.x)), fminf(1.0e-3f, fmaxf(1.0e-6f, 1.0e-17f / rho.y)));
          open = sweeps<N1, GL>(c, sc, op, impl, rmax, rel, args.c1, args.c2, open);
          if (open) {
            for (int e = 0; e < NeZ; ++e) {
#pragma unroll
              for (int v = 0; v < 3; ++v) {
                const float2 x = unpk(c.X[v * L + e * N1 + k]);
                double2& d = c.w(W_D, v, e);
                d = it == 0 ? make_double2(x.x, x.y) : make_double2(open & 1 ? d.x + x.x : d.x, open & 2 ? d.y + x.y : d.y);
              }
            }
            // what these sweeps left is below 1e-17 of b
            const int last = open & ((rho.x <= 1.0e-11f ? 1 : 0) | (rho.y <= 1.0e-11f ? 2 : 0));
            solved |= last;
            open &= ~last;
          }
          if (!__any_sync(FULL, open)) break;
          unsigned rm[2] = {0u, 0u};
          pass64<N1, GL>(
              args, c,
              [&](int e, double2 (&q)[5]) {  // linearised level quantities of delta
                const double2 dr = c.w(W_D, 0, e), dm = c.w(W_D, 1, e), dt = c.w(W_D, 2, e);
                const double2 pot = c.w(W_J, 0, e), wt = c.w(W_J, 1, e), dp = c.w(W_J, 2, e);
                q[0] = dm;
                q[1] = dr;
                q[2] = dp * dt;
                q[3] = fma2(pot, fma2(neg2(wt), dr, dm), wt * dt);
                q[4] = dt;
              },
              [&](int e, const double2 (&own)[3], const double2 (&s)[3]) {
                const int l = e * N1 + k;
                const float wt[3] = {1.f, args.c1, args.c2};
#pragma unroll
                for (int v = 0; v < 3; ++v) {
                  const u64x r = to_f((c.w(W_B, v, e) - own[v]) - s[v]);
                  if (c.act) c.B[v * L + l] = r;
                  const float2 f = unpk(r);
                  max_bits(rm[0], wt[v], f.x);
                  max_bits(rm[1], wt[v], f.y);
                }
              });
          rmax = make_float2(pair_max_bits<GL>(rm[0]), pair_max_bits<GL>(rm[1]));
          rho = make_float2(bmax.x > 0.f ? rmax.x / bmax.x : rmax.x, bmax.y > 0.f ? rmax.y / bmax.y : rmax.y);
          // NaN: neither solved nor open
          solved |= open & ((rho.x < 1.0e-16f ? 1 : 0) | (rho.y < 1.0e-16f ? 2 : 0));
          open &= ((rho.x < 0.1f ? 1 : 0) | (rho.y < 0.1f ? 2 : 0)) & ~solved;
          if (!__any_sync(FULL, open)) break;
        }
        give_up |= run & ~solved;
        run &= solved;
        ++nsolve;
        if (run) {
          for (int e = 0; e < NeZ; ++e) {
#pragma unroll
            for (int v = 0; v < 3; ++v) {
              const double2 d = c.w(W_D, v, e);
              double2& P = c.w(W_P, v, e);
              P = make_double2(run & 1 ? P.x + d.x : P.x, run & 2 ? P.y + d.y : P.y);
            }
          }
        }
        __syncwarp();
        if (args.v.max_iter <= 1) {  // one solve (the launcher sends a limit below 1 to block LU)
          stA = stB = 1;
          break;
        }
      }
      // block LU for these columns, by the kernel that follows
      if ((give_up & 1) && liveA) {
        if (k == 0) status[colA] = VI_REDO;
        liveA = false;
      }
      if ((give_up & 2) && liveB) {
        if (k == 0) status[colB] = VI_REDO;
        liveB = false;
      }
      __syncwarp();
      if (!__any_sync(FULL, liveA || liveB)) continue;
      for (int e = 0; e < NeZ; ++e) {
#pragma unroll
        for (int v = 0; v < 3; ++v)
          store(gv[v], e, args.inv_impl * (c.w(W_P, v, e) - c.ldg2(qin.v[gv[v]], e, k)));
      }
    }

    // ---- MOMX/MOMY (eval_Ax_uv / solve_uv): beta_ek = cLb[k] A_e, tau_ek = cLt[k] A_{e+1}.  impl_fac = 0: A
    // from the jumps of var0.  Otherwise the jumps J_e of Q from those of q*,
    //   (1 + beta_e0 + tau_{e-1,N}) J_e - tau_e0 J_{e+1} - beta_{e-1,N} J_{e-1} = q*(e, 0) - q*(e-1, N),
    // and Q - q* = tau_ek J_{e+1} - beta_ek J_e ----
    {
      __syncwarp();
      double2* Jm = reinterpret_cast<double2*>(c.X);  // [2][NeZ + 1]
      double2* Cp = Jm + 2 * (NeZ + 1);               // [NeZ + 1]
      const F5c& src = impl == 0.0 ? z : qin;
      for (int t = kl; t < 2 * (NeZ + 1); t += GL) {
        const int m = t & 1, e = t >> 1;
        Jm[m * (NeZ + 1) + e] = e > 0 && e < NeZ ? c.ldg2(src.v[VMX + m], e, 0) - c.ldg2(src.v[VMX + m], e - 1, N) : Z22;
      }
      __syncwarp();
      if (impl != 0.0) {
        if (kl < 2) {
          double2* J = Jm + kl * (NeZ + 1);
          const double diag = args.cLb[0] + args.cLt[N], lo = args.cLb[N], up = args.cLt[0];
          double2 cprev = Z22, rprev = Z22;
          for (int e = 1; e < NeZ; ++e) {
            const double2 a = c.A64[e], l = e > 1 ? lo * c.A64[e - 1] : Z22, u = e < NeZ - 1 ? up * c.A64[e + 1] : Z22;
            const double2 ip = make_double2(1.0 / (fma(diag, a.x, 1.0) - l.x * cprev.x), 1.0 / (fma(diag, a.y, 1.0) - l.y * cprev.y));
            cprev = u * ip;
            rprev = fma2(l, rprev, J[e]) * ip;
            J[e] = rprev;
            if (kl == 0) Cp[e] = cprev;
          }
        }
        __syncwarp();
        if (kl < 2) {
          double2* J = Jm + kl * (NeZ + 1);
          double2 x = Z22;
          for (int e = NeZ - 1; e >= 1; --e) {
            x = fma2(Cp[e], x, J[e]);
            J[e] = x;
          }
        }
        __syncwarp();
      }
      const double lb = args.cLb[k], lt = args.cLt[k], f = impl == 0.0 ? 1.0 : args.inv_impl;
      for (int e = 0; e < NeZ; ++e) {
        const double2 be = lb * c.A64[e], ta = lt * c.A64[e + 1];
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const double2* J = Jm + m * (NeZ + 1) + e;
          double2 d = ta * J[1] - be * J[0];
          if (impl != 0.0) {  // Q - q* of the rounded Q, as cal_vi forms it: zero where it is below Q's last bit
            const double2 qs = c.ldg2(qin.v[VMX + m], e, k);
            d = (qs + d) - qs;
          }
          store(VMX + m, e, f * d);
        }
      }
    }
    if (c.act && k == 0 && status) {
      if (liveA) status[colA] = stA;
      if (liveB) status[colB] = stB;
    }
    __syncwarp();
  }
}

struct Plan64 {
  int wpb = 0, grid = 0;
  size_t smem = 0, scratch = 0;
};

template <int N1>
constexpr int gl_of() { return N1 <= 2 ? 2 : (N1 <= 4 ? 4 : 8); }

template <int N1>
int plan_n(const Ops& op, Plan64& p) {
  constexpr int GL = gl_of<N1>(), G = 32 / GL;
  const S64Layout lay(N1, GL, op.NeZ);
  int dev = 0, nsm = 0, nb = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  auto kfn = k_vi64<N1, GL>;
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
  if (e != cudaSuccess) return (int)e;
  for (p.wpb = 2; p.wpb >= 1; --p.wpb) {
    p.smem = (size_t)lay.stride * G * p.wpb;
    if (p.smem <= 227 * 1024) break;
  }
  if (p.wpb == 0) return 0;  // the columns are too tall: block LU alone
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kfn, 32 * p.wpb, p.smem)) != cudaSuccess) return (int)e;
  const int ncp = (op.NeX * op.NeY * N1 * N1 + 1) / 2, per = G * p.wpb;
  p.grid = std::max(1, std::min((ncp + per - 1) / per, nb * nsm));
  p.scratch = (size_t)p.grid * p.wpb * s64_slice(op.NeZ);
  return 0;
}

template <int N1>
int launch_n(const Plan64& p, const Ops& op, const Prof& pf, const F5c& qin, const F5c& z, const F5& tout, int* status,
             const S64Args& a, double* gsc, cudaStream_t s) {
  k_vi64<N1, gl_of<N1>()><<<p.grid, 32 * p.wpb, p.smem, s>>>(op, pf, qin, z, tout, status, a, op.NeX * op.NeY * N1 * N1, gsc);
  return (int)cudaGetLastError();
}

int plan(const Ops& op, Plan64& p) {
  switch (op.N1) {
    case 2: return plan_n<2>(op, p);
    case 3: return plan_n<3>(op, p);
    case 4: return plan_n<4>(op, p);
    case 5: return plan_n<5>(op, p);
    case 6: return plan_n<6>(op, p);
    case 7: return plan_n<7>(op, p);
    case 8: return plan_n<8>(op, p);
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace

// Calls that block LU serves better: no solve allowed; sweeps that do not contract; and at p <= 3 the meshes whose
// pairs of columns give each scheduler at most one of LU's warps (four per SM).  There this kernel's few warps are
// held by the length of their chain, while LU's take the time of one.  Step in us, refinement / LU: p = 3, NeZ = 8, 512
// pairs of columns 797 / 660, 800 pairs 816 / 911, 2048 938 / 1776; p = 2, 288 pairs 1016 / 813, 648 873 / 880, 1152 838 /
// 896; p = 1, 128 pairs 910 / 574, 2048 1105 / 1196; p = 4, 200 pairs 747 / 774.  Not for a part of a decomposed
// domain, which has to take what the whole domain takes (bit-equal down to that size).
static bool block_lu_alone(const Ops& op, const ViArgs& v) {
  const int pairs = (op.NeX * op.NeY * op.N1 * op.N1 + 1) / 2;
  return v.max_iter < 1 || vi_courant(op, v.impl_fac) > vi_courant_max(op.N1) ||
         (op.N1 <= 4 && pairs <= 4 * op.nsm && !op.part);
}

size_t vi64_scratch_doubles(const Ops& op) {
  Plan64 p;
  return plan(op, p) ? 0 : p.scratch;
}

int launch_vi64(const Ops& op, const Prof& pf, const F5c& qin, const F5c& z, const F5& tout, int* status, const ViArgs& v,
                double* gsc, size_t gsc_doubles, cudaStream_t s) {
  Plan64 p;
  if (const int r = plan(op, p)) return r;
  if (p.wpb == 0 || (v.impl_fac != 0.0 && block_lu_alone(op, v))) return -1;
  if (!gsc || gsc_doubles < p.scratch) return (int)cudaErrorInvalidValue;
  S64Args a;
  a.v = v;
  const int N1 = op.N1;
  const double f = v.impl_fac != 0.0 ? v.impl_fac : 1.0;
  a.inv_impl = 1.0 / f;
  for (int i = 0; i < N1 * N1; ++i) a.cD[i] = f * op.E33 * op.D[i];
  // VPOrdM1 = I - R, R the projection on the highest mode, of rank one: R = R(:, 0) R(0, :) / R(0, 0)
  for (int k = 0; k < N1; ++k) {
    a.cLb[k] = 0.5 * f * op.FSz * op.Lb[k];
    a.cLt[k] = 0.5 * f * op.FSz * op.Lt[k];
    a.tv[k] = f * op.grav * ((k == 0 ? 1.0 : 0.0) - op.T[k * N1]) / (1.0 - op.T[0]);
    a.tw[k] = (k == 0 ? 1.0 : 0.0) - op.T[k];
  }
  a.cg = f * op.grav;
  double cn = 1.0;
  for (int n = 1; n <= 13; ++n) {
    cn *= (op.kap - (n - 1)) / n;
    a.cb[n - 1] = cn;
  }
  // MOMZ against 340 m/s of density, RHOT against 300 K of it
  a.c1 = (float)(1.0 / v.cref);
  a.c2 = 1.f / 300.f;
  a.tol_lo = (float)(v.tol * (1.0 - 1.0e-5));
  a.tol_hi = (float)(v.tol * (1.0 + 1.0e-5));
  switch (N1) {
    case 2: return launch_n<2>(p, op, pf, qin, z, tout, status, a, gsc, s);
    case 3: return launch_n<3>(p, op, pf, qin, z, tout, status, a, gsc, s);
    case 4: return launch_n<4>(p, op, pf, qin, z, tout, status, a, gsc, s);
    case 5: return launch_n<5>(p, op, pf, qin, z, tout, status, a, gsc, s);
    case 6: return launch_n<6>(p, op, pf, qin, z, tout, status, a, gsc, s);
    case 7: return launch_n<7>(p, op, pf, qin, z, tout, status, a, gsc, s);
    case 8: return launch_n<8>(p, op, pf, qin, z, tout, status, a, gsc, s);
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace fedg
