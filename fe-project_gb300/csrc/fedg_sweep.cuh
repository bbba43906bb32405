// fedg_sweep.cuh -- the fixed-point sweeps of the FP64 column solve (fedg_vi64.cu): FP32 solutions of J x = b, J = I + K the
// Jacobian of the DENS/MOMZ/RHOT system, for two columns per lane in packed arithmetic.
//
// x <- (1 - w) x + w (b - K x) with w = 1 / (1 + d), d the face dissipation's diagonal entry: K's spectrum
// is the dissipation's [0, 2 d] plus an almost imaginary acoustic part, and w centres it.  A sweep contracts by 0.08 to
// 0.14 on elements about as tall as wide at the step that the explicit horizontal terms allow, by up to 0.58 at the
// largest d that the solve is launched for (vi_courant_max).
#pragma once
#include "fedg_common.cuh"
#include "fedg_p2.cuh"

namespace fedg {
namespace {

constexpr unsigned FULL = 0xffffffffu;

// running maximum of w |a|, w > 0, as the bits of a non-negative float; NaN wins
__device__ __forceinline__ void max_bits(unsigned& m, float w, float a) { m = max(m, __float_as_uint(w * fabsf(a))); }
// over the GL lanes of a pair; e >= 0 or NaN (which wins)
template <int GL>
__device__ __forceinline__ float pair_max_bits(unsigned v) {
#pragma unroll
  for (int o = GL / 2; o > 0; o >>= 1) v = max(v, __shfl_xor_sync(FULL, v, o));
  return __uint_as_float(v);
}

// One pair of columns: GL >= N1 lanes, lane k < N1 (act) owns node k of every element; the other lanes
// hold a copy of node N1 - 1 and store nothing.
template <int N1, int GL>
struct SweepCtx {
  u64x* X;             // x [3][L]
  u64x* B;             // b [3][L]
  unsigned char* E;    // two exchange slots of 32 N1 + 16 bytes
  u64x* A;             // wave speed of face e (0 .. NeZ)
  u64x* J;             // pot = RHOT/DENS, wt = MOMZ/DENS, dpd = dP/dRHOT, private planes
  size_t pn, pb, ps;   // plane size; the lane's entry of element 0; stride of one element
  int k, NeZ, L;
  bool act;
  __device__ size_t pi(int v, int e) const { return (size_t)v * pn + pb + (size_t)e * ps; }
};

// One sweep x <- (1 - w) x + w (b - K x), from x = w b if first, stored for the columns in `run` (bit 0: A, 1: B); returns
// the lane's largest weighted change in each column.  (A NaN can drop out of the change; the FP64 residual that follows the sweeps looks at every node.)
template <int N1, int GL>
__device__ __forceinline__ float2 sweep(const SweepCtx<N1, GL>& c, const u64x (&Dk)[N1], const u64x (&Tk)[N1],
                                       u64x facB, u64x facT, u64x w, u64x w1, float c1, float c2, bool first, int run) {
  constexpr int N = N1 - 1;
  constexpr u64x SG = 0x8000000080000000ull;
  const int L = c.L, NeZ = c.NeZ;
  constexpr int SLOT = 32 * N1 + 16;
  u64x xn[3], jn[3];  // x and the Jacobian quantities of the element ahead
  auto load = [&](int e) {
#pragma unroll
    for (int v = 0; v < 3; ++v) jn[v] = c.J[c.pi(v, e)];
  };
  auto put = [&](int e) {  // quantities of element e into its slot
    unsigned char* s = c.E + (e & 1) * SLOT;
    const int k = c.k, l = e * N1 + k;
#pragma unroll
    for (int v = 0; v < 3; ++v) xn[v] = first ? xmul(w, c.B[v * L + l]) : c.X[v * L + l];
    const u64x p = xmul(jn[2], xn[2]);
    const u64x t = xfma(jn[0], xfma(jn[1], xn[0] ^ SG, xn[1]), xmul(jn[1], xn[2]));
    if (GL > N1 && !c.act) return;
    ulonglong2* q = reinterpret_cast<ulonglong2*>(s + 32 * k);
    q[0] = make_ulonglong2(xn[0], xn[1]);
    q[1] = make_ulonglong2(p, t);
    if (c.k == 0) *reinterpret_cast<u64x*>(s + 32 * N1) = xn[2];
    if (c.k == N1 - 1) *reinterpret_cast<u64x*>(s + 32 * N1 + 8) = xn[2];
  };
  load(0);
  put(0);
  if (NeZ > 1) load(1);
  const u64x upd = (run & 1 ? 0xffffffffull : 0ull) | (run & 2 ? 0xffffffffull << 32 : 0ull);  // columns to store
  u64x pr = 0, pm = 0, pp = 0, pt = 0, ph = 0;  // node N of the element below
  float2 dmax = make_float2(0.f, 0.f);
  for (int e = 0; e < NeZ; ++e) {
    u64x xo[3], be[3];  // this element's x and b
#pragma unroll
    for (int v = 0; v < 3; ++v) {
      xo[v] = xn[v];
      be[v] = c.B[v * L + e * N1 + c.k];
    }
    if (e + 1 < NeZ) {
      put(e + 1);
      if (e + 2 < NeZ) load(e + 2);
    }
    __syncwarp();
    const unsigned char* s = c.E + (e & 1) * SLOT;
    u64x y0 = 0, y1 = 0, y2 = 0, z1 = 0;
    u64x r0, m0, p0, t0, rN, mN, pN, tN;
#pragma unroll
    for (int m = 0; m < N1; ++m) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(s + 32 * m);
      const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(s + 32 * m + 16);
      y0 = xfma(Dk[m], a.y, y0);
      z1 = xfma(Tk[m], a.x, z1);
      y1 = xfma(Dk[m], b.x, y1);
      y2 = xfma(Dk[m], b.y, y2);
      if (m == 0) { r0 = a.x; m0 = a.y; p0 = b.x; t0 = b.y; }
      if (m == N) { rN = a.x; mN = a.y; pN = b.x; tN = b.y; }
    }
    const u64x h0 = *reinterpret_cast<const u64x*>(s + 32 * N1), hN = *reinterpret_cast<const u64x*>(s + 32 * N1 + 8);
    {  // bottom face (nz = -1); a slip lid reflects MOMZ and the heat flux
      u64x dr = xsub(r0, pr), dm = xsub(m0, pm), dp = xsub(p0, pp), dt = xsub(t0, pt), dh = xsub(h0, ph);
      if (e == 0) { dr = dp = dh = 0; dm = xadd(m0, m0); dt = xadd(t0, t0); }
      const u64x al = c.A[e], f0 = xfma(al, dr, dm), f1 = xfma(al, dm, dp), f2 = xfma(al, dh, dt);
      y0 = xfma(facB, f0, y0);
      y1 = xfma(facB, f1, y1);
      y2 = xfma(facB, f2, y2);
    }
    {  // top face (nz = +1)
      u64x dr, dm, dp, dt, dh;
      if (e + 1 < NeZ) {
        const unsigned char* sn = c.E + ((e + 1) & 1) * SLOT;
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(sn);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(sn + 16);
        const u64x hn = *reinterpret_cast<const u64x*>(sn + 32 * N1);
        dr = xsub(rN, a.x); dm = xsub(a.y, mN); dp = xsub(b.x, pN); dt = xsub(b.y, tN); dh = xsub(hN, hn);
      } else {
        dr = dp = dh = 0;
        dm = xadd(mN, mN) ^ SG;
        dt = xadd(tN, tN) ^ SG;
      }
      const u64x al = c.A[e + 1], f0 = xfma(al, dr, dm), f1 = xfma(al, dm ^ SG, dp), f2 = xfma(al, dh, dt);
      y0 = xfma(facT, f0, y0);
      y1 = xfma(facT, f1, y1);
      y2 = xfma(facT, f2, y2);
    }
    pr = rN; pm = mN; pp = pN; pt = tN; ph = hN;
    const int l = e * N1 + c.k;
    const u64x nr = xfma(w, xsub(be[0], y0), xmul(w1, xo[0]));
    const u64x nm = xfma(w, xsub(be[1], xadd(y1, z1)), xmul(w1, xo[1]));
    const u64x nh = xfma(w, xsub(be[2], y2), xmul(w1, xo[2]));
    if (GL == N1 || c.act) {  // a column that has stopped keeps its x
      c.X[l] = (nr & upd) | (xo[0] & ~upd);
      c.X[L + l] = (nm & upd) | (xo[1] & ~upd);
      c.X[2 * L + l] = (nh & upd) | (xo[2] & ~upd);
    }
    const float2 a = unpk(xsub(nr, xo[0])), b = unpk(xsub(nm, xo[1])), d = unpk(xsub(nh, xo[2]));
    dmax.x = fmaxf(dmax.x, fmaxf(fmaxf(fabsf(a.x), c1 * fabsf(b.x)), c2 * fabsf(d.x)));
    dmax.y = fmaxf(dmax.y, fmaxf(fmaxf(fabsf(a.y), c1 * fabsf(b.y)), c2 * fabsf(d.y)));
    __syncwarp();
  }
  return dmax;
}

// relaxation of the two columns' sweeps: w from the wave speed of each one's lowest face
template <int N1>
struct SweepCoef {
  u64x w, w1;
  float2 wr;
  __device__ __forceinline__ SweepCoef(const Ops& op, double impl_fac, u64x a0) {
    const float2 a = unpk(a0);
    const float f = 0.5f * (float)impl_fac * (float)op.Lb[0] * (float)op.FSz;
    wr = make_float2(1.f / (1.f + f * a.x), 1.f / (1.f + f * a.y));
    w = pk(wr.x, wr.y);
    w1 = pk(1.f - wr.x, 1.f - wr.y);
  }
};

// Sweeps from x = w b until the change that the next one would make (the last change times the observed
// contraction) is below rel times the first change.  bmax: the columns' largest weighted |b| (weights 1, c1, c2).  The
// change falls in beats (K's spectrum is complex), so it is held against a geometric envelope, not step to step: above
// 4 SWEEP_RATE^n of the first change the column's sweeps end and it is left to block LU.  At FP32's floor (a
// small change that falls no more) the result stands.  Each column in `run` (bit 0: A, 1: B) stops by itself, so its x
// does not depend on the warp's other columns; returns those that came to the end, uniform over a pair's lanes.
constexpr float SWEEP_RATE = 0.65f;
struct SweepStop {
  float d0, stop, prev, env;
  __device__ __forceinline__ SweepStop(float wr, float bmax, float rel) : d0(wr * bmax), stop(rel * d0), prev(d0), env(4.f * d0) {}
  // 0: go on, 1: done, 2: given up
  __device__ __forceinline__ int step(float d) {
    const float r = __fdividef(d, prev);
    prev = d;
    env *= SWEEP_RATE;
    if (d * r <= stop || (!(r <= 0.8f) && d <= 1.0e-4f * d0)) return 1;
    return d <= env ? 0 : 2;
  }
};
template <int N1, int GL>
__device__ __forceinline__ int sweeps(const SweepCtx<N1, GL>& c, const SweepCoef<N1>& sc, const Ops& op, double impl_fac,
                                      float2 bmax, float2 rel, float c1, float c2, int run) {
  const int k = c.k;
  const float fi = (float)impl_fac;
  const float fdzs = (float)op.E33 * fi;
  u64x Dk[N1], Tk[N1];
#pragma unroll
  for (int m = 0; m < N1; ++m) {
    Dk[m] = pk1(fdzs * (float)op.D[k * N1 + m]);
    Tk[m] = pk1(fi * (float)op.grav * (float)op.T[k * N1 + m]);
  }
  const u64x facB = pk1(0.5f * fi * (float)op.Lb[k] * (float)op.FSz);
  const u64x facT = pk1(0.5f * fi * (float)op.Lt[k] * (float)op.FSz);
  SweepStop sa(sc.wr.x, bmax.x, rel.x), sb(sc.wr.y, bmax.y, rel.y);
  int ok = 0;
  for (int n = 0; n < 32; ++n) {
    const float2 d = sweep<N1, GL>(c, Dk, Tk, facB, facT, sc.w, sc.w1, c1, c2, n == 0, run);
    const int a = sa.step(pair_max_bits<GL>(__float_as_uint(d.x))), b = sb.step(pair_max_bits<GL>(__float_as_uint(d.y)));
    ok |= run & ((a == 1 ? 1 : 0) | (b == 1 ? 2 : 0));
    run &= (a == 0 ? 1 : 0) | (b == 0 ? 2 : 0);
    if (!__any_sync(FULL, run)) break;
  }
  return ok;
}

}  // namespace
}  // namespace fedg
