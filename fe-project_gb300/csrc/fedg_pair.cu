// fedg_pair.cu -- the explicit stage kernels of the float-pair precision mode (FEDG_PREC_PAIR).
//
// Same algorithm and fusion as k_stage_mixed (fedg_mixed.cu), with every quantity that carries
// the solution kept as an unevaluated float pair (hi + lo, fedg_f2.cuh):
//   - the deviation state and pressure deviation;
//   - the 15 flux components and the Rusanov face fluxes;
//   - the Dx/Dy/Dz contractions (compensated sums of exact products) and the Lift;
//   - the RK accumulators and the modal filter.
// Only the Rusanov wave speed and the reference-wind velocities inside it stay FP32: they
// multiply face jumps, which are small against the fields.
//
// Why the mode exists: in FP32, the rounding of a flux value is amplified by the DG derivative,
// whose row norms grow like N^2/h.  Relative to the tendency the error is about
// 6e-8 N^2 |F| / |dF| per stage, where dF is the flux variation across one element.  On strong
// flows (a -15 K density current at p = 7) that drifts from FP64 by ~4e-8 of the state per step.
// Pairs bring the same amplification down to ~1e-14.
//
// Layout: one thread owns the two nodes (i, j, k) and (i, j, k + N1/2) of an element and carries both
// in the packed pair arithmetic of fedg_p2.cuh, so an element takes Np/2 threads and two blocks of
// 256 threads share an SM at p = 7.  Shared memory holds each field as 16-byte entries (hi of both
// nodes, lo of both nodes).  The x and y contractions read one entry per term; along z an entry holds
// two terms of the same line.  All three directions and the Lift accumulate into one compensated sum
// per variable, with the metric factors multiplied into the operator tables on the host.  A face node
// takes its own side's normal flux from the volume fluxes and computes the neighbour's side only in
// the face's direction (one warp per face at p = 7).
//
// What bounds it: the FP32 pipe (62 % of its cycles at p = 7, 24x24x12 elements; issue slots 49 %), then
// the barriers between the volume fluxes, the faces and the Lift.  With one node per thread, scalar
// pairs and one 512-thread block per SM the same pipe was 44 % busy.  HEVE step (three launches) at
// p = 7, 45x37x13 elements: 7.25 -> 4.95 ms.  The derivative loops stay rolled (unrolled, the code
// misses the instruction caches: 5.5 ms), and an L2 prefetch of the following block's fields, which the
// one-block form needed, costs 2-3 % here: the SM's second block already covers a block's first loads.
//
// FElib counterparts: cal_tend for HEVI (FElib/src/atmosphere/dynamics/
// scale_atm_dyn_dgm_nonhydro3d_rhot_hevi.F90:289-482), the HEVI numerical flux
// (scale_atm_dyn_dgm_nonhydro3d_rhot_hevi_numflux.F90:232-418), the implicit operator at var0
// (scale_atm_dyn_dgm_nonhydro3d_hevi_common_2.F90:1016-1328), timeint_rk (FElib/src/common/
// scale_timeint_rk.F90:2201-2565) and the modal filter (scale_atm_dyn_dgm_modalfilter.F90:49-130);
// with HEVE = true, cal_tend for HEVE (…_rhot_heve.F90:292-489), its numerical flux
// (…_rhot_heve_numflux.F90:946-1139) and the SSP-RK3 stages (scale_timeint_rk.F90:1182-1278).
// The sponge layer (…_dgm_spongelayer.F90:134-219) is added to the explicit tendency when a
// profile is given.
#include "fedg_ctx.cuh"
#include "fedg_mixed.cuh"
#include "fedg_p2.cuh"

namespace fedg {
namespace {

__device__ __forceinline__ p2 ld2(const float2* p, size_t a, size_t b) { return p2_of(__ldg(p + a), __ldg(p + b)); }
__device__ __forceinline__ void st2(float2* p, size_t a, size_t b, p2 v) {
  const float2 h = unpk(v.h), l = unpk(v.l);
  p[a] = make_float2(h.x, l.x);
  p[b] = make_float2(h.y, l.y);
}
__device__ __forceinline__ double to64(f2 v) { return (double)v.h + (double)v.l; }

// pressure deviation PRES_hyd ((1 + DRHOT/THERM_hyd)^kappa - 1): leading term in pairs, the rest
// of the binomial series in FP32 (relative size |r|), pow() in FP64 beyond rmax
__device__ __noinline__ f2 dpres_pow(float rh, float rl, double kap64) {
  return f2_split(pow(1.0 + ((double)rh + (double)rl), kap64) - 1.0);
}
__device__ __forceinline__ p2 dpres2(const OpsP& o, p2 dr, p2 rth, p2 ph) {
  const p2 r = dr * rth;
  u64x tl = pk1(o.cb[11]);
#pragma unroll
  for (int m = 10; m >= 1; --m) tl = xfma(tl, r.h, pk1(o.cb[m]));
  p2 S = p2_add_x(p2_dup(o.kap) * r, xmul(xmul(r.h, r.h), tl));
  const float2 rh = unpk(r.h);
  if (!(fabsf(rh.x) <= o.rmax && fabsf(rh.y) <= o.rmax)) {
    const float2 rl = unpk(r.l);
    f2 a = p2_a(S), b = p2_b(S);
    if (!(fabsf(rh.x) <= o.rmax)) a = dpres_pow(rh.x, rl.x, o.kap64);
    if (!(fabsf(rh.y) <= o.rmax)) b = dpres_pow(rh.y, rl.y, o.kap64);
    S = p2_of(a, b);
  }
  return ph * S;
}

// operator tables of one block in shared memory, built from OpsP: entries for the lane's row of D
// along x and y with both halves equal, and for the rows k and k + H along z
template <int N1>
struct Tab {
  static constexpr int H = N1 / 2;
  p2m dx[N1 * N1], dy[N1 * N1];              // [l][i]: metric times D(i, l)
  p2m dz[N1 * H], tg[N1 * H];                // [l][k]: rows k, k + H; tg: grav times VPOrdM1
  p2m lxb[N1], lxt[N1], lyb[N1], lyt[N1];    // Fscale/2 times the Lift of the -1 and +1 faces
  p2m lzb[H], lzt[H];
};
template <int N1>
struct TabF {  // modal filter, stage 3
  static constexpr int H = N1 / 2;
  p2m f[N1 * N1], fz[N1 * H];
};

template <int N1, bool LAST>
__device__ __forceinline__ void fill_tables(const OpsP& op, Tab<N1>& T, TabF<N1>* F) {
  constexpr int H = N1 / 2;
  for (int e = threadIdx.x; e < N1 * N1; e += blockDim.x) {
    const int l = e / N1, r = e % N1;
    st(T.dx[e], p2_dup(op.Dx[r * N1 + l]));
    st(T.dy[e], p2_dup(op.Dy[r * N1 + l]));
    if (LAST) st(F->f[e], p2_dup(op.F[r * N1 + l]));
    if (r < H) {
      st(T.dz[l * H + r], p2_of(op.Dz[r * N1 + l], op.Dz[(r + H) * N1 + l]));
      st(T.tg[l * H + r], p2_of(op.Tg[r * N1 + l], op.Tg[(r + H) * N1 + l]));
      if (LAST) st(F->fz[l * H + r], p2_of(op.Fv[r * N1 + l], op.Fv[(r + H) * N1 + l]));
    }
  }
  for (int e = threadIdx.x; e < N1; e += blockDim.x) {
    st(T.lxb[e], p2_dup(op.Lxb[e]));
    st(T.lxt[e], p2_dup(op.Lxt[e]));
    st(T.lyb[e], p2_dup(op.Lyb[e]));
    st(T.lyt[e], p2_dup(op.Lyt[e]));
    if (e < H) {
      st(T.lzb[e], p2_of(op.Lzb[e], op.Lzb[e + H]));
      st(T.lzt[e], p2_of(op.Lzt[e], op.Lzt[e + H]));
    }
  }
}

// shared memory of one element
template <int N1, bool IMP>
struct ElemSm {
  static constexpr int NH = N1 * N1 * N1 / 2, NF = N1 * N1;
  p2m st[6 * NH];             // deviation state and pressure deviation
  p2m fl[15 * NH];            // volume fluxes [direction * 5 + variable]
  p2m df[5 * 4 * (NF / 2)];   // lateral face fluxes [variable][face][a + N1 b], nodes b and b + H
  float2 dz[5 * 2 * NF];      // bottom and top face fluxes
  float2 di[IMP ? 5 * 2 * NF : 1];  // vertical faces of the implicit operator
};

// one variable's filtered output in the three passes of the modal filter; q^{n+1} = ref + F(dev)
template <int N1>
__device__ __forceinline__ void filter_store(const TabF<N1>& F, p2m* fa, p2m* fb, const p2 (&ref)[5],
                                             const StagePairBufs& B, size_t gA, size_t gB, bool valid, int i, int j,
                                             int k, int t) {
  constexpr int NF = N1 * N1, H = N1 / 2, NH = NF * H;
  __syncthreads();
  p2acc s[5];
#pragma unroll 1
  for (int l = 0; l < N1; ++l) {
    const p2 f = ld(F.f[l * N1 + i]);
#pragma unroll
    for (int v = 0; v < 5; ++v) s[v].add(f, ld(fa[v * NH + l + N1 * j + NF * k]));
  }
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    st(fb[v * NH + t], s[v].get());
    s[v] = p2acc{};
  }
  __syncthreads();
#pragma unroll 1
  for (int l = 0; l < N1; ++l) {
    const p2 f = ld(F.f[l * N1 + j]);
#pragma unroll
    for (int v = 0; v < 5; ++v) s[v].add(f, ld(fb[v * NH + i + N1 * l + NF * k]));
  }
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    st(fa[v * NH + t], s[v].get());
    s[v] = p2acc{};
  }
  __syncthreads();
#pragma unroll 1
  for (int l = 0; l < H; ++l) {
    const p2 f0 = ld(F.fz[l * H + k]), f1 = ld(F.fz[(l + H) * H + k]);
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const p2 x = ld(fa[v * NH + i + N1 * j + NF * l]);
      s[v].add(f0, p2_dup(p2_a(x)));
      s[v].add(f1, p2_dup(p2_b(x)));
    }
  }
  if (!valid) return;
#pragma unroll
  for (int v = 0; v < 5; ++v) {
    const p2 fil = s[v].get();
    const p2 out = v == VMX || v == VMY ? ref[v] + fil : fil;
    const double a = to64(p2_a(out)), b = to64(p2_b(out));
    B.qn[v][gA] = a;
    B.qn[v][gB] = b;
    if (B.qh[0]) {
      B.qh[v][gA] = a;
      B.qh[v][gB] = b;
    }
    st2(B.qnf[v], gA, gB, fil);
  }
}

// HEVE: the explicit HEVE operator (heve.F90:292-489, heve_numflux.F90:946-1139: vertical DENS/RHOT
// fluxes, the vertical pressure gradient and -g VFilterPM1(DDENS) explicit, unmasked wave speed) with
// the SSP-RK3 low-storage update (timeint_rk.F90:1182-1278) in place of the IMEX ARK232 stages
template <int N1, int EPB, int MINB, int STAGE, bool HEVE = false>
__global__ void __launch_bounds__(EPB* N1* N1* N1 / 2, MINB)
    k_stage_pair(const __grid_constant__ OpsP op, const ProfP pf, const __grid_constant__ StagePairBufs B,
                 const PairCoef cf, int Ne, int filter_on, int ke0) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1, H = N1 / 2, NH = NF * H, N = N1 - 1, PF = NF / 2;
  constexpr bool IMP = !HEVE && STAGE == 1;       // the implicit operator at q^n too
  constexpr bool ZDT = HEVE || STAGE == 1;        // vertical DENS/RHOT fluxes are needed
  using Sm = ElemSm<N1, IMP>;
  extern __shared__ __align__(16) unsigned char smraw[];
  Tab<N1>& T = *reinterpret_cast<Tab<N1>*>(smraw);
  TabF<N1>* F = reinterpret_cast<TabF<N1>*>(smraw + sizeof(Tab<N1>));
  unsigned char* sm_el = smraw + sizeof(Tab<N1>) + (STAGE == 3 ? sizeof(TabF<N1>) : 0);
  const int le = threadIdx.x / NH, t = threadIdx.x - le * NH;
  const int ke = ke0 + blockIdx.x * EPB + le;  // elements [ke0, Ne)
  const bool valid = ke < Ne;
  const int i = t % N1, j = (t / N1) % N1, k = t / NF;  // nodes k and k + H
  const int nxy = op.NeX * op.NeY;
  const int ez = valid ? ke / nxy : 0;
  const int ey = valid ? (ke - ez * nxy) / op.NeX : 0;
  const int ex = valid ? ke - ez * nxy - ey * op.NeX : 0;
  Sm& sm = reinterpret_cast<Sm*>(sm_el)[le];
  const size_t gA = (size_t)ke * Np + t, gB = gA + NH;
  const int levA = ez * N1 + k, levB = levA + H;
  const p2 U = p2_dup(op.Uref), V = p2_dup(op.Vref);

  fill_tables<N1, STAGE == 3>(op, T, F);
  const p2 dh = ld2(pf.dh, levA, levB);
  if (valid) {
    const p2 dd = ld2(B.qs[VD], gA, gB), mx = ld2(B.qs[VMX], gA, gB), my = ld2(B.qs[VMY], gA, gB);
    const p2 mz = ld2(B.qs[VMZ], gA, gB), dr = ld2(B.qs[VRT], gA, gB);
    const p2 dp = dpres2(op, dr, ld2(pf.rth, levA, levB), ld2(pf.ph, levA, levB));
    st(sm.st[VD * NH + t], dd);
    st(sm.st[VMX * NH + t], mx);
    st(sm.st[VMY * NH + t], my);
    st(sm.st[VMZ * NH + t], mz);
    st(sm.st[VRT * NH + t], dr);
    st(sm.st[5 * NH + t], dp);
    const p2 rd = p2_recip(dd + dh);
    const p2 ptr = ld2(pf.ptr, levA, levB);
    const p2 ptd = (dr - ptr * dd) * rd, pt = ptr + ptd;
    const p2 ud = (mx - U * dd) * rd, vd = (my - V * dd) * rd;
    const p2 u = U + ud, v = V + vd, w = mz * rd;
    auto put = [&](int dir, int var, p2 x) { st(sm.fl[(dir * 5 + var) * NH + t], x); };
    {
      const p2 R = dh * U;
      put(0, VD, mx);
      put(0, VRT, R * ptd + mx * pt);
      put(0, VMZ, (R + mx) * w);
      put(0, VMX, R * ud + mx * u + dp);
      put(0, VMY, R * vd + mx * v);
    }
    {
      const p2 R = dh * V;
      put(1, VD, my);
      put(1, VRT, R * ptd + my * pt);
      put(1, VMZ, (R + my) * w);
      put(1, VMX, R * ud + my * u);
      put(1, VMY, R * vd + my * v + dp);
    }
    if (ZDT) {
      put(2, VD, mz);
      put(2, VRT, mz * pt);
    }
    put(2, VMZ, HEVE ? mz * w + dp : mz * w);
    put(2, VMX, mz * u);
    put(2, VMY, mz * v);
  }
  __syncthreads();

  // --- Rusanov face flux, own side minus neighbour in pairs (wave speed in FP32); two face nodes per
  // pass: (a, b) and (a, b + H) ---
  if (valid) {
    const float gamm = op.kap.x;
    for (int task = t; task < 6 * PF; task += NH) {
      const int f = task / PF, ab = task - f * PF, a = ab % N1, b = ab / N1;
      const bool vert = f >= 4, isx = (f & 1) != 0;
      const int dir = vert ? 2 : (isx ? 0 : 1);
      const float sg = (f == 1 || f == 2 || f == 5) ? 1.f : -1.f;
      // own side: entry of the two nodes (lateral), or node a, b (+H) of the bottom / top plane
      const int e = vert ? a + N1 * b + (f == 5 ? NF * (H - 1) : 0) : (isx ? (f == 1 ? N : 0) + N1 * a : a + (f == 2 ? N1 * N : 0)) + NF * b;
      auto own = [&](const p2m* s) -> p2 {
        if (!vert) return ld(s[e]);
        const float* x = reinterpret_cast<const float*>(s + e) + (f == 5 ? 1 : 0);
        return p2{pk(x[0], x[4 * N1 * H]), pk(x[2], x[2 + 4 * N1 * H])};
      };
      // exterior side: neighbour element, or the own node with MOMZ reflected at a lid
      long kn;
      switch (f) {
        case 0: kn = (long)ke + (ey > 0 ? -op.NeX : (op.NeY - 1) * op.NeX); break;
        case 1: kn = (long)ke + (ex < op.NeX - 1 ? 1 : -(op.NeX - 1)); break;
        case 2: kn = (long)ke + (ey < op.NeY - 1 ? op.NeX : -(op.NeY - 1) * op.NeX); break;
        case 3: kn = (long)ke + (ex > 0 ? -1 : op.NeX - 1); break;
        case 4: kn = ez > 0 ? (long)ke - nxy : -1; break;
        default: kn = ez < op.NeZ - 1 ? (long)ke + nxy : -1; break;
      }
      const bool lid = kn < 0;
      const int plM = f == 5 ? N : 0;                    // own plane of a vertical face
      const int plP = lid ? plM : (f == 5 ? 0 : N);
      const int lM0 = vert ? ez * N1 + plM : ez * N1 + b, lM1 = vert ? lM0 : lM0 + H;
      const int lP0 = vert ? (lid ? lM0 : (f == 5 ? lM0 + 1 : lM0 - 1)) : lM0, lP1 = vert ? lP0 : lM1;
      size_t gP = (size_t)(lid ? ke : kn) * Np;
      if (vert) gP += a + N1 * b + NF * plP;
      else if (isx) gP += (f == 1 ? 0 : N) + N1 * a + NF * b;
      else gP += a + (f == 2 ? 0 : N1 * N) + NF * b;
      const size_t gP1 = gP + (vert ? N1 * H : NF * H);
      p2 ddP, mxP, myP, mzP, drP;
      // a boundary of a decomposed mesh: the exterior face layer comes from the halo exchange
      const int hsd = halo_side(f, ex, ey, op.NeX, op.NeY);
      const float2* hxs = hsd >= 0 ? op.hx[hsd] : nullptr;
      if (hxs) {
        const size_t per = halo_stride(hsd, op.NeX, op.NeY, op.NeZ, NF), h0 = halo_index(hsd, ex, ey, ez, ab, op.NeX, op.NeY, NF);
        const size_t h1 = h0 + N1 * H;
        ddP = ld2(hxs, h0, h1); mxP = ld2(hxs + per, h0, h1); myP = ld2(hxs + 2 * per, h0, h1);
        mzP = ld2(hxs + 3 * per, h0, h1); drP = ld2(hxs + 4 * per, h0, h1);
      } else {
        ddP = ld2(B.qs[VD], gP, gP1); mxP = ld2(B.qs[VMX], gP, gP1); myP = ld2(B.qs[VMY], gP, gP1);
        mzP = ld2(B.qs[VMZ], gP, gP1); drP = ld2(B.qs[VRT], gP, gP1);
        if (lid) mzP = p2_neg(mzP);
      }
      const p2 dhM = ld2(pf.dh, lM0, lM1), dhP = ld2(pf.dh, lP0, lP1), ptrP = ld2(pf.ptr, lP0, lP1);
      const p2 dpP = dpres2(op, drP, ld2(pf.rth, lP0, lP1), ld2(pf.ph, lP0, lP1));
      const p2 ddM = own(sm.st + VD * NH), dpM = own(sm.st + 5 * NH);
      const p2 rdM = p2_recip(ddM + dhM), rdP = p2_recip(ddP + dhP);
      const p2 udP = (mxP - U * ddP) * rdP, vdP = (myP - V * ddP) * rdP;
      const p2 uP = U + udP, vP = V + vdP, wP = mzP * rdP;
      const p2 ptdP = (drP - ptrP * ddP) * rdP, ptP = ptrP + ptdP;
      const p2 jdd = ddP - ddM, jdr = drP - own(sm.st + VRT * NH);
      const p2 jmx = mxP - own(sm.st + VMX * NH), jmy = myP - own(sm.st + VMY * NH), jmz = mzP - own(sm.st + VMZ * NH);
      // normal velocities (leading parts) and the exterior side's normal fluxes
      float2 vnM, vnP;
      p2 fD, fT, fX, fY, fZ;
      if (vert) {
        vnM = unpk((own(sm.st + VMZ * NH) * rdM).h);
        vnP = unpk(wP.h);
        fD = mzP;
        fT = mzP * ptP;
        fX = mzP * uP;
        fY = mzP * vP;
        fZ = HEVE ? mzP * wP + dpP : mzP * wP;
      } else {
        const p2 Wn = isx ? U : V, mnP = isx ? mxP : myP, R = dhP * Wn;
        vnM = unpk((Wn + (own(sm.st + (isx ? VMX : VMY) * NH) - Wn * ddM) * rdM).h);
        vnP = unpk(isx ? uP.h : vP.h);
        fD = mnP;
        fT = R * ptdP + mnP * ptP;
        fZ = (R + mnP) * wP;
        fX = R * udP + mnP * uP;
        fY = R * vdP + mnP * vP;
        if (isx) fX = fX + dpP;
        else fY = fY + dpP;
      }
      const float2 dpMh = unpk(dpM.h), dpPh = unpk(dpP.h), rMh = unpk(rdM.h), rPh = unpk(rdP.h);
      const float csM0 = sqrtf(gamm * (__ldg(pf.phf + lM0) + dpMh.x) * rMh.x), csM1 = sqrtf(gamm * (__ldg(pf.phf + lM1) + dpMh.y) * rMh.y);
      const float csP0 = sqrtf(gamm * (__ldg(pf.phf + lP0) + dpPh.x) * rPh.x), csP1 = sqrtf(gamm * (__ldg(pf.phf + lP1) + dpPh.y) * rPh.y);
      const u64x al = pk(fmaxf(csM0 + fabsf(vnM.x), csP0 + fabsf(vnP.x)), fmaxf(csM1 + fabsf(vnM.y), csP1 + fabsf(vnP.y)));
      const u64x sg2 = pk1(sg);
      const p2m* flM = sm.fl + dir * 5 * NH;
      auto jump = [&](p2 fP, int var) { return p2_scale(fP - own(flM + var * NH), sg2); };
      if (!vert) {
        p2m* o = sm.df + f * PF + ab;
        constexpr int S = 4 * PF;
        st(o[VD * S], jump(fD, VD) - p2_mul_x(jdd, al));
        st(o[VRT * S], jump(fT, VRT) - p2_mul_x(jdr, al));
        st(o[VMZ * S], jump(fZ, VMZ) - p2_mul_x(jmz, al));
        st(o[VMX * S], jump(fX, VMX) - p2_mul_x(jmx, al));
        st(o[VMY * S], jump(fY, VMY) - p2_mul_x(jmy, al));
      } else {
        auto putz = [&](float2* s, int var, p2 x) {
          float2* o = s + (var * 2 + (f - 4)) * NF + ab;
          st2(o, 0, N1 * H, x);
        };
        if (HEVE) {
          putz(sm.dz, VD, jump(fD, VD) - p2_mul_x(jdd, al));
          putz(sm.dz, VRT, jump(fT, VRT) - p2_mul_x(jdr, al));
          putz(sm.dz, VMZ, jump(fZ, VMZ) - p2_mul_x(jmz, al));
          putz(sm.dz, VMX, jump(fX, VMX) - p2_mul_x(jmx, al));
          putz(sm.dz, VMY, jump(fY, VMY) - p2_mul_x(jmy, al));
        } else {  // HEVI: no vertical mass and RHOT flux, no vertical wave speed
          putz(sm.dz, VMZ, jump(fZ, VMZ));
          putz(sm.dz, VMX, jump(fX, VMX));
          putz(sm.dz, VMY, jump(fY, VMY));
        }
        if (IMP) {  // vertical faces of the implicit operator at var0 = q^n (hevi_common_2.F90:1016-1328)
          putz(sm.di, VD, p2_scale(jmz, sg2) - p2_mul_x(jdd, al));
          putz(sm.di, VMZ, p2_scale(dpP - dpM, sg2) - p2_mul_x(jmz, al));
          putz(sm.di, VRT, jump(fT, VRT) - p2_mul_x(jdr, al));
          putz(sm.di, VMX, p2_neg(p2_mul_x(jmx, al)));
          putz(sm.di, VMY, p2_neg(p2_mul_x(jmy, al)));
        }
      }
    }
  }
  // --- the derivative along x, y and z and the Lift, one compensated sum per variable; the
  // derivatives need the volume fluxes only, so they run before the barrier that completes the faces
  // (the loops stay rolled: the kernel's code competes for the instruction caches) ---
  const int col = i + N1 * j;
  p2acc s[5];
  if (valid) {
#pragma unroll 1
    for (int l = 0; l < N1; ++l) {
      const p2 dx = ld(T.dx[l * N1 + i]), dy = ld(T.dy[l * N1 + j]);
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        s[v].add(dx, ld(sm.fl[v * NH + l + N1 * j + NF * k]));
        s[v].add(dy, ld(sm.fl[(5 + v) * NH + i + N1 * l + NF * k]));
      }
    }
#pragma unroll 1
    for (int l = 0; l < H; ++l) {
      const p2 d0 = ld(T.dz[l * H + k]), d1 = ld(T.dz[(l + H) * H + k]);
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        if (!HEVE && (v == VD || v == VRT)) continue;
        const p2 z = ld(sm.fl[(10 + v) * NH + col + NF * l]);
        s[v].add(d0, p2_dup(p2_a(z)));
        s[v].add(d1, p2_dup(p2_b(z)));
      }
    }
    if (HEVE) {  // -g VFilterPM1(DDENS) (heve.F90:447-452)
#pragma unroll 1
      for (int l = 0; l < H; ++l) {
        const p2 z = ld(sm.st[VD * NH + col + NF * l]);
        s[VMZ].add(ld(T.tg[l * H + k]), p2_dup(p2_a(z)));
        s[VMZ].add(ld(T.tg[(l + H) * H + k]), p2_dup(p2_b(z)));
      }
    }
  }
  __syncthreads();

  p2 tex[5], tim[5];
  if (valid) {
    {
      const p2 lyb = ld(T.lyb[j]), lxt = ld(T.lxt[i]), lyt = ld(T.lyt[j]), lxb = ld(T.lxb[i]);
      const p2 lzb = ld(T.lzb[k]), lzt = ld(T.lzt[k]);
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        const p2m* d = sm.df + v * 4 * PF;
        s[v].add(lyb, ld(d[i + N1 * k]));
        s[v].add(lxt, ld(d[PF + j + N1 * k]));
        s[v].add(lyt, ld(d[2 * PF + i + N1 * k]));
        s[v].add(lxb, ld(d[3 * PF + j + N1 * k]));
        if (HEVE || (v != VD && v != VRT)) {
          s[v].add(lzb, p2_dup(sm.dz[v * 2 * NF + col]));
          s[v].add(lzt, p2_dup(sm.dz[(v * 2 + 1) * NF + col]));
        }
      }
    }
#pragma unroll
    for (int v = 0; v < 5; ++v) tex[v] = p2_neg(s[v].get());
    if (op.cor.x != 0.f || pf.sl) {
      const p2 mx = ld(sm.st[VMX * NH + t]) + dh * U, my = ld(sm.st[VMY * NH + t]) + dh * V;
      tex[VMX] = tex[VMX] + p2_dup(op.cor) * my;
      tex[VMY] = tex[VMY] - p2_dup(op.cor) * mx;
      if (pf.sl) {  // sponge layer on the explicit tendency (driver_nonhydro3d.F90:831-841)
        const p2 cz = ld2(pf.sl, levA, levB);
        tex[VMZ] = tex[VMZ] - cz * ld(sm.st[VMZ * NH + t]);
        if (pf.sl_h != 0.f) {
          tex[VMX] = tex[VMX] - cz * mx;
          tex[VMY] = tex[VMY] - cz * my;
        }
      }
    }
    if constexpr (IMP) {  // the implicit operator at q^n
      p2acc a[5];
      const p2 lzb = ld(T.lzb[k]), lzt = ld(T.lzt[k]);
#pragma unroll 1
      for (int l = 0; l < H; ++l) {
        const p2 d0 = ld(T.dz[l * H + k]), d1 = ld(T.dz[(l + H) * H + k]);
        const p2 g0 = ld(T.tg[l * H + k]), g1 = ld(T.tg[(l + H) * H + k]);
        const p2 m = ld(sm.fl[(10 + VD) * NH + col + NF * l]), r = ld(sm.fl[(10 + VRT) * NH + col + NF * l]);
        const p2 p = ld(sm.st[5 * NH + col + NF * l]), d = ld(sm.st[VD * NH + col + NF * l]);
        a[VD].add(d0, p2_dup(p2_a(m)));
        a[VD].add(d1, p2_dup(p2_b(m)));
        a[VRT].add(d0, p2_dup(p2_a(r)));
        a[VRT].add(d1, p2_dup(p2_b(r)));
        a[VMZ].add(d0, p2_dup(p2_a(p)));
        a[VMZ].add(d1, p2_dup(p2_b(p)));
        a[VMZ].add(g0, p2_dup(p2_a(d)));
        a[VMZ].add(g1, p2_dup(p2_b(d)));
      }
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        a[v].add(lzb, p2_dup(sm.di[v * 2 * NF + col]));
        a[v].add(lzt, p2_dup(sm.di[(v * 2 + 1) * NF + col]));
        tim[v] = p2_neg(a[v].get());
      }
      if (B.a0[0]) {
        st2(B.a0[0], gA, gB, tim[VD]);
        st2(B.a0[1], gA, gB, tim[VMZ]);
        st2(B.a0[2], gA, gB, tim[VRT]);
      }
    }
  }

  // --- fused RK epilogue in pairs ---
  auto qn64 = [&](int v) { return p2_split(__ldg(B.qn[v] + gA), __ldg(B.qn[v] + gB)); };
  if constexpr (HEVE) {
    // ERK_SSP_3s3o on the deviations (the reference state does not change in time): q1 = qn + dt t(qn),
    // q2 = 3/4 qn + 1/4 (q1 + dt t(q1)), q3 = 1/3 qn + 2/3 (q2 + dt t(q2)); the stage inputs and
    // outputs are deviation pairs, qn is split from the FP64 state
    if (STAGE < 3) {
      if (valid) {
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          const p2 up = ld(sm.st[v * NH + t]) + p2_dup(cf.dt) * tex[v];
          p2 dev = up;
          if (STAGE == 2) {
            p2 qnd = qn64(v);
            if (v == VMX || v == VMY) qnd = qnd - dh * (v == VMX ? U : V);
            dev = p2_dup(cf.ssp[0]) * qnd + p2_dup(cf.ssp[1]) * up;
          }
          st2(B.qi[v], gA, gB, dev);
        }
      }
      return;
    }
  }
  if constexpr (!HEVE && STAGE < 3) {
    float xqA[3] = {0.f, 0.f, 0.f}, xqB[3] = {0.f, 0.f, 0.f};
    if (valid) {
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        p2 qs;
        if (STAGE == 1) {
          qs = qn64(v) + (p2_dup(cf.q1e) * tex[v] + p2_dup(cf.q1i) * tim[v]);
          st2(B.S3[v], gA, gB, p2_dup(cf.s3e) * tex[v] + p2_dup(cf.s3i) * tim[v]);
          st2(B.SF[v], gA, gB, p2_dup(cf.sf1) * (tex[v] + tim[v]));
        } else {
          const p2 ti = ld2(B.TI[v], gA, gB);
          qs = qn64(v) + (ld2(B.S3[v], gA, gB) + p2_dup(cf.q2e) * tex[v] + p2_dup(cf.q2i) * ti);
          st2(B.SF[v], gA, gB, ld2(B.SF[v], gA, gB) + p2_dup(cf.sf2) * (tex[v] + ti));
        }
        st2(B.qi[v], gA, gB, qs);
        const int m = v == VD ? 0 : (v == VMZ ? 1 : (v == VRT ? 2 : -1));
        if (m >= 0) {
          xqA[m] = unpk(qs.h).x;
          xqB[m] = unpk(qs.h).y;
        }
      }
    }
    if (B.X) {  // the element's q* as feature rows of the guess network
      __syncthreads();
      __nv_bfloat16* sx = reinterpret_cast<__nv_bfloat16*>(sm.st);  // [NF][3][N1]
#pragma unroll
      for (int v = 0; v < 3; ++v) {
        sx[((i + N1 * j) * 3 + v) * N1 + k] = __float2bfloat16_rn(xqA[v] * B.xs[v]);
        sx[((i + N1 * j) * 3 + v) * N1 + k + H] = __float2bfloat16_rn(xqB[v] * B.xs[v]);
      }
      __syncthreads();
      if (valid) {
        for (int c = t; c < 3 * NF; c += NH) {
          const int cij = c / 3, v = c - 3 * cij;
          const size_t row = (size_t)(ex + op.NeX * ey) * NF + cij;
          __nv_bfloat16* dst = B.X + row * B.xdinp + v * op.L + ez * N1;
          if constexpr (N1 == 8) *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(sx + (cij * 3 + v) * N1);
          else *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(sx + (cij * 3 + v) * N1);
        }
      }
    }
    return;
  }
  if constexpr (STAGE == 3) {
    // q^{n+1}, then the modal filter (tensorprod3D_kernel.F90:2555-2618) of its deviation from the
    // reference state (DENS_hyd*(Uref, Vref) for MOMX/MOMY, 0 otherwise)
    p2 dev[5], ref[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) {
      const bool mom = v == VMX || v == VMY;
      ref[v] = mom ? dh * (v == VMX ? U : V) : p2_zero();
      dev[v] = p2_zero();
      if (!valid) continue;
      const p2 qn = qn64(v);
      if (HEVE) {
        const p2 up = ld(sm.st[v * NH + t]) + p2_dup(cf.dt) * tex[v];
        dev[v] = p2_dup(cf.ssp[2]) * (mom ? qn - ref[v] : qn) + p2_dup(cf.ssp[3]) * up;
      } else {
        const p2 qnew = qn + (ld2(B.SF[v], gA, gB) + p2_dup(cf.sf3) * (tex[v] + ld2(B.TI[v], gA, gB)));
        dev[v] = mom ? qnew - ref[v] : qnew;
      }
    }
    if (B.dtrc && valid) {  // DDENS_TRC: before the filter
      B.dtrc[gA] = to64(p2_a(dev[VD]));
      B.dtrc[gB] = to64(p2_b(dev[VD]));
    }
    if (!filter_on) {
      if (valid) {
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          const p2 out = v == VMX || v == VMY ? ref[v] + dev[v] : dev[v];
          const double a = to64(p2_a(out)), b = to64(p2_b(out));
          B.qn[v][gA] = a;
          B.qn[v][gB] = b;
          if (B.qh[0]) {
            B.qh[v][gA] = a;
            B.qh[v][gB] = b;
          }
          st2(B.qnf[v], gA, gB, dev[v]);
        }
      }
      return;
    }
    // every thread of the block is past its reads of the other nodes' state (HEVE reads it in the
    // gravity term above), and the own entries are read; the flux arrays are read until here
    __syncthreads();
#pragma unroll
    for (int v = 0; v < 5; ++v) st(sm.st[v * NH + t], dev[v]);
    filter_store<N1>(*F, sm.st, sm.fl, ref, B, gA, gB, valid, i, j, k, t);
  }
}

template <int N1>
constexpr int epb_p() { return N1 == 4 ? 2 : 1; }
template <int N1>
constexpr int minb_p() { return N1 == 4 ? 8 : 2; }

template <int N1, int STAGE, bool HEVE = false>
int launch_pair_n(const OpsP& op, const ProfP& pf, const StagePairBufs& B, const PairCoef& cf, int Ne, int filt,
                  cudaStream_t s, int ke0 = 0) {
  constexpr int EPB = epb_p<N1>(), Np = N1 * N1 * N1;
  constexpr size_t smem = sizeof(Tab<N1>) + (STAGE == 3 ? sizeof(TabF<N1>) : 0) + EPB * sizeof(ElemSm<N1, !HEVE && STAGE == 1>);
  auto kfn = k_stage_pair<N1, EPB, minb_p<N1>(), STAGE, HEVE>;
  cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (Ne <= ke0) return (int)cudaSuccess;
  kfn<<<(Ne - ke0 + EPB - 1) / EPB, EPB * Np / 2, smem, s>>>(op, pf, B, cf, Ne, filt, ke0);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_stage_pair_heve(int N1, int stage, const OpsP& op, const ProfP& pf, const StagePairBufs& B,
                           const PairCoef& cf, int Ne, int filt, cudaStream_t s) {
  if (N1 == 8) {
    if (stage == 1) return launch_pair_n<8, 1, true>(op, pf, B, cf, Ne, filt, s);
    if (stage == 2) return launch_pair_n<8, 2, true>(op, pf, B, cf, Ne, filt, s);
    return launch_pair_n<8, 3, true>(op, pf, B, cf, Ne, filt, s);
  }
  if (N1 == 4) {
    if (stage == 1) return launch_pair_n<4, 1, true>(op, pf, B, cf, Ne, filt, s);
    if (stage == 2) return launch_pair_n<4, 2, true>(op, pf, B, cf, Ne, filt, s);
    return launch_pair_n<4, 3, true>(op, pf, B, cf, Ne, filt, s);
  }
  return (int)cudaErrorInvalidValue;
}

int launch_stage_pair(int N1, int stage, const OpsP& op, const ProfP& pf, const StagePairBufs& B,
                      const PairCoef& cf, int Ne, int filt, cudaStream_t s, int ke0) {
  if (N1 == 8) {
    if (stage == 1) return launch_pair_n<8, 1>(op, pf, B, cf, Ne, filt, s, ke0);
    if (stage == 2) return launch_pair_n<8, 2>(op, pf, B, cf, Ne, filt, s, ke0);
    return launch_pair_n<8, 3>(op, pf, B, cf, Ne, filt, s, ke0);
  }
  if (N1 == 4) {
    if (stage == 1) return launch_pair_n<4, 1>(op, pf, B, cf, Ne, filt, s, ke0);
    if (stage == 2) return launch_pair_n<4, 2>(op, pf, B, cf, Ne, filt, s, ke0);
    return launch_pair_n<4, 3>(op, pf, B, cf, Ne, filt, s, ke0);
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace fedg
