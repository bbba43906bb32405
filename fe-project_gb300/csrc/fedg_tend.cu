// fedg_tend.cu -- explicit DG tendency (volume + Rusanov face flux + Lift), the modal
// filter and DRHOT->DPRES, FP64, one thread block per element (or per few elements).
//
// Restates, on the flat cube domain (Gsqrt = 1, GI3 = 0):
//   HEVE  FElib/src/fluid_dyn_solver/scale_atm_dyn_dgm_nonhydro3d_rhot_heve.F90:292-489
//         + Rusanov flux ..._rhot_heve_numflux.F90:946-1139
//   HEVI  ..._rhot_hevi.F90:289-482 + ..._rhot_hevi_numflux.F90:232-418
//   Div_var5 / Lift / VFilterPM1 of scale_element_operation_tensorprod3D(_kernel).F90
//   modal filter ..._dgm_modalfilter.F90:49-130, DRHOT2PRES ..._nonhydro3d_common.F90:428-479
//
// Data layout in HBM: five (Np, Ne) FP64 fields, node fastest -- the FElib layout, so a
// thread block reads each field of its element as one contiguous Np*8-byte run.
// Exterior states: periodic neighbours in x/y; at the lids the element's own state with
// MOMZ reflected (what FElib's halo copy + slip ApplyBC produce, dgm_bnd.F90:323-341).
#include "fedg_common.cuh"
#include "fedg_kernels.cuh"

namespace fedg {

// Modal filter of one field at node (i, j, k): value x in, filtered value out; a, b: Np doubles each of the
// element's shared memory.  All threads of the block call it.
template <int N1>
__device__ __forceinline__ double filter_node(const Ops& op, double* a, double* b, double x, int p, int i, int j, int k) {
  constexpr int NF = N1 * N1;
  a[p] = x;
  __syncthreads();
  double s = 0.0;
#pragma unroll
  for (int l = 0; l < N1; ++l) s = fma(op.F[i * N1 + l], a[p - i + l], s);
  b[p] = s;
  __syncthreads();
  s = 0.0;
#pragma unroll
  for (int l = 0; l < N1; ++l) s = fma(op.F[j * N1 + l], b[p + (l - j) * N1], s);
  a[p] = s;  // every thread's reads of a are before the last barrier
  __syncthreads();
  s = 0.0;
#pragma unroll
  for (int l = 0; l < N1; ++l) s = fma(op.Fv[k * N1 + l], a[p + (l - k) * NF], s);
  return s;
}

// Explicit tendency, or with SSP the whole stage of SSP-RK3.
//
// What bounds it: the FP64 pipe, two lane-instructions per clock and SM, so the kernel is built to need few of
// them: metric factors, signs and the Lift's 1/2 are in the tables of each block, a face takes its own side's
// flux from the volume fluxes and one reciprocal per exterior node, and a HEVI lid face (no pressure term, no
// dissipation) only the momentum flux.  HEVI tendency of 16x16x8 elements at p = 7: 568 -> 332 us (with the face state
// recomputed on both sides by divisions and the factors applied per node).
//
// SSP: the whole SSP-RK3 stage instead of the tendency -- q_new (and for the last stage the modal filter) into
// x.qn, DPRES of it into x.dpn; the neighbours still read q, so q_new is another buffer.  8x8x8 elements at p = 3: 20 us (FP64 pipe 83 % busy on the
// fullest SMs) against 10 + 24 + 6 us for the pressure, tendency and update kernels of that stage.
template <int N1, int EPB, bool HEVI, bool SSP>
__global__ void __launch_bounds__(EPB* N1* N1* N1, EPB* N1* N1* N1 > 256 ? 2 : 1)
    k_tend_fp64(const __grid_constant__ Ops op, const Prof pf, const F5c q, const double* __restrict__ dpres,
                const F5 t, const __grid_constant__ SspArgs x, int Ne) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1, N = N1 - 1, S = 6 * NF;
  extern __shared__ double sm[];
  double* s_d = sm;                        // [4][NF]  -E11 D, -E22 D, -E33 D, -grav VPOrdM1 (HEVE)
  double* s_l = s_d + 4 * NF;              // [6][N1]  Lift of face f with -Fscale/2 and the face normal's sign
  double* s_st = s_l + 6 * N1;             // [EPB][7][Np]   state, DPRES, 1/DENS
  double* s_fl = s_st + EPB * 7 * Np;      // [EPB][15][Np]  fluxes, c = dir*5 + var
  double* s_df = s_fl + EPB * 15 * Np;     // [EPB][5][6*NF] face flux differences
  const int tid = threadIdx.x;
  const int le = tid / Np, p = tid - le * Np;
  const int ke = blockIdx.x * EPB + le;
  const bool valid = ke < Ne;
  const int i = p % N1, j = (p / N1) % N1, k = p / NF;
  const int nxy = op.NeX * op.NeY;
  const int ez = valid ? ke / nxy : 0;
  const int ey = valid ? (ke - ez * nxy) / op.NeX : 0;
  const int ex = valid ? ke - ez * nxy - ey * op.NeX : 0;
  double* st = s_st + le * 7 * Np;
  double* fl = s_fl + le * 15 * Np;
  double* df = s_df + le * 5 * S;
  const size_t g = (size_t)ke * Np + p;
  const int lev = ez * N1 + k;

  for (int c = tid; c < NF; c += EPB * Np) {
    s_d[c] = -op.E11 * op.D[c];
    s_d[NF + c] = -op.E22 * op.D[c];
    s_d[2 * NF + c] = -op.E33 * op.D[c];
    s_d[3 * NF + c] = -op.grav * op.T[c];
    if (c < N1) {
      s_l[c] = 0.5 * op.FSy * op.Lb[c];
      s_l[N1 + c] = -0.5 * op.FSx * op.Lt[c];
      s_l[2 * N1 + c] = -0.5 * op.FSy * op.Lt[c];
      s_l[3 * N1 + c] = 0.5 * op.FSx * op.Lb[c];
      s_l[4 * N1 + c] = 0.5 * op.FSz * op.Lb[c];
      s_l[5 * N1 + c] = -0.5 * op.FSz * op.Lt[c];
    }
  }

  // --- volume fluxes (heve.F90:385-418 / hevi.F90:384-413) ---
  if (valid) {
    double qv[5];
#pragma unroll
    for (int v = 0; v < 5; ++v) qv[v] = __ldg(q.v[v] + g);
    const double dp = __ldg(dpres + g);
    const double mx = qv[VMX], my = qv[VMY], mz = qv[VMZ];
    const double r = 1.0 / (qv[VD] + __ldg(pf.dens + lev));
    const double pt = (__ldg(pf.therm + lev) + qv[VRT]) * r;
    const double u = mx * r, v = my * r, w = mz * r;
    const double uv = mx * v, uw = mx * w, vw = my * w;
#pragma unroll
    for (int c = 0; c < 5; ++c) st[c * Np + p] = qv[c];
    st[5 * Np + p] = dp;
    st[6 * Np + p] = r;
    fl[(0 * 5 + VD) * Np + p] = mx;
    fl[(1 * 5 + VD) * Np + p] = my;
    fl[(0 * 5 + VRT) * Np + p] = mx * pt;
    fl[(1 * 5 + VRT) * Np + p] = my * pt;
    fl[(0 * 5 + VMX) * Np + p] = fma(mx, u, dp);
    fl[(1 * 5 + VMX) * Np + p] = uv;
    fl[(2 * 5 + VMX) * Np + p] = uw;
    fl[(0 * 5 + VMY) * Np + p] = uv;
    fl[(1 * 5 + VMY) * Np + p] = fma(my, v, dp);
    fl[(2 * 5 + VMY) * Np + p] = vw;
    fl[(0 * 5 + VMZ) * Np + p] = uw;
    fl[(1 * 5 + VMZ) * Np + p] = vw;
    fl[(2 * 5 + VMZ) * Np + p] = HEVI ? mz * w : fma(mz, w, dp);
    if (!HEVI) {
      fl[(2 * 5 + VD) * Np + p] = mz;
      fl[(2 * 5 + VRT) * Np + p] = mz * pt;
    }
  }
  __syncthreads();

  // --- Rusanov face flux (numflux get_generalvc): F_n the flux along the face's axis, del_flux = n (F* - F^-)
  //     = n/2 ((F_n^+ - F_n^-) - n alpha (q^+ - q^-)), here without the n/2 ---
  if (valid) {
    const double gamm = op.kap;
    for (int fi = p; fi < 6 * NF; fi += Np) {
      const int f = fi / NF, ab = fi - f * NF, a = ab % N1, b = ab / N1;
      int iM, jM, kM;
      face_node<N1>(f, a, b, iM, jM, kM);
      const int pM = iM + N1 * jM + NF * kM;
      long kn;
      int levP = ez * N1 + kM;
      switch (f) {
        case 0: kn = (long)ke + (ey > 0 ? -op.NeX : (op.NeY - 1) * op.NeX); break;
        case 1: kn = (long)ke + (ex < op.NeX - 1 ? 1 : -(op.NeX - 1)); break;
        case 2: kn = (long)ke + (ey < op.NeY - 1 ? op.NeX : -(op.NeY - 1) * op.NeX); break;
        case 3: kn = (long)ke + (ex > 0 ? -1 : op.NeX - 1); break;
        case 4: kn = ez > 0 ? (long)ke - nxy : -1; levP = (ez - 1) * N1 + N; break;
        default: kn = ez < op.NeZ - 1 ? (long)ke + nxy : -1; levP = (ez + 1) * N1; break;
      }
      const int levM = ez * N1 + kM;
      const double mxM = st[VMX * Np + pM], myM = st[VMY * Np + pM], mzM = st[VMZ * Np + pM];
      double ddP, mxP, myP, mzP, drP, dpP;
      // a boundary of a decomposed mesh: the exterior face layer comes from the halo exchange
      const int hsd = halo_side(f, ex, ey, op.NeX, op.NeY);
      const double* hxs = hsd >= 0 ? op.hx[hsd] : nullptr;
      if (hxs) {
        const size_t per = halo_stride(hsd, op.NeX, op.NeY, op.NeZ, NF), h = halo_index(hsd, ex, ey, ez, ab, op.NeX, op.NeY, NF);
        ddP = __ldg(hxs + h); mxP = __ldg(hxs + per + h); myP = __ldg(hxs + 2 * per + h);
        mzP = __ldg(hxs + 3 * per + h); drP = __ldg(hxs + 4 * per + h); dpP = __ldg(hxs + 5 * per + h);
      } else if (kn >= 0) {
        int i2, j2, k2;
        face_node<N1>(face_opp(f), a, b, i2, j2, k2);
        const size_t gP = (size_t)kn * Np + i2 + N1 * j2 + NF * k2;
        ddP = __ldg(q.v[VD] + gP); mxP = __ldg(q.v[VMX] + gP); myP = __ldg(q.v[VMY] + gP);
        mzP = __ldg(q.v[VMZ] + gP); drP = __ldg(q.v[VRT] + gP); dpP = __ldg(dpres + gP);
      } else {  // slip lid
        levP = levM;
        ddP = st[VD * Np + pM]; mxP = mxM; myP = myM; mzP = -mzM; drP = st[VRT * Np + pM]; dpP = st[5 * Np + pM];
      }
      const int dir = f >= 4 ? 2 : (f & 1 ? 0 : 1);
      const double rP = 1.0 / (ddP + __ldg(pf.dens + levP));
      const double mnP = dir == 0 ? mxP : (dir == 1 ? myP : mzP);
      const double vP = mnP * rP;
      const double* fM = fl + dir * 5 * Np + pM;
      double* o = df + ab + f * NF;
      if (HEVI && f >= 4) {
        o[VMX * S] = fma(mxP, vP, -fM[VMX * Np]);
        o[VMY * S] = fma(myP, vP, -fM[VMY * Np]);
        o[VMZ * S] = fma(mzP, vP, -fM[VMZ * Np]);
      } else {
        const double ddM = st[VD * Np + pM], drM = st[VRT * Np + pM], dpM = st[5 * Np + pM], rM = st[6 * Np + pM];
        const double mnM = dir == 0 ? mxM : (dir == 1 ? myM : mzM);
        const double cM = sqrt(gamm * (__ldg(pf.pres + levM) + dpM) * rM), cP = sqrt(gamm * (__ldg(pf.pres + levP) + dpP) * rP);
        double alpha = fmax(fma(fabs(mnM), rM, cM), fma(fabs(mnP), rP, cP));
        if (f == 1 || f == 2 || f == 5) alpha = -alpha;  // -n alpha
        const double rtP = __ldg(pf.therm + levP) + drP;
        o[VD * S] = fma(alpha, ddP - ddM, mnP - fM[VD * Np]);
        o[VRT * S] = fma(alpha, drP - drM, fma(rtP, vP, -fM[VRT * Np]));
        o[VMX * S] = fma(alpha, mxP - mxM, fma(mxP, vP, dir == 0 ? dpP : 0.0) - fM[VMX * Np]);
        o[VMY * S] = fma(alpha, myP - myM, fma(myP, vP, dir == 1 ? dpP : 0.0) - fM[VMY * Np]);
        o[VMZ * S] = fma(alpha, mzP - mzM, fma(mzP, vP, dir == 2 && !HEVI ? dpP : 0.0) - fM[VMZ * Np]);
      }
    }
  }
  __syncthreads();

  // --- Div_var5 (D1D along x, y, z) + tensor-product Lift, combined (heve.F90:424-465) ---
  double out[5] = {};
  if (valid) {
#pragma unroll
    for (int dir = 0; dir < 3; ++dir) {
      const int row = dir == 0 ? i : (dir == 1 ? j : k), stp = dir == 0 ? 1 : (dir == 1 ? N1 : NF);
      const int fb = dir == 0 ? 3 : (dir == 1 ? 0 : 4), ft = dir == 0 ? 1 : (dir == 1 ? 2 : 5);
      const int ab = dir == 0 ? j + N1 * k : (dir == 1 ? i + N1 * k : i + N1 * j);
      const double* fd = fl + dir * 5 * Np + (p - row * stp);
      const double lb = s_l[fb * N1 + row], lt = s_l[ft * N1 + row];
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        if (HEVI && dir == 2 && (v == VD || v == VRT)) continue;
        out[v] = fma(lb, df[v * S + fb * NF + ab], out[v]);
        out[v] = fma(lt, df[v * S + ft * NF + ab], out[v]);
      }
#pragma unroll
      for (int l = 0; l < N1; ++l) {
        const double d = s_d[dir * NF + row * N1 + l];
#pragma unroll
        for (int v = 0; v < 5; ++v) {
          if (HEVI && dir == 2 && (v == VD || v == VRT)) continue;
          out[v] = fma(d, fd[v * Np + l * stp], out[v]);
        }
      }
    }
    if (!HEVI) {  // -g * VFilterPM1(DDENS)
#pragma unroll
      for (int l = 0; l < N1; ++l) out[VMZ] = fma(s_d[3 * NF + k * N1 + l], st[VD * Np + p + (l - k) * NF], out[VMZ]);
    }
    out[VMX] = fma(op.coriolis_f, st[VMY * Np + p], out[VMX]);
    out[VMY] = fma(-op.coriolis_f, st[VMX * Np + p], out[VMY]);
  }
  if (!SSP) {
    if (valid) {
#pragma unroll
      for (int v = 0; v < 5; ++v) t.v[v][g] = out[v];
    }
    return;
  }
  // --- the stage: q_new = A q0 + B q + C t, the last stage's filter, DPRES of q_new ---
  if (valid) {
#pragma unroll
    for (int v = 0; v < 5; ++v) out[v] = rk_low(x.A, x.q0.v[v][g], x.B, st[v * Np + p], x.C, out[v]);
  }
  if (x.filter) {
    double* a = fl;
    __syncthreads();  // all reads of the fluxes are done
#pragma unroll
    for (int v = 0; v < 5; ++v) out[v] = filter_node<N1>(op, a + 2 * v * Np, a + (2 * v + 1) * Np, out[v], p, i, j, k);
  }
  if (valid) {
#pragma unroll
    for (int v = 0; v < 5; ++v) x.qn.v[v][g] = out[v];
    if (x.dpn) x.dpn[g] = dpres_of(op, pf, lev, out[VRT]);
  }
}

// ---------------------------------------------------------------------------------------
// modal filter, in place: q <- Fv_z Fh_y Fh_x q  (tensorprod3D_kernel.F90:2555-2618)
// ---------------------------------------------------------------------------------------
template <int N1, int EPB>
__global__ void __launch_bounds__(EPB* N1* N1* N1) k_filter_fp64(const __grid_constant__ Ops op, F5 q, int Ne) {
  constexpr int Np = N1 * N1 * N1, NF = N1 * N1;
  extern __shared__ double sm[];
  const int tid = threadIdx.x, le = tid / Np, p = tid - le * Np;
  const int ke = blockIdx.x * EPB + le;
  const bool valid = ke < Ne;
  const int i = p % N1, j = (p / N1) % N1, k = p / NF;
  double* a = sm + le * 4 * Np;
  const size_t g = (size_t)ke * Np + p;
#pragma unroll
  for (int v = 0; v < 5; ++v) {  // two buffer pairs in turn: filter_node's last read is before the next but one's first write
    const double s = filter_node<N1>(op, a + (v & 1) * 2 * Np, a + ((v & 1) * 2 + 1) * Np, valid ? q.v[v][g] : 0.0, p, i, j, k);
    if (valid) q.v[v][g] = s;
  }
}

// DRHOT -> (PRES, DPRES), FP64 (nonhydro3d_common.F90:428-479)
__global__ void k_drhot2pres(const Ops op, const Prof pf, const double* __restrict__ drhot,
                             double* __restrict__ pres, double* __restrict__ dpres, size_t n) {
  const size_t g = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  const int p = (int)(g % op.Np);
  const size_t ke = g / op.Np;
  const int ez = (int)(ke / ((size_t)op.NeX * op.NeY));
  const int lev = ez * op.N1 + p / (op.N1 * op.N1);
  double pr;
  dpres[g] = dpres_of(op, pf, lev, drhot[g], &pr);
  if (pres) pres[g] = pr;
}

// ---------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------
template <int N1>
// two elements of p = 3 per block (a step of 8x8x8 elements, 256 blocks, 91 us, of 40x40x20 2702; four per block 90 and
// 2741)
static constexpr int epb_of() { return N1 <= 4 ? (N1 <= 2 ? 16 : (N1 == 3 ? 4 : 2)) : 1; }

template <int N1, bool HEVI, bool SSP>
static int launch_tend_n(const Ops& op, const Prof& pf, const F5c& q, const double* dpres, const F5& t, const SspArgs& x,
                         int Ne, cudaStream_t s) {
  constexpr int EPB = epb_of<N1>();
  constexpr int Np = N1 * N1 * N1;
  const size_t smem = sizeof(double) * (4 * N1 * N1 + 6 * N1 + EPB * (22 * Np + 5 * 6 * N1 * N1));
  auto kfn = k_tend_fp64<N1, EPB, HEVI, SSP>;
  cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  kfn<<<(Ne + EPB - 1) / EPB, EPB * Np, smem, s>>>(op, pf, q, dpres, t, x, Ne);
  return (int)cudaGetLastError();
}

int launch_tend_fp64(const Ops& op, const Prof& pf, const F5c& q, const double* dpres, const F5& t, int Ne,
                     int hevi, cudaStream_t s) {
  const SspArgs x{};
#define FEDG_TEND(n) \
  case n: return hevi ? launch_tend_n<n, true, false>(op, pf, q, dpres, t, x, Ne, s) : launch_tend_n<n, false, false>(op, pf, q, dpres, t, x, Ne, s);
  switch (op.N1) {
    FEDG_TEND(2) FEDG_TEND(3) FEDG_TEND(4) FEDG_TEND(5) FEDG_TEND(6) FEDG_TEND(7) FEDG_TEND(8)
  }
#undef FEDG_TEND
  return (int)cudaErrorInvalidValue;
}

int launch_ssp_stage_fp64(const Ops& op, const Prof& pf, const F5c& q, const double* dpres, const SspArgs& x, int Ne,
                          cudaStream_t s) {
  const F5 t{};
#define FEDG_SSP(n) case n: return launch_tend_n<n, false, true>(op, pf, q, dpres, t, x, Ne, s);
  switch (op.N1) {
    FEDG_SSP(2) FEDG_SSP(3) FEDG_SSP(4) FEDG_SSP(5) FEDG_SSP(6) FEDG_SSP(7) FEDG_SSP(8)
  }
#undef FEDG_SSP
  return (int)cudaErrorInvalidValue;
}

template <int N1>
static int launch_filter_n(const Ops& op, const F5& q, int Ne, cudaStream_t s) {
  constexpr int EPB = epb_of<N1>();
  constexpr int Np = N1 * N1 * N1;
  const size_t smem = sizeof(double) * EPB * 4 * Np;
  k_filter_fp64<N1, EPB><<<(Ne + EPB - 1) / EPB, EPB * Np, smem, s>>>(op, q, Ne);
  return (int)cudaGetLastError();
}

int launch_filter_fp64(const Ops& op, const F5& q, int Ne, cudaStream_t s) {
  switch (op.N1) {
    case 2: return launch_filter_n<2>(op, q, Ne, s);
    case 3: return launch_filter_n<3>(op, q, Ne, s);
    case 4: return launch_filter_n<4>(op, q, Ne, s);
    case 5: return launch_filter_n<5>(op, q, Ne, s);
    case 6: return launch_filter_n<6>(op, q, Ne, s);
    case 7: return launch_filter_n<7>(op, q, Ne, s);
    case 8: return launch_filter_n<8>(op, q, Ne, s);
  }
  return (int)cudaErrorInvalidValue;
}

int launch_drhot2pres(const Ops& op, const Prof& pf, const double* drhot, double* pres, double* dpres, size_t n,
                      cudaStream_t s) {
  const int bs = 256;
  k_drhot2pres<<<(unsigned)((n + bs - 1) / bs), bs, 0, s>>>(op, pf, drhot, pres, dpres, n);
  return (int)cudaGetLastError();
}

}  // namespace fedg
