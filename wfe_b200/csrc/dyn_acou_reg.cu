// Acoustic column kernel with every level's inputs in registers (the w - pi'
// solve of one substep, src/dynamics/kernels.cu:531-645).
//
// A CTA owns CX columns of one row and all their levels: thread (tx, lane)
// holds KCH consecutive levels of column tx.  It issues the loads of its levels'
// state, coefficients and moisture before anything waits, so a launch pays
// their latency once per resident CTA instead of once per level and phase, and
// each field value is read once.  (The slow pi' tendency of relaxed runs is read
// behind the edge exchange, theta's and d theta_b / dz while the column is
// swept.)  Only what crosses the edge between two lanes' chunks goes
// through shared memory (nine values up, three down), then the tridiagonal
// rows and the solution; the Thomas sweep is the serial one of the other
// exact column kernels (one thread per column, one reciprocal per level) with
// the next rows' shared loads issued ahead.  The expressions are those of the
// column tile kernel (dyn_acou.cu, column_core): the same values bit for bit.
//
// PROF: the coefficients that depend on the level alone from per-level tables
// (PipeColParams::prof in kernels.cuh) instead of seven fields.
//
// What bounds it: the barrier behind the serial sweep (9 of 19 cycles between
// a warp's issues with two CTAs per SM) and the latency of each warp's own
// instructions (about 260 a level), not memory: DRAM is at a fifth of its
// rate.  So the shapes trade registers against
// resident warps; 16 to 32 columns with three or four levels a thread win on
// large grids, 8 columns on small ones, and the tuner picks.  A shape has one
// cap per precision for all its forms, and most forms spill under it (bytes
// stored, three / four levels a thread; dry, moist from the terms, from the
// fields).  FP32 with the level tables 0, 12, 16 / 0, 28, 52, without 8, 24,
// 40 / 32, 48, 72, relaxed 0, 36, 44 / 28, 60, 80; FP64 in 16 columns with
// the tables 0, 0, 8 / 8, 24, 104, without 0, 8, 40 / 24, 80, 216.  Per launch
// (event-timed inside a step, 4.7 us of event nodes included) against the
// best of the kernels it replaced -- contiguous level chunks in registers with
// recomputed edges, and a producer warp's ring of bulk loads in front of the
// same sweep: 160x160x40 flat FP32 29.7 against 48.3 us, FP64 59.6 against
// 84.4, 181x203x53 60 against 85.6, 300x200x45 over terrain 121-127 against
// 142, 512x4x64 13.2 against 16.8.  With the moisture as the step's two terms
// (MOIST_TERMS) instead of four fields: 27.7, 49.6, 54.6 and 115.7 us.
#include <cuda_runtime.h>

#include "core.cuh"
#include "kernels.cuh"
#include "dyn_common.cuh"

namespace wfe {

namespace {

// where a column's moisture comes from: nowhere (dry), qv, qc, qr and qv_b, or
// the two terms they make on w levels, the same in every substep of a step
// (AcouArgs::mq, mb)
enum { MOIST_NONE = 0, MOIST_FIELDS = 1, MOIST_TERMS = 2 };

// The two moisture terms of the inner w levels from the time-n species, which
// no substep changes: the factor of theta_v^w and the moist part of the
// buoyancy, rounded as the column kernels round them.
template <typename R>
__global__ void __launch_bounds__(256) k_moist_terms(Layout L, const R* __restrict__ qv, const R* __restrict__ qc,
                                                     const R* __restrict__ qr, const R* __restrict__ qvb,
                                                     R* __restrict__ mq, R* __restrict__ mb) {
  const int i = blockIdx.x * 32 + threadIdx.x, j = blockIdx.y * 8 + threadIdx.y, k = 1 + blockIdx.z;
  if (i >= L.nx || j >= L.ny) return;
  const int c = L.ati(i, j, k), cm = c - L.planei();
  mq[c] = (R)1 + Phys<R>::eps61 * (R)0.5 * (qv[cm] + qv[c]);
  const R dqv = (R)0.5 * (qv[cm] + qv[c]) - (R)0.5 * (qvb[cm] + qvb[c]);
  const R qcr = (R)0.5 * (qc[cm] + qc[c]) + (R)0.5 * (qr[cm] + qr[c]);
  mb[c] = fma_rn(Phys<R>::eps61, dqv, -qcr);
}

// shared values per (lane, column): the chunk edges
enum { XU_SU = 0, XU_SV, XU_AV, XU_PI, XU_TH, XU_QV, XU_QC, XU_QR, XU_QVB, XU_P, XU_E, XD_AV, XD_W, XD_SV, X_N };

// a b - c d as the other column kernels' compiled expression rounds it (the
// second product rounded, the first fused): left to the compiler, a product
// two neighbouring levels of a thread share would be rounded for both
template <typename R>
__device__ __forceinline__ R flux_diff(R a, R b, R c, R d) {
  return fma_rn(a, b, -mul_rn(c, d));
}

template <typename R, int CX, int KCH, bool PROF, int MOIST, bool TPI>
__device__ __forceinline__ void column_reg_body(const AcouArgs<R>& a, const R* __restrict__ prof, R* smem) {
  const Layout& L = a.L;
  const int nz = L.nz;
  const int KL = blockDim.y;
  const int tx = threadIdx.x, lane = threadIdx.y;
  const int i = blockIdx.x * CX + tx, j = blockIdx.y;
  const bool active = i < L.nx;
  R* X = smem;                                // X_N x KL x CX chunk edges
  R* sA = X + (size_t)X_N * KL * CX;          // rows, (nz + 1) x CX each
  R* sB = sA + (size_t)(nz + 1) * CX;
  R* sC = sB + (size_t)(nz + 1) * CX;
  R* sD = sC + (size_t)(nz + 1) * CX;         // right-hand side, then the solution w
#define EX(f, l) X[((f) * KL + (l)) * CX + tx]
#define SQ(A, k) A[(k) * CX + tx]
  const R dtau = a.dtau;
  const R c1 = ((R)1 + a.p.acoustic_beta) * (R)0.5;
  const R c2 = ((R)1 - a.p.acoustic_beta) * (R)0.5;
  const int c2d = L.at2i(active ? i : 0, j);
  const int sy = L.px, pl = L.planei();
  const int klo = lane * KCH;
  const int c0 = L.ati(active ? i : 0, j, 0);
  const int n1 = nz + 1;
  const R* __restrict__ u = a.u_out;
  const R* __restrict__ v = a.v_out;

  // ---- loads of the chunk's levels; slots above the top level read level
  // nz - 1 (nothing they compute is used), so no load waits for a predicate
  R u0[KCH], u1[KCH], v0[KCH], v1[KCH], Dh[KCH], av[KCH + 1], w[KCH + 1], pi[KCH], th[KCH], kt[KCH];
  R thbw[KCH], tw[KCH], qv[KCH], qc[KCH], qr[KCH], qvb[KCH];
  const R J = a.m.jac[c2d], hxc = a.m.hx[c2d], hyc = a.m.hy[c2d], mc = a.m.mapf[c2d];
  R rx0[KCH], rx1[KCH], ry0[KCH], ry1[KCH];
  R idzc[KCH], idzw[KCH];  // the level tables: 1 / dzeta at the cell and the w level
#pragma unroll
  for (int q = 0; q < KCH; ++q) {
    const int k = klo + q < nz ? klo + q : nz - 1;
    const int c = c0 + k * pl;
    idzc[q] = a.co.inv_dzc[L.at1(k)];
    idzw[q] = a.co.inv_dzw[L.at1(k)];
    u0[q] = u[c];
    u1[q] = u[c + 1];
    v0[q] = v[c];
    v1[q] = v[c + sy];
    if (PROF) {
      rx0[q] = rx1[q] = prof[PF_RTJX * n1 + k];
      ry0[q] = ry1[q] = prof[PF_RTJY * n1 + k];
      kt[q] = prof[PF_KT3 * n1 + k];
      av[q] = prof[PF_AW * n1 + k];
      thbw[q] = prof[PF_THBW * n1 + k];
    } else {
      rx0[q] = a.co.rtjx[c];
      rx1[q] = a.co.rtjx[c + 1];
      ry0[q] = a.co.rtjy[c];
      ry1[q] = a.co.rtjy[c + sy];
      kt[q] = a.co.kt3[c];
      av[q] = a.co.aw[c];
      thbw[q] = a.b.thbw[c];
    }
    pi[q] = a.pi_cur[c];
    th[q] = a.th_in[c];
    tw[q] = a.tw[c];
    if (MOIST == MOIST_FIELDS) {
      qv[q] = a.qv[c];
      qc[q] = a.qc[c];
      qr[q] = a.qr[c];
      qvb[q] = PROF ? prof[PF_QVB * n1 + k] : a.b.qvb[c];
    } else if (MOIST == MOIST_TERMS) {
      qv[q] = a.mq[c];
      qc[q] = a.mb[c];
    }
    w[q] = a.w_in[c0 + (klo + q < nz ? klo + q : nz) * pl];
    if (klo + q == 0 || klo + q >= nz) av[q] = 0;
  }
  const R invJ = (R)1 / J;
  const R mcx = mc * a.co.inv_dx, mcy = mc * a.co.inv_dy;
  const bool terrain = active && (hxc != (R)0 || hyc != (R)0);
#pragma unroll
  for (int q = 0; q < KCH; ++q)
    Dh[q] = (rx1[q] * u1[q] - rx0[q] * u0[q]) * mcx + (ry1[q] * v1[q] - ry0[q] * v0[q]) * mcy;

  // ---- chunk edges: the top level's values up, the first level's down
  constexpr int T = KCH - 1;
  EX(XU_AV, lane) = av[T];
  EX(XU_PI, lane) = pi[T];
  EX(XU_TH, lane) = th[T];
  EX(XD_AV, lane) = av[0];
  EX(XD_W, lane) = w[0];
  if (MOIST == MOIST_FIELDS) {
    EX(XU_QV, lane) = qv[T];
    EX(XU_QC, lane) = qc[T];
    EX(XU_QR, lane) = qr[T];
    EX(XU_QVB, lane) = qvb[T];
  }
  if (terrain) {
    EX(XU_SU, lane) = u0[T] + u1[T];
    EX(XU_SV, lane) = v0[T] + v1[T];
  }
  const bool hills = __syncthreads_or(terrain);
  av[KCH] = w[KCH] = 0;
  if (lane + 1 < KL) {
    av[KCH] = EX(XD_AV, lane + 1);
    w[KCH] = EX(XD_W, lane + 1);
  }
  // ---- the explicit terrain cross flux (kernels.cu:552-568)
  R sv[KCH + 1];
#pragma unroll
  for (int q = 0; q < KCH + 1; ++q) sv[q] = 0;
  if (hills) {
    if (terrain) {
#pragma unroll
      for (int q = 0; q < KCH; ++q) {
        const int k = klo + q;
        if (k >= 1 && k < nz) {
          const R su = q ? u0[q ? q - 1 : 0] + u1[q ? q - 1 : 0] : EX(XU_SU, lane - 1);
          const R sw = q ? v0[q ? q - 1 : 0] + v1[q ? q - 1 : 0] : EX(XU_SV, lane - 1);
          R uw = (R)0.25 * (su + u0[q] + u1[q]);
          R vw = (R)0.25 * (sw + v0[q] + v1[q]);
          sv[q] = av[q] * (uw * hxc + vw * hyc) * a.co.fac_w[L.at1(k)];
        }
      }
    }
    EX(XD_SV, lane) = sv[0];
    __syncthreads();
    if (lane + 1 < KL) sv[KCH] = EX(XD_SV, lane + 1);
  }
  // ---- the explicit part of the pi' equation (kernels.cu:570-587)
  R P[KCH], E[KCH];
#pragma unroll
  for (int q = 0; q < KCH; ++q) {
    const int k = klo + q;
    const R idz = idzc[q];
    const R tpi = TPI ? a.tpi[c0 + (k < nz ? k : nz - 1) * pl] : (R)0;
    P[q] = pi[q] + dtau * tpi -
           dtau * kt[q] * (Dh[q] - (sv[q + 1] - sv[q]) * idz + c2 * flux_diff(av[q + 1], w[q + 1], av[q], w[q]) * idz);
    E[q] = dtau * kt[q] * c1 * idz;
  }
  EX(XU_P, lane) = P[T];
  EX(XU_E, lane) = E[T];
  __syncthreads();
  // ---- the tridiagonal rows of the inner levels (kernels.cu:589-611)
#pragma unroll
  for (int q = 0; q < KCH; ++q) {
    const int k = klo + q;
    if (k >= 1 && k < nz) {
      const int p = q ? q - 1 : 0;
      const R thm = q ? th[p] : EX(XU_TH, lane - 1), thc = th[q];
      const R Em = q ? E[p] : EX(XU_E, lane - 1), Ek = E[q];
      const R Pm = q ? P[p] : EX(XU_P, lane - 1);
      const R pim = q ? pi[p] : EX(XU_PI, lane - 1);
      const R avm = q ? av[p] : EX(XU_AV, lane - 1);
      R qvm = 0;
      if (MOIST == MOIST_FIELDS) qvm = q ? qv[p] : EX(XU_QV, lane - 1);
      const R iJdz = invJ * idzw[q];
      R thvw = thbw[q] + (R)0.5 * (thm + thc);
      if (MOIST == MOIST_FIELDS) thvw *= (R)1 + Phys<R>::eps61 * (R)0.5 * (qvm + qv[q]);
      if (MOIST == MOIST_TERMS) thvw *= qv[q];
      R G = dtau * Phys<R>::cp * thvw * c1 * iJdz;
      SQ(sA, k) = -G * Em * avm;
      SQ(sB, k) = (R)1 + G * av[q] * (Ek + Em);
      SQ(sC, k) = -G * Ek * av[q + 1];
      R buoy = Phys<R>::grav * (R)0.5 * (thm + thc) / thbw[q];
      if (MOIST == MOIST_TERMS) buoy = fma_rn(Phys<R>::grav, qc[q], buoy);
      if (MOIST == MOIST_FIELDS) {
        const R qcm = q ? qc[p] : EX(XU_QC, lane - 1), qrm = q ? qr[p] : EX(XU_QR, lane - 1);
        const R qbm = q ? qvb[p] : EX(XU_QVB, lane - 1);
        R dqv = (R)0.5 * (qvm + qv[q]) - (R)0.5 * (qbm + qvb[q]);
        R qcr = (R)0.5 * (qcm + qc[q]) + (R)0.5 * (qrm + qr[q]);
        buoy += Phys<R>::grav * (Phys<R>::eps61 * dqv - qcr);
      }
      R RHS = w[q] + dtau * (buoy + tw[q]) - dtau * Phys<R>::cp * thvw * c2 * (pi[q] - pim) * iJdz;
      SQ(sD, k) = RHS - G * (P[q] - Pm);
    }
  }
  if (lane == 0) {
    // diagnostic surface w from the new u, v: the solution's level 0
    R us = (R)0.5 * (u0[0] + u1[0]);
    R vs = (R)0.5 * (v0[0] + v1[0]);
    SQ(sD, 0) = us * hxc + vs * hyc;
    SQ(sD, nz) = 0;
  }
  __syncthreads();
  // the way out's own inputs arrive while the column is swept
  R tt[KCH], db[KCH];
#pragma unroll
  for (int q = 0; q < KCH; ++q) {
    const int k = klo + q < nz ? klo + q : nz - 1;
    tt[q] = a.tth[c0 + k * pl];
    db[q] = PROF ? prof[PF_DTHB * n1 + k] : a.b.dthbdz[c0 + k * pl];
  }
  // ---- Thomas sweep, one thread per column (kernels.cu:612-634)
  if (lane == 0) {
    // rows in blocks of four, the next block's shared loads issued ahead of
    // this block's chain; A at level 1 is taken as 0 (level 0 is no unknown)
    R cprev = 0, dprev = 0;
    R Ak[4], Bk[4], Ck[4], Dk[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int k = 1 + q < nz ? 1 + q : nz - 1;
      Ak[q] = SQ(sA, k), Bk[q] = SQ(sB, k), Ck[q] = SQ(sC, k), Dk[q] = SQ(sD, k);
    }
    Ak[0] = 0;
    for (int kb = 1; kb < nz; kb += 4) {
      R An[4], Bn[4], Cn[4], Dn[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int k = kb + 4 + q < nz ? kb + 4 + q : nz - 1;
        An[q] = SQ(sA, k), Bn[q] = SQ(sB, k), Cn[q] = SQ(sC, k), Dn[q] = SQ(sD, k);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const R r = (R)1 / (Bk[q] - Ak[q] * cprev);
        cprev = Ck[q] * r;
        dprev = (Dk[q] - Ak[q] * dprev) * r;
        if (kb + q < nz) {
          SQ(sC, kb + q) = cprev;
          SQ(sD, kb + q) = dprev;
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) Ak[q] = An[q], Bk[q] = Bn[q], Ck[q] = Cn[q], Dk[q] = Dn[q];
    }
    // back substitution in blocks of eight levels whose rows are read first
    R wabove = 0;
    int k = nz - 1;
    for (; k >= 8; k -= 8) {
      R cb[8], dd[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) cb[q] = SQ(sC, k - q), dd[q] = SQ(sD, k - q);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        wabove = dd[q] - cb[q] * wabove;
        SQ(sD, k - q) = wabove;
      }
    }
    for (; k >= 1; --k) {
      wabove = SQ(sD, k) - SQ(sC, k) * wabove;
      SQ(sD, k) = wabove;
    }
  }
  __syncthreads();
  // ---- pi', theta', w (kernels.cu:636-644)
  if (active) {
#pragma unroll
    for (int q = 0; q < KCH; ++q) {
      const int k = klo + q;
      if (k > nz) continue;
      const int c = c0 + k * pl;
      if (k < nz) {
        const R wn = SQ(sD, k), wn1 = SQ(sD, k + 1);
        a.pi_next[c] = P[q] - E[q] * flux_diff(av[q + 1], wn1, av[q], wn);
        R wc = (R)0.5 * (wn + wn1);
        a.th_out[c] = th[q] + dtau * (tt[q] - wc * db[q]);
        a.w_out[c] = wn;
      } else {
        a.w_out[c] = 0;
      }
    }
  }
#undef EX
#undef SQ
}

template <typename R, int CX, int KCH, int REGS, bool PROF, int MOIST, bool TPI>
__global__ void __maxnreg__(REGS) k_acoustic_column_reg(AcouArgs<R> a, const R* __restrict__ prof) {
  extern __shared__ __align__(16) unsigned char smem_reg[];
  column_reg_body<R, CX, KCH, PROF, MOIST, TPI>(a, prof, reinterpret_cast<R*>(smem_reg));
}

// columns per CTA, levels per thread, registers per thread in FP32 and FP64
struct Shape {
  int cx, kch, regs32, regs64;
};
constexpr Shape kShapes[] = {{16, 3, 72, 136}, {32, 3, 72, 128}, {16, 4, 80, 152},
                             {32, 4, 80, 152}, {8, 2, 64, 104}, {8, 3, 72, 136}};
constexpr int kNumShapes = 6;

template <typename R>
constexpr int regs_of(int s) {
  return sizeof(R) == 4 ? kShapes[s].regs32 : kShapes[s].regs64;
}

int lanes(int nz, int kch) { return (nz + kch) / kch; }

template <typename R>
size_t reg_smem(int nz, int s) {
  return ((size_t)X_N * lanes(nz, kShapes[s].kch) + (size_t)4 * (nz + 1)) * kShapes[s].cx * sizeof(R);
}

// the forms of a shape: dry, moist from the fields or from the step's terms,
// with and without the slow pi' tendency (only operator calls and relaxed
// runs have one; with it the tables are not used)
template <typename R, int S, bool PROF, bool TPI, class F>
void with_moisture(int moist, F&& f) {
  constexpr int CX = kShapes[S].cx, KCH = kShapes[S].kch, G = regs_of<R>(S);
  if (moist == MOIST_TERMS) f(k_acoustic_column_reg<R, CX, KCH, G, PROF, MOIST_TERMS, TPI>);
  else if (moist == MOIST_FIELDS) f(k_acoustic_column_reg<R, CX, KCH, G, PROF, MOIST_FIELDS, TPI>);
  else f(k_acoustic_column_reg<R, CX, KCH, G, PROF, MOIST_NONE, TPI>);
}
template <typename R, int S, class F>
void with_kernel(bool prof, int moist, bool tpi, F&& f) {
  if (tpi) with_moisture<R, S, false, true>(moist, f);
  else if (prof) with_moisture<R, S, true, false>(moist, f);
  else with_moisture<R, S, false, false>(moist, f);
}
template <typename R, class F>
void for_shape(int s, bool prof, int moist, bool tpi, F&& f) {
  switch (s) {
    case 0: with_kernel<R, 0>(prof, moist, tpi, f); break;
    case 1: with_kernel<R, 1>(prof, moist, tpi, f); break;
    case 2: with_kernel<R, 2>(prof, moist, tpi, f); break;
    case 3: with_kernel<R, 3>(prof, moist, tpi, f); break;
    case 4: with_kernel<R, 4>(prof, moist, tpi, f); break;
    default: with_kernel<R, 5>(prof, moist, tpi, f); break;
  }
}

}  // namespace

int acoustic_reg_shapes() { return kNumShapes; }

template <typename R>
void launch_moist_terms(const Layout& L, const DBase<R>& b, const R* qv, const R* qc, const R* qr, R* mq, R* mb,
                        cudaStream_t st) {
  if (L.nz < 2) return;
  k_moist_terms<R><<<dim3((L.nx + 31) / 32, (L.ny + 7) / 8, L.nz - 1), dim3(32, 8), 0, st>>>(L, qv, qc, qr, b.qvb,
                                                                                            mq, mb);
}

template <typename R>
bool acoustic_reg_fits(int nz, int s) {
  if (s < 0 || s >= kNumShapes || nz < 2) return false;
  const int threads = kShapes[s].cx * lanes(nz, kShapes[s].kch), warps = (threads + 31) / 32;
  // a scheduler's quarter of the register file holds a quarter of the warps
  return threads <= 1024 && (warps + 3) / 4 * 32 * regs_of<R>(s) <= 16384 && reg_smem<R>(nz, s) <= 200 * 1024;
}

template <typename R>
int prepare_acoustic_reg(int nz) {
  int rc = 0;
  for (int s = 0; s < kNumShapes; ++s) {
    if (!acoustic_reg_fits<R>(nz, s)) continue;
    for (int p = 0; p < 12; ++p)
      for_shape<R>(s, p & 1, p / 4, p & 2, [&](auto* k) { rc |= raise_smem_limit(k, reg_smem<R>(nz, s)) != cudaSuccess; });
  }
  return rc;
}

template <typename R>
int launch_acoustic_column_reg(const AcouArgs<R>& a, const R* prof, int s, cudaStream_t st) {
  const int nz = a.L.nz;
  if (!acoustic_reg_fits<R>(nz, s)) return 2;
  const dim3 grd((a.L.nx + kShapes[s].cx - 1) / kShapes[s].cx, a.L.ny), blk(kShapes[s].cx, lanes(nz, kShapes[s].kch));
  const int moist = !a.p.moisture ? MOIST_NONE : a.mq ? MOIST_TERMS : MOIST_FIELDS;
  for_shape<R>(s, prof != nullptr, moist, a.tpi != nullptr, [&](auto* k) { k<<<grd, blk, reg_smem<R>(nz, s), st>>>(a, prof); });
  return 0;
}

#define WFE_INST(R)                                       \
  template bool acoustic_reg_fits<R>(int, int);           \
  template int prepare_acoustic_reg<R>(int);              \
  template void launch_moist_terms<R>(const Layout&, const DBase<R>&, const R*, const R*, const R*, R*, R*, \
                                      cudaStream_t);      \
  template int launch_acoustic_column_reg<R>(const AcouArgs<R>&, const R*, int, cudaStream_t);
WFE_INST(float)
WFE_INST(double)
#undef WFE_INST

}  // namespace wfe
