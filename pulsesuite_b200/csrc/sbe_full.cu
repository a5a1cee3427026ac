// sbe_full.cu -- the full-matrix (Nk x Nk) SBE step of one quantum wire in
// FP64, for drives that vary along the wire: the reference's general case.
//
// A wire's state is three complex matrices p[kh][ke] (YY), C[k1][k2] (CC)
// and D[k1][k2] (DD) per stored level (SBEs.py:4782-4790); with a field that
// is not uniform along the wire the coupling Meh and the Hamiltonians are
// full matrices and the right-hand side is O(Nk^3).  One call of
// psb_full_step_f64 is one step of the reference's integrator for one wire
// (SBESolver._sbe_calculator, SBEs.py:5624-5836) with the flags Optics,
// Excitons, LF and Screened:
//   Meh   = CalcMeh of the wire-space fields (SBEs.py:5165-5175)
//   H     = CalcH with the exchange (and, with LF, direct) Coulomb sums
//           along the diagonals of p, C, D (SBEs.py:819-935, lf branch)
//   dX    = dpdt, dCdt, dDdt (SBEs.py:1952-1975, 2318-2337, 2617-2636)
//   X3    = X1 + 2 dt dX, occupations |C3_kk|, |D3_kk| rescaled to a common
//           total, X2 = (X1 + X3) / 2 (SBEs.py:5681-5718)
// psb_full_step_mb_f64 adds the many-body terms mb.params switches on
// (DiagDph, OffDiagDph: k-dependent and off-diagonal dephasing in dpdt;
// EHs, Phonon: carrier-carrier and LO-phonon relaxation of the new
// occupations before the rescale; Recomb: spontaneous emission after that
// relaxation; DCTrans: the DC-field shift of X3 in k); see the mb_* kernels.
// psb_full_sources_f64 evaluates the wire-space source terms of the new
// level: the polarisation components of QWPolarization3 and the charge
// densities of QWRho5 before their transforms (qwoptics.py:56-84, 367-381).
// FP64 throughout.  The sums are regrouped for the machine and agree with the
// reference's to rounding (tests: 1e-10 of its own runs, 1e-12 of 64-bit
// restatements).  Three keep one fixed order and rounding whatever the launch,
// because the charge density is a difference that cancels to their last digits:
// the density sums, the occupations' sums and the DC shift.
#include <type_traits>

#include "dmma.cuh"
#include "psb_common.cuh"

namespace psb {
namespace full {

__device__ __forceinline__ double2 cm(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 ca(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 cs(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 rs(double s, double2 a) { return make_double2(s * a.x, s * a.y); }
// x / (i hbar)
__device__ __forceinline__ double2 div_ih(double2 x, double hb) {
  return make_double2(x.y / hb, -x.x / hb);
}

struct Step {
  int nk, nr, nq0;
  const double* kr;     // [nk] (unused by the step; kept for symmetry)
  const double* V3;     // [3][nk]: V_eh, V_ee, V_hh at index distance q
  const double* Ee;     // [nk]
  const double* Eh;     // [nk]
  const double2* E;     // [3][nr] wire-space fields Ex, Ey, Ez (q space)
  PsbFullParams prm;
  double2* L1;          // levels, [3][nk][nk] each: p, C, D
  double2* L2;
  double2* L3;
  double* fac;          // work [3]: the occupations' common total, their sums
  double2* H;           // work [3][nk][nk]: Heh, Hee, Hhh
  double2* X3;          // work or many-body scratch [3][nk][nk]: X1 + 2 dt dX
  // many-body terms (null when off): k-dependent dephasing rates and the
  // off-diagonal dephasing term of dpdt
  const double* GamE;   // [nk]
  const double* GamH;   // [nk]
  const double2* OffP;  // [nk][nk], OffP[kh][ke]
  // a batch of wires of one grid, wire = blockIdx.y: byte strides between
  // the wires' V3, fields, levels, work and many-body scratch, and the
  // per-wire [nw][4] = yw, (-1)^w, dc_dk, 0 (null: prm.yw, prm.sgnw)
  int64_t st_v3, st_e, st_lv, st_wk, st_sc, st_x3;
  const double* wpar;
};

template <class T>
__device__ __forceinline__ T* bump(T* p, int64_t bytes) {
  return p ? reinterpret_cast<T*>(reinterpret_cast<uintptr_t>(p) + bytes) : p;
}

// the Step of wire blockIdx.y of a batch
__device__ __forceinline__ Step at_wire(Step s) {
  const int64_t w = blockIdx.y;
  s.V3 = bump(s.V3, w * s.st_v3);
  s.E = bump(s.E, w * s.st_e);
  s.L1 = bump(s.L1, w * s.st_lv);
  s.L2 = bump(s.L2, w * s.st_lv);
  s.L3 = bump(s.L3, w * s.st_lv);
  s.fac = bump(s.fac, w * s.st_wk);
  s.H = bump(s.H, w * s.st_wk);
  s.GamE = bump(s.GamE, w * s.st_sc);
  s.GamH = bump(s.GamH, w * s.st_sc);
  s.OffP = bump(s.OffP, w * s.st_sc);
  s.X3 = bump(s.X3, w * s.st_x3);
  if (s.wpar) {
    s.prm.yw = s.wpar[4 * w];
    s.prm.sgnw = s.wpar[4 * w + 1];
  }
  return s;
}

// CalcMeh (SBEs.py:5165-5175) and CalcH (SBEs.py:819-935).  Every element
// (k1, k2) sums along its diagonal d = k1 - k2 of p, C, D (the exchange terms)
// and, with LF, the whole diagonals d and -d of C and D (the direct terms,
// the same for all its elements).  The coupling
//   Meh[ke][kh] = -ehint (Xcv Ex[q] + Ycv Ey[q] yw + Zcv Ez[q] (-1)^w),
// q = ke - kh + NQ0, Xcv = dcv (-1)^(kh+1), Ycv = dcv, Zcv = -dcv (QWOptics
// dipoles, qwoptics.py:619-623) has one set of fields per diagonal too.
//
// One warp per diagonal and wire, neighbouring diagonals in a CTA (their
// strided elements share cache lines).  The runs of p, C and D lie in shared
// memory; lane b sums R = 4 neighbouring elements with the last 4 values of
// each table in registers, so a step over the run costs one new value per
// table and one broadcast per matrix for 24 FMAs.  The tables are stored with
// one pad every 4 values, which spreads the lanes' stride of 4 over the banks.
// 64 wires of Nk 114: 0.10 ms, bound by the strided reads and writes of the
// diagonals; 0.24 with a CTA per diagonal and one element per thread.
constexpr int kHDiags = 8, kHR = 4;  // diagonals per CTA at most (fewer when memory is short)
__host__ __device__ inline int h_skew(int i) { return i + i / kHR; }
// doubles of one table, positions u - t in [-(nk + 3), nk + 3], and of a run
__host__ __device__ inline int h_vlen(int nk) { return h_skew(2 * (nk + kHR)) + 1; }
inline size_t h_smem(int nk, int diags) {
  const int nr = (nk + kHR - 1) / kHR * kHR;
  return 3 * (size_t)((h_vlen(nk) + 1) / 2 * 2) * 8 + diags * 3 * (size_t)nr * 16;
}

__device__ __forceinline__ double2 warp_sum2(double2 v) {
  return make_double2(warp_sum(v.x), warp_sum(v.y));
}

__global__ void __launch_bounds__(32 * kHDiags) calch_kernel(Step s0) {
  const Step s = at_wire(s0);
  const int nk = s.nk, n2 = nk * nk, lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  extern __shared__ __align__(16) double hsm[];
  const int vlen = (h_vlen(nk) + 1) / 2 * 2, vo = nk + kHR;  // table t at t vlen, q = 0 at vo
  const int nr = (nk + kHR - 1) / kHR * kHR;
  double2* run = reinterpret_cast<double2*>(hsm + 3 * vlen) + wp * 3 * nr;
  for (int i = threadIdx.x; i < 2 * vo; i += blockDim.x) {
    const int q = i < vo ? vo - i : i - vo;
#pragma unroll
    for (int t = 0; t < 3; ++t)
      hsm[t * vlen + h_skew(i)] = q > 0 && q < nk ? s.V3[t * nk + q] : 0.0;
  }
  const int d = (int)(blockIdx.x * blockDim.x + threadIdx.x) / 32 - (nk - 1);  // k1 - k2
  const bool mine = d < nk;
  const int ad = d < 0 ? -d : d, len = mine ? nk - ad : 0;
  const int o1 = d > 0 ? d : 0, o2 = d < 0 ? -d : 0;  // k1 = t + o1, k2 = t + o2
  const double2* M[3] = {s.L3, s.L3 + n2, s.L3 + 2 * n2};
  const double2 z = make_double2(0.0, 0.0);
  double2 dir1 = z, dir2 = z;  // the direct terms of Hee and Hhh
  const bool exc = s.prm.excitons != 0, lf = s.prm.lf != 0;
  if (exc) {
    // element u of the run: row o2 + u, column o1 + u; mirrored: (o1 + u, o2 + u)
    double2 sc = z, sd = z, mc = z, md = z;
    for (int u = lane; u < nr; u += 32) {
      const bool in = u < len;
      const int a = (o2 + u) * nk + o1 + u, b = (o1 + u) * nk + o2 + u;
      const double2 pv = in ? M[0][a] : z, cv = in ? M[1][a] : z, dv = in ? M[2][a] : z;
      run[u] = pv;
      run[nr + u] = cv;
      run[2 * nr + u] = dv;
      if (lf && d != 0 && in) {
        sc = ca(sc, cv);
        sd = ca(sd, dv);
        mc = ca(mc, M[1][b]);
        md = ca(md, M[2][b]);
      }
    }
    if (lf && d != 0 && mine) {
      // Vee(d) sum C[k][k + d] - Veh(d) sum D[k + d][k], and Vhh(d), D, C
      const double v0 = s.V3[ad], v1 = s.V3[nk + ad], v2 = s.V3[2 * nk + ad];
      dir1 = cs(rs(v1, warp_sum2(sc)), rs(v0, warp_sum2(md)));
      dir2 = cs(rs(v2, warp_sum2(sd)), rs(v0, warp_sum2(mc)));
    }
  }
  __syncthreads();
  if (!mine) return;
  const int q = d + s.nq0;
  const bool inq = q >= 0 && q < s.nr;
  const double dcv = s.prm.dcv, eh = s.prm.ehint;
  const double2 ex = inq ? s.E[q] : z, ey = inq ? s.E[s.nr + q] : z,
                ez = inq ? s.E[2 * s.nr + q] : z;
  // sums of Hee and Hhh: everywhere with LF, else on the diagonal only
  const bool occ = exc && (lf || d == 0);
  for (int t0 = kHR * lane; t0 < len; t0 += kHR * 32) {
    double2 h0[kHR], h1[kHR], h2[kHR];
    double w0[kHR], w1[kHR], w2[kHR];
#pragma unroll
    for (int r = 0; r < kHR; ++r) {
      h0[r] = h1[r] = h2[r] = z;
      const int i = h_skew(vo - t0 - r);  // u = 0
      w0[r] = hsm[i];
      w1[r] = hsm[vlen + i];
      w2[r] = hsm[2 * vlen + i];
    }
    if (exc) {
      // (the runs are zero from len to a multiple of kHR)
      for (int u0 = 0; u0 < len; u0 += kHR) {
#pragma unroll
        for (int uu = 0; uu < kHR; ++uu) {
          const double2 pv = run[u0 + uu];
#pragma unroll
          for (int r = 0; r < kHR; ++r) {
            h0[r].x = fma(w0[r], pv.x, h0[r].x);
            h0[r].y = fma(w0[r], pv.y, h0[r].y);
          }
          if (occ) {
            const double2 cv = run[nr + u0 + uu], dv = run[2 * nr + u0 + uu];
#pragma unroll
            for (int r = 0; r < kHR; ++r) {
              h1[r].x = fma(w1[r], cv.x, h1[r].x);
              h1[r].y = fma(w1[r], cv.y, h1[r].y);
              h2[r].x = fma(w2[r], dv.x, h2[r].x);
              h2[r].y = fma(w2[r], dv.y, h2[r].y);
            }
          }
          // position u + 1: r takes r - 1's value, r = 0 the new one
#pragma unroll
          for (int r = kHR - 1; r > 0; --r) {
            w0[r] = w0[r - 1];
            w1[r] = w1[r - 1];
            w2[r] = w2[r - 1];
          }
          const int i = h_skew(vo - t0 + u0 + uu + 1);
          w0[0] = hsm[i];
          w1[0] = hsm[vlen + i];
          w2[0] = hsm[2 * vlen + i];
        }
      }
    }
#pragma unroll
    for (int r = 0; r < kHR; ++r) {
      const int t = t0 + r;
      if (t >= len) break;
      const int k1 = t + o1, k2 = t + o2, e = k1 * nk + k2;
      const double xcv = ((k2 + 1) & 1) ? -dcv : dcv;
      double2 m = rs(-eh * xcv, ex);
      m = cs(m, rs(s.prm.yw, rs(eh * dcv, ey)));
      m = cs(m, rs(s.prm.sgnw, rs(eh * -dcv, ez)));
      double2 hee = cs(dir1, h1[r]), hhh = cs(dir2, h2[r]);
      if (d == 0) {
        hee.x += s.Ee[k1] + s.prm.gap;
        hhh.x += s.Eh[k1];
      }
      s.H[e] = ca(m, h0[r]);
      s.H[n2 + e] = hee;
      s.H[2 * n2 + e] = hhh;
    }
  }
}

// dpdt / dCdt / dDdt (SBEs.py:1952-1975, 2318-2337, 2617-2636) and X3 = X1 +
// 2 dt dX (SBEs.py:5685-5687): twelve complex matrix products of nk x nk,
//   i hbar dp = Hhh p + p Hee^T - Heh^T C - D^T Heh^T + Heh^T - i hbar G p + Off
//   i hbar dC = C Hee^T - Hee^T C + p^H Heh^T - conj(Heh) p
//   i hbar dD = D Hhh^T - Hhh^T D + conj(p) Heh - Heh^H p^T
// on the FP64 matrix instructions.  One CTA computes a TM x TM block of all
// three; per 4 values of the summation index k the 18 operand tiles its
// products read come to shared memory by asynchronous copies, kDStages ahead.
// A warp owns MT x 1 tiles of 8 x 8: 48 MT matrix instructions against 8 + 10
// MT fragment loads per step.  Tiles [row][k] have rows of 4 and tiles
// [k][column] rows of TM + 2 elements of 16 bytes: no bank conflicts.  An
// element's sums run over k in steps of 4 whatever the block size, so its
// bits do not depend on it.  Bound by the FP64 pipe (96 Nk^3 flops per wire,
// 120 of 114 rows and columns computed at Nk 114): 64 wires of Nk 114 take 0.34
// ms, 0.94 with scalar FMAs from 16 x 16 tiles in shared memory.
constexpr int kDStages = 3;
enum DTile {  // [row block][k]: rows of I or J; [k][column block]
  T_HHH_IK, T_P_IK, T_C_IK, T_HEH_IK, T_D_IK, T_HEE_JK, T_HEH_JK, T_HHH_JK, T_P_JK,
  T_HEH_KI, T_D_KI, T_HEE_KI, T_P_KI, T_HHH_KI, T_P_KJ, T_C_KJ, T_D_KJ, T_HEH_KJ, T_NUM,
  T_ROWS = T_HEH_KI
};
// elements of a stage: T_ROWS tiles of 4 TM, the others of 4 (TM + 2)
template <int TM>
constexpr int kDStage = T_ROWS * 4 * TM + (T_NUM - T_ROWS) * 4 * (TM + 2);

template <int TM>
__global__ void __launch_bounds__(TM * 8, TM == 32 ? 2 : 4) derivs_kernel(Step s0) {
  const Step s = at_wire(s0);
  constexpr int MT = TM / 16, NT = TM * 8;  // 8 x 8 tiles per warp, threads
  const int nk = s.nk, n2 = nk * nk, tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  extern __shared__ __align__(16) double2 dsm[];
  const int I0 = blockIdx.x * TM, J0 = blockIdx.z * TM;
  const double2* p = s.L3;
  const double2* C = s.L3 + n2;
  const double2* D = s.L3 + 2 * n2;
  const double2* Heh = s.H;
  const double2* Hee = s.H + n2;
  const double2* Hhh = s.H + 2 * n2;
  // this thread's copies of a stage: element tid % (4 TM) of every second tile
  auto load = [&](int st, int k0) {
    double2* dst = dsm + st * kDStage<TM>;
    const int half = tid / (4 * TM), el = tid % (4 * TM);
    const int r = el >> 2, c = el & 3, kk = el / TM, cc = el % TM;
    auto row_tile = [&](int t, const double2* M, int R0) {
      const bool in = R0 + r < nk && k0 + c < nk;
      cp16(dst + t * 4 * TM + el, in ? M + (R0 + r) * nk + k0 + c : M, in);
    };
    auto col_tile = [&](int t, const double2* M, int C0) {
      const bool in = k0 + kk < nk && C0 + cc < nk;
      cp16(dst + T_ROWS * 4 * TM + (t - T_ROWS) * 4 * (TM + 2) + kk * (TM + 2) + cc,
           in ? M + (k0 + kk) * nk + C0 + cc : M, in);
    };
    if (half == 0) {
      row_tile(T_HHH_IK, Hhh, I0);
      row_tile(T_P_IK, p, I0);
      row_tile(T_C_IK, C, I0);
      row_tile(T_HEH_IK, Heh, I0);
      row_tile(T_D_IK, D, I0);
      col_tile(T_P_KJ, p, J0);
      col_tile(T_C_KJ, C, J0);
      col_tile(T_D_KJ, D, J0);
      col_tile(T_HEH_KJ, Heh, J0);
    } else {
      row_tile(T_HEE_JK, Hee, J0);
      row_tile(T_HEH_JK, Heh, J0);
      row_tile(T_HHH_JK, Hhh, J0);
      row_tile(T_P_JK, p, J0);
      col_tile(T_HEH_KI, Heh, I0);
      col_tile(T_D_KI, D, I0);
      col_tile(T_HEE_KI, Hee, I0);
      col_tile(T_P_KI, p, I0);
      col_tile(T_HHH_KI, Hhh, I0);
    }
  };
  static_assert(NT == 8 * TM, "two tiles per pass of the threads");
  const int wi = (wp & 1) * 8 * MT, wj = (wp >> 1) * 8;  // the warp's rows and columns
  const int fr = lane >> 2, fk = lane & 3;               // fragment row (or column), k
  CAcc dp[MT] = {}, dC[MT] = {}, dD[MT] = {};
  const int nks = (nk + 3) / 4;
#pragma unroll
  for (int st = 0; st < kDStages - 1; ++st) {
    if (st < nks) load(st, 4 * st);
    cp_commit();
  }
  for (int ks = 0; ks < nks; ++ks) {
    cp_wait<kDStages - 2>();
    __syncthreads();
    if (ks + kDStages - 1 < nks) load((ks + kDStages - 1) % kDStages, 4 * (ks + kDStages - 1));
    cp_commit();
    if (J0 + wj >= nk || I0 + wi >= nk) continue;
    const double2* sm = dsm + (ks % kDStages) * kDStage<TM>;
    auto rowf = [&](int t, int r0) { return sm[t * 4 * TM + (r0 + fr) * 4 + fk]; };
    auto colf = [&](int t, int c0) {
      return sm[T_ROWS * 4 * TM + (t - T_ROWS) * 4 * (TM + 2) + fk * (TM + 2) + c0 + fr];
    };
    const double2 b_p = colf(T_P_KJ, wj), b_c = colf(T_C_KJ, wj), b_d = colf(T_D_KJ, wj),
                  b_h = colf(T_HEH_KJ, wj);
    const double2 b_ee = rowf(T_HEE_JK, wj), b_eh = rowf(T_HEH_JK, wj),
                  b_hh = rowf(T_HHH_JK, wj), b_pt = rowf(T_P_JK, wj);
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const int r0 = wi + 8 * m;
      if (m > 0 && I0 + r0 >= nk) break;
      const double2 a_pi = rowf(T_P_IK, r0), a_hki = colf(T_HEH_KI, r0);
      cmma<false>(dp[m], rowf(T_HHH_IK, r0), b_p);
      cmma<false>(dC[m], rowf(T_C_IK, r0), b_ee);
      cmma<false>(dD[m], rowf(T_D_IK, r0), b_hh);
      cmma<false>(dp[m], a_pi, b_ee);
      cmma<false>(dC[m], neg(colf(T_HEE_KI, r0)), b_c);
      cmma<false>(dD[m], neg(colf(T_HHH_KI, r0)), b_d);
      cmma<false>(dp[m], neg(a_hki), b_c);
      cmma<true>(dC[m], colf(T_P_KI, r0), b_eh);
      cmma<true>(dD[m], a_pi, b_h);
      cmma<false>(dp[m], neg(colf(T_D_KI, r0)), b_eh);
      cmma<true>(dC[m], neg(rowf(T_HEH_IK, r0)), b_p);
      cmma<true>(dD[m], neg(a_hki), b_pt);
    }
  }
  const double hb = s.prm.hbar, dt2 = 2.0 * s.prm.dt;
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int i = I0 + wi + 8 * m + fr, j = J0 + wj + 2 * fk + c;
      if (i >= nk || j >= nk) continue;
      const int e = i * nk + j;
      double2 r = ca(make_double2(dp[m].re[c], dp[m].im[c]), Heh[j * nk + i]);
      // GamE[ke] + GamH[kh]: the constant rates, or CalcGammaE/H's
      const double g = s.GamE ? s.GamE[j] + s.GamH[i] : s.prm.gam_e + s.prm.gam_h;
      r = cs(r, cm(make_double2(0.0 * g, hb * g), p[e]));
      if (s.OffP) r = ca(r, s.OffP[e]);  // + OffP[kh][ke]
      s.X3[e] = ca(s.L2[e], rs(dt2, div_ih(r, hb)));
      s.X3[n2 + e] =
          ca(s.L2[n2 + e], rs(dt2, div_ih(make_double2(dC[m].re[c], dC[m].im[c]), hb)));
      s.X3[2 * n2 + e] =
          ca(s.L2[2 * n2 + e], rs(dt2, div_ih(make_double2(dD[m].re[c], dD[m].im[c]), hb)));
    }
}

// Neutrality and reshuffle of the leapfrog (SBEs.py:5704-5718): the sums of
// the new occupations' moduli, then every element of the three levels.
constexpr int kLfThreads = 256;
__global__ void __launch_bounds__(kLfThreads) occ_sums_kernel(Step s0) {
  const Step s = at_wire(s0);
  const int nk = s.nk, n2 = nk * nk;
  __shared__ double red_e[kLfThreads], red_h[kLfThreads];
  double se = 0.0, sh = 0.0;
  for (int k = threadIdx.x; k < nk; k += kLfThreads) {
    const double2 c3 = s.X3[n2 + k * nk + k], d3 = s.X3[2 * n2 + k * nk + k];
    se += hypot(c3.x, c3.y);
    sh += hypot(d3.x, d3.y);
  }
  red_e[threadIdx.x] = se;
  red_h[threadIdx.x] = sh;
  __syncthreads();
  for (int o = kLfThreads / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      red_e[threadIdx.x] += red_e[threadIdx.x + o];
      red_h[threadIdx.x] += red_h[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double small = 1e-200;
    s.fac[0] = (red_e[0] + red_h[0]) / 2.0;
    s.fac[1] = red_e[0] + small;
    s.fac[2] = red_h[0] + small;
  }
}

__global__ void __launch_bounds__(kLfThreads) leapfrog_kernel(Step s0) {
  const Step s = at_wire(s0);
  const int nk = s.nk, n2 = nk * nk;
  const int e = blockIdx.x * kLfThreads + threadIdx.x;
  if (e >= 3 * n2) return;
  const double2 x1 = s.L2[e];
  double2 x3 = s.X3[e];
  const int m = e / n2, r = e - m * n2;
  if (m > 0 && r / nk == r % nk)  // occupation: |X3_kk| total / sum
    x3 = make_double2(hypot(x3.x, x3.y) * s.fac[0] / s.fac[m], 0.0);
  s.L1[e] = x1;
  s.L3[e] = x3;
  s.L2[e] = make_double2((x1.x + x3.x) / 2.0, (x1.y + x3.y) / 2.0);
}

// Wire-space sources of one level: the QWPolarization3 sums (before the
// 2 ehint / (area L) factor and the transform) and the QWRho5 sums (before
// the boundary offset, normalisation and transform),
//   Px(r) = W(r) sum_{kh,ke} Re(conj(Xcv[ke][kh]) p[kh][ke] E[ke] conj(E[kh])),
//   Py, Pz likewise with dcv yw, -dcv (-1)^w,
//   Re(r) = W(r)/(2L) sum_{k1,k2} C[k1][k2] conj(E[k1]) E[k2],
//   Rh(r) = W(r)/(2L) sum_{k1,k2} conj(D[k1][k2]) conj(E[k1]) E[k2],
// E[k] = exp(i kr[k] r) (qwoptics.py:56-84, 367-381); blockIdx.y the wire of a
// batch (levels [nw][3][nk][nk], out [nw][5][nr], yw and (-1)^w from wpar[4 w],
// wpar[4 w + 1] when set).
//
// Polarisation.  On a uniform k grid (the reference's) conj(E[i]) E[c] =
// exp(i (c - i) dk r) depends on c - i alone, so a CTA first sums p along its
// diagonals, plain and with Xcv's sign, thread d over the rows (the threads of
// a warp read neighbouring columns), and then each warp evaluates the 2 nk - 1
// terms of one position after another, the diagonals d and -d together: nk^2 +
// nk nr operations instead of nk^2 nr.  gridDim.x CTAs share the positions of a
// wire; each makes its own diagonal sums.  Phases advance by a rotation of 32
// dk r from an exact first value per lane.  On any other k grid
// densities_kernel takes the sums over (i, c) as they stand, beside its own.

// Whether kr[k] = kr[0] + k dk for all k; every thread of the CTA calls it (a
// barrier).  Two kernels ask, so its rounding is spelled out.
__device__ __forceinline__ bool equidistant(int nk, const double* kr) {
  const double k0 = kr[0], dk = (kr[nk - 1] - k0) / (nk - 1);
  const double tol = 0x1p-47 * fmax(fabs(k0), fabs(kr[nk - 1]));
  bool off = !(fabs(dk) > 0.0);
  for (int k = threadIdx.x; k < nk; k += blockDim.x)
    off |= !(fabs(kr[k] - fma((double)k, dk, k0)) <= tol);
  return !__syncthreads_or(off);
}

// the three components at position r from the sums with and without Xcv's sign
__device__ __forceinline__ void put_polarisation(double2* out, int nr, int r, double W, double dcv,
                                                 double yw, double sgnw, double sx, double sp) {
  out[r] = make_double2(W * dcv * sx, 0.0);
  out[nr + r] = make_double2(W * yw * dcv * sp, 0.0);
  out[2 * nr + r] = make_double2(W * sgnw * -dcv * sp, 0.0);
}

constexpr int kPolThreads = 512, kPolLanes = 128, kPolGroups = kPolThreads / kPolLanes;
__global__ void __launch_bounds__(kPolThreads) polarisation_kernel(
    int nk, int nr, const double* kr, const double* rpos, const double* window, double dcv,
    double yw, double sgnw, const double* wpar, const double2* lev, double2* out) {
  extern __shared__ __align__(16) double2 ssm[];  // [2][2 nk - 1]
  const int nd = 2 * nk - 1, tid = threadIdx.x, lane = tid & 31, wp = tid >> 5;
  const int64_t w = blockIdx.y;
  const double2* p = lev + w * 3 * nk * nk;
  out += w * 5 * nr;
  if (wpar) {
    yw = wpar[4 * w];
    sgnw = wpar[4 * w + 1];
  }
  if (!equidistant(nk, kr)) return;  // densities_kernel's
  const double dk = (kr[nk - 1] - kr[0]) / (nk - 1);
  const int npos = (nr + gridDim.x - 1) / gridDim.x, r0 = blockIdx.x * npos,
            r1 = min(nr, r0 + npos);
  const double2 z = make_double2(0.0, 0.0);
  // diagonal sums: d = c - i at d + nk - 1; row groups add up in turn
  const int grp = tid / kPolLanes;
  for (int d0 = 0; d0 < nd; d0 += kPolLanes) {
    const int di = d0 + tid % kPolLanes, d = di - (nk - 1);
    double2 fx = z, fp = z;
    if (di < nd) {
      const int i0 = d < 0 ? -d : 0, i1 = d < 0 ? nk : nk - d;
#pragma unroll 4
      for (int i = i0 + grp; i < i1; i += kPolGroups) {
        const double2 pv = p[i * nk + i + d];
        fx = ((i + 1) & 1) ? cs(fx, pv) : ca(fx, pv);
        fp = ca(fp, pv);
      }
    }
    for (int g = 0; g < kPolGroups; ++g) {
      if (grp == g && di < nd) {
        ssm[di] = g == 0 ? fx : ca(ssm[di], fx);
        ssm[nd + di] = g == 0 ? fp : ca(ssm[nd + di], fp);
      }
      __syncthreads();
    }
  }
  // positions: Re sum_d F[d] exp(i d phi), phi = dk r
  for (int r = r0 + wp; r < r1; r += kPolThreads / 32) {
    const double phi = dk * rpos[r];
    double2 e, st;
    sincos((double)lane * phi, &e.y, &e.x);
    sincos(32.0 * phi, &st.y, &st.x);
    double sx = 0.0, sp = 0.0;
    for (int d = lane; d < nk; d += 32) {
      const double2* f = ssm + nk - 1;
      // Re(F[d] e + F[-d] conj(e))
      auto term = [&](const double2* g) {
        const double x = g[d].x * e.x - g[d].y * e.y;
        return d == 0 ? x : x + (g[-d].x * e.x + g[-d].y * e.y);
      };
      sx += term(f);
      sp += term(f + nd);
      e = cm(e, st);
    }
    sx = warp_sum(sx);
    sp = warp_sum(sp);
    if (lane == 0) put_polarisation(out, nr, r, window[r], dcv, yw, sgnw, sx, sp);
  }
}

// Densities.  A caller takes the difference of the two (Rho = RhoH - RhoE),
// which cancels to the last digits while electrons and holes move alike, so
// every position's two sums keep the same order and phases: one CTA per R
// positions and wire, the phases of its positions in shared memory, threads
// over the column k2 so the rows of C, D are read coalesced, each element once
// for all R positions and four rows ahead, then a block reduction.  64 wires,
// Nk 114, 230 positions: 0.29 ms (FP64 floor of these products 0.21), with the
// polarisation 0.03 ms; 0.43 with all sums in one kernel of 4 positions.  On a
// k grid that is not equidistant the same pass takes the polarisation's sums
// over (i, c) too: 0.44 ms, one wire of Nk 288 0.17 (1.68 and 2.55 with three
// warps of polarisation_kernel on them).
constexpr int kSrcThreads = 128;
template <int kSrcR>
__global__ void __launch_bounds__(kSrcThreads) densities_kernel(
    int nk, int nr, const double* kr, const double* rpos, const double* window, double L,
    double dcv, double yw, double sgnw, const double* wpar, const double2* lev, double2* out) {
  extern __shared__ double2 ph[];  // [kSrcR][nk]
  __shared__ double red[kSrcR][4][kSrcThreads / 32];
  const int n2 = nk * nk, r0 = blockIdx.x * kSrcR;
  const int64_t w = blockIdx.y;
  lev += w * 3 * n2;
  out += w * 5 * nr;
  for (int e = threadIdx.x; e < kSrcR * nk; e += kSrcThreads) {
    const int j = e / nk, k = e - j * nk;
    const int r = min(r0 + j, nr - 1);
    double sn, cn;
    sincos(kr[k] * rpos[r], &sn, &cn);
    ph[e] = make_double2(cn, sn);
  }
  const bool even = equidistant(nk, kr);  // (a barrier)
  const double2* C = lev + n2;
  const double2* D = lev + 2 * n2;
  double2 se[kSrcR], sh[kSrcR];
  double sx[kSrcR], sp[kSrcR];
#pragma unroll
  for (int j = 0; j < kSrcR; ++j) {
    se[j] = sh[j] = make_double2(0.0, 0.0);
    sx[j] = sp[j] = 0.0;
  }
  auto sums = [&](auto P) {
    constexpr bool POL = decltype(P)::value;  // with the polarisation
    for (int c = threadIdx.x; c < nk; c += kSrcThreads) {
      double2 ec[kSrcR];
#pragma unroll
      for (int j = 0; j < kSrcR; ++j) ec[j] = ph[j * nk + c];
      constexpr int kAhead = 4;
      double2 cb[kAhead], db[kAhead], pb[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int i = min(u, nk - 1);
        cb[u] = C[i * nk + c];
        db[u] = D[i * nk + c];
        if (POL) pb[u] = lev[i * nk + c];
      }
      for (int i0 = 0; i0 < nk; i0 += kAhead) {
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
          const int i = i0 + u, n = min(i + kAhead, nk - 1);
          const double2 cv = cb[u], dv = cconj(db[u]);
          cb[u] = C[n * nk + c];
          db[u] = D[n * nk + c];
          const double2 pv = POL ? pb[u] : make_double2(0.0, 0.0);
          if (POL) pb[u] = lev[n * nk + c];
          if (i >= nk) break;
#pragma unroll
          for (int j = 0; j < kSrcR; ++j) {
            const double2 ei = cconj(ph[j * nk + i]);
            se[j] = ca(se[j], cm(cm(cv, ei), ec[j]));
            sh[j] = ca(sh[j], cm(cm(dv, ei), ec[j]));
            if (POL) {
              const double x = cm(cm(pv, ec[j]), ei).x;
              sx[j] += ((i + 1) & 1) ? -x : x;  // conj(Xcv) / dcv at kh = i
              sp[j] += x;
            }
          }
        }
      }
    }
  };
  if (even)
    sums(std::false_type{});
  else
    sums(std::true_type{});
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < kSrcR; ++j) {
    const double v[4] = {se[j].x, se[j].y, sh[j].x, sh[j].y};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double u = warp_sum(v[q]);
      if (lane == 0) red[j][q][wp] = u;
    }
  }
  __syncthreads();
  if (threadIdx.x < kSrcR) {
    const int j = threadIdx.x, r = r0 + j;
    if (r < nr) {
      double t[4];
      for (int q = 0; q < 4; ++q) {
        t[q] = 0.0;
        for (int u = 0; u < kSrcThreads / 32; ++u) t[q] += red[j][q][u];
      }
      const double W = window[r], h = W / (2.0 * L);
      out[3 * nr + r] = make_double2(h * t[0], h * t[1]);
      out[4 * nr + r] = make_double2(h * t[2], h * t[3]);
    }
  }
  if (even) return;  // polarisation_kernel's
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSrcR; ++j) {
    const double ux = warp_sum(sx[j]), up = warp_sum(sp[j]);
    if (lane == 0) {
      red[j][0][wp] = ux;
      red[j][1][wp] = up;
    }
  }
  __syncthreads();
  const int r = r0 + threadIdx.x;
  if (threadIdx.x >= kSrcR || r >= nr) return;
  double t[2] = {0.0, 0.0};
  for (int u = 0; u < kSrcThreads / 32; ++u) {
    t[0] += red[threadIdx.x][0][u];
    t[1] += red[threadIdx.x][1][u];
  }
  if (wpar) {
    yw = wpar[4 * w];
    sgnw = wpar[4 * w + 1];
  }
  put_polarisation(out, nr, r, window[r], dcv, yw, sgnw, t[0], t[1]);
}

// ---------------------------------------------------------------------------
// Many-body terms switched on by mb.params (PsbFullMB).  Their sums are split
// over lanes and regrouped (each kernel says how): the reference's values to
// rounding, and the same bits for a wire alone and in any batch.
// ---------------------------------------------------------------------------
struct MBView {
  int nk;
  const double* V3;    // screened [3][nk] (VC[q, 0, n])
  const double* Ee;
  const double* Eh;
  const double2* L;    // the level the right-hand side reads (p2, C2, D2)
  double hbar;
  PsbFullMB mb;
  double* GamE;
  double* GamH;
  double* De;          // [(2 nk + 1)][nk]
  double* Dh;
  double2* OffP;
  double2* X3;         // [3][nk][nk]
  double* rates;       // [5][nk]: WinE, WoutE, WinH, WoutH, Rsp
  double2* shift;      // [nk]: circulant kernel of the DC shift; before it [2][nk] occupations
  double2* tr;         // [3][nk][nk]: DC-shift intermediate; before it R1, R2, R4, R3 of
                       // the scattering rates (5 nk^2 doubles at most)
  double gap;          // J
  int lf;
  // a batch of wires (blockIdx.y): byte strides of V3, the levels, the
  // scratch and eps between wires; wpar[4 w + 2] = dc_dk of wire w
  int64_t st_v3, st_lv, st_sc, st_eps;
  const double* wpar;
};

// the MBView of wire blockIdx.y of a batch
__device__ __forceinline__ MBView at_wire(MBView v) {
  const int64_t w = blockIdx.y;
  v.V3 = bump(v.V3, w * v.st_v3);
  v.L = bump(v.L, w * v.st_lv);
  const int64_t b = w * v.st_sc;
  v.GamE = bump(v.GamE, b);
  v.GamH = bump(v.GamH, b);
  v.De = bump(v.De, b);
  v.Dh = bump(v.Dh, b);
  v.OffP = bump(v.OffP, b);
  v.X3 = bump(v.X3, b);
  v.rates = bump(v.rates, b);
  v.shift = bump(v.shift, b);
  v.tr = bump(v.tr, b);
  v.mb.eps = bump(v.mb.eps, w * v.st_eps);
  if (v.wpar) v.mb.dc_dk = v.wpar[4 * w + 2];
  return v;
}

// CalcGammaE / CalcGammaH (dephasing.py:28-105): ne, nh the real parts of
// the diagonal of C2, D2; Vxx2[q] = V(iq[q])^2.  One warp per k, its lanes over
// q (the index maps are read along q), four sums and a reduction: 64 wires of
// Nk 114 take 0.013 ms, 0.12 with a thread per k.
constexpr int kGamWarps = 4;
__global__ void __launch_bounds__(32 * kGamWarps) mb_gamma_kernel(MBView v0) {
  const MBView v = at_wire(v0);
  const int nk = v.nk, k = blockIdx.x * kGamWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k >= nk) return;
  const int n2 = nk * nk;
  const int32_t* kpq = v.mb.maps;
  const int32_t* kmq = kpq + n2;
  const int32_t* k1p = kpq + 2 * n2;
  const int32_t* k1pmq = kpq + 3 * n2;
  const int32_t* k1 = kpq + 4 * n2;
  const int32_t* k1mq = kpq + 5 * n2;
  const double2* C = v.L + n2;
  const double2* D = v.L + 2 * n2;
  auto ne = [&](int i) { return C[i * nk + i].x; };
  auto nh = [&](int i) { return D[i * nk + i].x; };
  auto in = [&](int i) { return i >= 0 && i < nk; };
  const double ph = kPi / v.hbar;
  double ge = 0.0, gh = 0.0;
  for (int q = lane; q < nk; q += 32) {
    const int e = k * nk + q, iq = v.mb.iq[q];
    const double veh = v.V3[iq], vee = v.V3[nk + iq], vhh = v.V3[2 * nk + iq];
    const double xe = fabs(v.mb.xe[q]), xh = fabs(v.mb.xh[q]);
    // electron-electron and hole-hole scattering
    const int a = kpq[e], c = kmq[e];
    if (in(a)) {
      ge = ge + ph * (vee * vee) * ne(a) * (1.0 - ne(a)) * xe;
      gh = gh + ph * (vhh * vhh) * nh(a) * (1.0 - nh(a)) * xh;
    }
    // electron-hole scattering of electrons, of holes
    if (in(c)) {
      const int a1 = k1pmq[e], b1 = k1p[e], a2 = k1mq[e], b2 = k1[e];
      if (in(a1) && in(b1))
        ge = ge + ph * (veh * veh) *
                      (nh(a1) * (1.0 - nh(b1)) * ne(c) + (1.0 - nh(a1)) * nh(b1) * (1.0 - ne(c))) *
                      xh;
      if (in(a2) && in(b2))
        gh = gh + ph * (veh * veh) *
                      (ne(a2) * (1.0 - ne(b2)) * nh(c) + (1.0 - ne(a2)) * ne(b2) * (1.0 - nh(c))) *
                      xe;
    }
  }
  ge = warp_sum(ge);
  gh = warp_sum(gh);
  if (lane == 0) {
    v.GamE[k] = ge;
    v.GamH[k] = gh;
  }
}

// (b / pi) / (x^2 + b^2) and (c / pi) / (y^2 + c^2) with one division
__device__ __forceinline__ void lrtz2(double x, double b, double y, double c, double& lx,
                                      double& ly) {
  const double dx = fma(x, x, __dmul_rn(b, b)), dy = fma(y, y, __dmul_rn(c, c));
  const double r = (1.0 / kPi) / __dmul_rn(dx, dy);
  lx = __dmul_rn(__dmul_rn(b, r), dy);
  ly = __dmul_rn(__dmul_rn(c, r), dx);
}

// CalcOffDiagDeph_E2 / _H2 (dephasing.py:226-318): De[q + nk][k] and
// Dh[q + nk][k] for q in [-nk, nk], with |C_kk|, |D_kk| as occupations and
// Vsq(q) = V(|q|)^2 for 0 < |q| < nk, times pi / hbar: one thread per (q, k),
// the sums over the partner momentum p.  The Lorentzians of the energy
// differences (most of the work, a division each) do not depend on the wire,
// so a CTA takes W wires of the batch: 64 wires of Nk 114 take 0.18 ms with W
// = 8, 0.76 with one wire per CTA.  A wire's own operations and their order do
// not depend on W.
template <int W>
__global__ void __launch_bounds__(128) mb_offd_kernel(MBView v0, int nw) {
  const int nk = v0.nk, n2 = nk * nk, wv0 = blockIdx.y * W;
  extern __shared__ double osm[];  // Ee, Eh [nk]; [2][nk][W]: |C_kk|, |D_kk|
  double* Ee = osm;
  double* Eh = osm + nk;
  double* occ = osm + 2 * nk;
  for (int i = threadIdx.x; i < nk; i += blockDim.x) {
    Ee[i] = v0.Ee[i];
    Eh[i] = v0.Eh[i];
  }
  for (int i = threadIdx.x; i < nk * W; i += blockDim.x) {
    const int w = min(wv0 + i / nk, nw - 1), k = i % nk;
    const double2* L = bump(v0.L, w * v0.st_lv);
    const double2 c = L[n2 + k * nk + k], d = L[2 * n2 + k * nk + k];
    occ[k * W + i / nk] = hypot(c.x, c.y);
    occ[(nk + k) * W + i / nk] = hypot(d.x, d.y);
  }
  __syncthreads();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (2 * nk + 1) * nk) return;
  const int qi = e / nk, k = e - qi * nk, q = qi - nk, kq = k + q;
  const int aq = q < 0 ? -q : q;
  const double* ne = occ;
  const double* nh = occ + nk * W;
  const double hb = v0.hbar;
  const double b_ee = hb * v0.mb.gam_eh, b_eh = hb * v0.mb.gam_h;  // De: gee = g[0], geh = g[2]
  const double b_hh = hb * v0.mb.gam_e;                             // Dh: ghh = g[1], geh = g[2]
  // sums of L n n: same-band (ee, hh), electron-hole (eh, he), per wire
  double see[W], shh[W], seh[W], she[W];
#pragma unroll
  for (int w = 0; w < W; ++w) see[w] = shh[w] = seh[w] = she[w] = 0.0;
  // a (1 - b)(1 - c) + (1 - a) b c, c the occupation at k, as
  // (a - a b) + c (b - a)
  auto add = [&](double& s, double L, double a, double b, double c) {
    s = fma(L, fma(c, b - a, fma(-a, b, a)), s);
  };
  if (kq >= 0 && kq < nk) {
    const double ek = Ee[k], hk = Eh[k], ekq = Ee[kq], hkq = Eh[kq];
    // same-band scattering: partners p and p - q in [1, nk - 1]
    for (int p = max(0, q + 1); p <= min(nk - 1, nk - 1 + q); ++p) {
      const int pm = p - q;
      double le, lh;
      lrtz2(((ekq + Ee[pm]) - Ee[p]) - ek, b_ee, ((hkq + Eh[pm]) - Eh[p]) - hk, b_hh, le, lh);
#pragma unroll
      for (int w = 0; w < W; ++w) {
        add(see[w], le, ne[pm * W + w], ne[p * W + w], ne[k * W + w]);
        add(shh[w], lh, nh[pm * W + w], nh[p * W + w], nh[k * W + w]);
      }
    }
    // electron-hole scattering: partners p and p + q
    for (int p = max(0, -q); p <= min(nk - 1, nk - 1 - q); ++p) {
      const int pp = p + q;
      double le, lh;
      lrtz2(((ekq + Eh[pp]) - Eh[p]) - ek, b_eh, ((hkq + Ee[pp]) - Ee[p]) - hk, b_eh, le, lh);
#pragma unroll
      for (int w = 0; w < W; ++w) {
        add(seh[w], le, nh[pp * W + w], nh[p * W + w], ne[k * W + w]);
        add(she[w], lh, ne[pp * W + w], ne[p * W + w], nh[k * W + w]);
      }
    }
  }
#pragma unroll
  for (int w = 0; w < W; ++w) {
    const int wv = wv0 + w;
    if (wv >= nw) break;
    const double* V3 = bump(v0.V3, wv * v0.st_v3);
    double vs[3];
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      const double x = (aq > 0 && aq < nk) ? V3[t * nk + aq] : 0.0;
      vs[t] = __dmul_rn(x, x);
    }
    const double f = kPi / hb;
    bump(v0.De, wv * v0.st_sc)[e] = fma(vs[1], see[w], __dmul_rn(vs[0], seh[w])) * f;
    bump(v0.Dh, wv * v0.st_sc)[e] = fma(vs[2], shh[w], __dmul_rn(vs[0], she[w])) * f;
  }
}

// OffDiagDephasing2 (dephasing.py:320-359): x[kh][ke] = i hbar (sum_q
// Dh[q][kh] p[kh + q][ke] + sum_q De[q][ke] p[kh][ke + q]), q != 0: two
// products of p with the real matrices MH[kh][k'] = Dh[k' - kh][kh] and
// ME[k'][ke] = De[k' - ke][ke] (zero for k' = kh, ke) on the FP64 matrix
// instructions.  One CTA per 32 x 32 block, a warp per 16 x 8 of it; per 8
// values of k' the four operand tiles come through shared memory, read one
// step ahead.  64 wires of Nk 114: 0.04 ms, 0.23 with a thread per element.
constexpr int kOT = 32, kOK = 8;
__global__ void __launch_bounds__(256) mb_offp_kernel(MBView v0) {
  const MBView v = at_wire(v0);
  const int nk = v.nk, nb = (nk + kOT - 1) / kOT, tid = threadIdx.x;
  const int I0 = (blockIdx.x / nb) * kOT, J0 = (blockIdx.x % nb) * kOT;
  const int lane = tid & 31, wp = tid >> 5, fr = lane >> 2, fk = lane & 3;
  // [row][k'] with rows of kOK + 4, [k'][column] with rows of kOT + 2 (p) and
  // + 4 (ME): no bank conflicts in the fragments
  __shared__ double mh[kOT][kOK + 4], me[kOK][kOT + 4];
  __shared__ double2 pi[kOT][kOK + 4], pj[kOK][kOT + 2];
  const double2* p = v.L;
  const double2 z = make_double2(0.0, 0.0);
  const int lr = tid >> 3, lk = tid & 7, ck = tid >> 5, cc = tid & 31;
  double nh, ne;
  double2 npi, npj;
  auto fetch = [&](int k0) {
    const int kh = I0 + lr, kr = k0 + lk, kc = k0 + ck, ke = J0 + cc;
    const bool inr = kh < nk && kr < nk, inc = kc < nk && ke < nk;
    nh = inr && kr != kh ? v.Dh[(kr - kh + nk) * nk + kh] : 0.0;
    npi = inr ? p[kh * nk + kr] : z;
    ne = inc && kc != ke ? v.De[(kc - ke + nk) * nk + ke] : 0.0;
    npj = inc ? p[kc * nk + ke] : z;
  };
  const int wi = (wp & 1) * 16, wj = (wp >> 1) * 8;
  CAcc acc[2] = {};
  fetch(0);
  for (int k0 = 0; k0 < nk; k0 += kOK) {
    __syncthreads();
    mh[lr][lk] = nh;
    pi[lr][lk] = npi;
    me[ck][cc] = ne;
    pj[ck][cc] = npj;
    __syncthreads();
    if (k0 + kOK < nk) fetch(k0 + kOK);
#pragma unroll
    for (int s = 0; s < kOK; s += 4) {
      const double2 bp = pj[s + fk][wj + fr];
      const double be = me[s + fk][wj + fr];
#pragma unroll
      for (int m = 0; m < 2; ++m) {
        const double ah = mh[wi + 8 * m + fr][s + fk];
        const double2 ap = pi[wi + 8 * m + fr][s + fk];
        dmma(acc[m].re, ah, bp.x);
        dmma(acc[m].im, ah, bp.y);
        dmma(acc[m].re, ap.x, be);
        dmma(acc[m].im, ap.y, be);
      }
    }
  }
#pragma unroll
  for (int m = 0; m < 2; ++m)
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int kh = I0 + wi + 8 * m + fr, ke = J0 + wj + 2 * fk + c;
      if (kh < nk && ke < nk)  // x * i * hbar
        v.OffP[kh * nk + ke] = make_double2(-acc[m].im[c] * v.hbar, acc[m].re[c] * v.hbar);
    }
}

// In/out scattering rates of the new occupations (SBESolver._relaxation_E/H,
// SBEs.py:5248-5291): MBCE / MBCH (coulomb.py:957-1071) with |Re n|, k3(a, b,
// c) = a + b - c, and the reference's C arrays read at [k - 1][..][..] (its
// 1-based grid; row 0 of an array is zero); then MBPE / MBPH (phonons.py:
// 140-271) with Re n; with recomb also SpontEmission's Rsp.
//
// The eight double sums are built from four families of single sums,
//   R1[k][k1] = sum_kp Ceh[k][kp][k1] (1 - nh[kp]) nh[kp + k1 - k]
//   R2[k][k4] = sum_k2 Cee[k][k2][k4] (1 - ne[k2]) ne[k2 + k - k4]
//   R4 as R2 with Chh and nh
//   R3[kp][d] = sum_kk Ceh[kk][kp][kk + d] (1 - ne[kk]) ne[kk + d]
// e.g. electrons in: sum_k1 Veh^2(k - k1) ne[k1] R1[k][k1] + ..., electrons out:
// sum_k1 Veh^2(k - k1) (1 - ne[k1]) R1[k1][k] + ....  For a fixed difference d
// (k1 - k or k4 - k) each family is one matrix product: the slice of C with
// that difference, the same for every wire, times the occupation products of
// the batch's wires.  mb_scatter_kernel does these on the FP64 matrix
// instructions, one CTA per (d, family) and 8 NT wires; mb_rates_kernel adds
// up per (k, wire).  A wire's column does not depend on the others.  64 wires
// of Nk 114: 0.14 ms, bound by the strided reads of the slices of C (L2); 1.15
// with the double sums per (k, wire), which read C once per wire.
__global__ void mb_occ_kernel(MBView v0) {
  const MBView v = at_wire(v0);
  const int nk = v.nk, i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nk) return;
  double* occ = reinterpret_cast<double*>(v.shift);  // [2][nk], free until the DC shift
  occ[i] = fabs(v.X3[nk * nk + i * nk + i].x);
  occ[nk + i] = fabs(v.X3[2 * nk * nk + i * nk + i].x);
}

constexpr int kScWarps = 8, kScK = 128;  // k values of the occupation products at a time
// rows of the occupation products: 8 NT wires + 4 (no bank conflicts)
__host__ __device__ constexpr int sc_ld(int nt) { return 8 * nt + 4; }

template <int NT>
__global__ void __launch_bounds__(32 * kScWarps) mb_scatter_kernel(MBView v0, int nw) {
  const int nk = v0.nk, n2 = nk * nk, N1 = nk + 1;
  const int d = (int)blockIdx.x - (nk - 1), fam = blockIdx.y, w0 = blockIdx.z * 8 * NT;
  const int tid = threadIdx.x, lane = tid & 31, wp = tid >> 5, fr = lane >> 2, fk = lane & 3;
  extern __shared__ double gsm[];  // [kScK][sc_ld(NT)]
  const int lo = d < 0 ? -d : 0, hi = d < 0 ? nk : nk - d;  // i with i and i + d on the grid
  const size_t cs3 = (size_t)N1 * N1 * N1;
  // families 0, 1, 2: rows k of [lo, hi), summed over all kp; 3: rows kp, over kk
  const double* C = v0.mb.C + (fam == 1 ? cs3 : (fam == 2 ? 2 * cs3 : 0)) + d;
  const bool by_row = fam < 3;
  const int row_lo = by_row ? lo : 0, row_hi = by_row ? hi : nk;
  const int sum_lo = by_row ? 0 : lo, sum_hi = by_row ? nk : hi;
  const size_t row_st = by_row ? (size_t)N1 * N1 + 1 : N1;
  const size_t sum_st = by_row ? N1 : (size_t)N1 * N1 + 1;
  // partner of i in the occupation products, the occupations it takes
  const int pd = fam == 1 || fam == 2 ? -d : d, band = fam == 0 || fam == 2 ? 1 : 0;
  const int tiles = (row_hi - row_lo + 7) / 8, chunks = (sum_hi - sum_lo + kScK - 1) / kScK;
  for (int t0 = 0; t0 < tiles; t0 += kScWarps) {
    const int row = row_lo + 8 * (t0 + wp) + fr;
    double acc[NT][2];
#pragma unroll
    for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = 0.0;
    for (int c = 0; c < chunks; ++c) {
      const int s0 = sum_lo + c * kScK, sn = min(kScK, sum_hi - s0);
      if (t0 == 0 || chunks > 1) {
        __syncthreads();
        for (int e = tid; e < kScK * 8 * NT; e += 32 * kScWarps) {
          const int w = e / kScK, i = e % kScK, k = s0 + i, r = k + pd;
          double g = 0.0;
          if (i < sn && r >= 0 && r < nk && w0 + w < nw) {
            const double* o = reinterpret_cast<const double*>(
                                  bump(v0.shift, (int64_t)(w0 + w) * v0.st_sc)) + band * nk;
            g = (1.0 - o[k]) * o[r];
          }
          gsm[i * sc_ld(NT) + w] = g;
        }
        __syncthreads();
      }
      if (t0 + wp >= tiles) continue;
      const double* a = C + (size_t)row * row_st + (size_t)(s0 + fk) * sum_st;
      const bool in = row < row_hi;
#pragma unroll 8
      for (int k = 0; k < sn; k += 4) {
        const double x = in && k + fk < sn ? a[(size_t)k * sum_st] : 0.0;
        const double* b = gsm + (k + fk) * sc_ld(NT) + fr;
#pragma unroll
        for (int n = 0; n < NT; ++n) dmma(acc[n], x, b[8 * n]);
      }
    }
    if (row >= row_hi || t0 + wp >= tiles) continue;
    // families 0, 1, 2 at [k][k + d], family 3 at [kp][d + nk - 1]
    const size_t o = (size_t)fam * n2 +
                     (by_row ? (size_t)row * nk + row + d : (size_t)row * (2 * nk - 1) + blockIdx.x);
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int w = w0 + 8 * n + 2 * fk + u;
        if (w < nw)
          reinterpret_cast<double*>(bump(v0.tr, (int64_t)w * v0.st_sc))[o] = acc[n][u];
      }
  }
}

constexpr int kRateThreads = 128;

// sum of K values over the CTA (kRateThreads threads); every thread gets them
template <int K>
__device__ __forceinline__ void rate_block_sum(double (&v)[K], double (*red)[kRateThreads / 32]) {
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < K; ++q) {
    const double u = warp_sum(v[q]);
    if (lane == 0) red[q][wp] = u;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < K; ++q) {
    double t = 0.0;
    for (int u = 0; u < kRateThreads / 32; ++u) t += red[q][u];
    v[q] = t;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(kRateThreads) mb_rates_kernel(MBView v0) {
  const MBView v = at_wire(v0);
  const int nk = v.nk, k0 = blockIdx.x;
  const int n2 = nk * nk;
  __shared__ double red[4][kRateThreads / 32];
  const double2* C3 = v.X3 + n2;
  const double2* D3 = v.X3 + 2 * n2;
  double acc[4] = {0.0, 0.0, 0.0, 0.0};  // WinE, WoutE, WinH, WoutH
  if (v.mb.ehs) {
    const double* R1 = reinterpret_cast<const double*>(v.tr);
    const double* R2 = R1 + n2;
    const double* R4 = R2 + n2;
    const double* R3 = R4 + n2;
    const double* ne = reinterpret_cast<const double*>(v.shift);
    const double* nh = ne + nk;
    for (int i = threadIdx.x; i < nk; i += kRateThreads) {
      const int q = i > k0 ? i - k0 : k0 - i;
      const double veh = v.V3[q], vee = v.V3[nk + q], vhh = v.V3[2 * nk + q];
      const double eh2 = veh * veh, ee2 = vee * vee, hh2 = vhh * vhh;
      const int a = k0 * nk + i, b = i * nk + k0;
      // MBCE: from i into k0, from k0 into i
      acc[0] += ne[i] * (eh2 * R1[a] + ee2 * R2[a]);
      acc[1] += (1.0 - ne[i]) * (eh2 * R1[b] + ee2 * R2[b]);
      // MBCH: the partner hole at i = kp + d, and at i = kp - d
      acc[2] += nh[i] * (eh2 * R3[k0 * (2 * nk - 1) + i - k0 + nk - 1] + hh2 * R4[a]);
      acc[3] += (1.0 - nh[i]) * (eh2 * R3[i * (2 * nk - 1) + k0 - i + nk - 1] + hh2 * R4[b]);
    }
  }
  rate_block_sum<4>(acc, red);
  if (v.mb.phonon) {
    // Vep[k][i] = VC_ee[k][i] / E1D[k][i] * Vscale (VC already screened)
    const double* EP = v.mb.ph;
    const double* EPT = EP + n2;
    const double* HP = EP + 2 * n2;
    const double* HPT = EP + 3 * n2;
    double ph[4] = {0.0, 0.0, 0.0, 0.0};
    for (int i = threadIdx.x; i < nk; i += kRateThreads) {
      const int d = i > k0 ? i - k0 : k0 - i;
      const double e = v.mb.eps ? v.mb.eps[d] : 1.0;
      const double vep = v.V3[nk + d] / e * v.mb.vscale;
      const double vhp = v.V3[2 * nk + d] / e * v.mb.vscale;
      const double nei = C3[i * nk + i].x, nhi = D3[i * nk + i].x;
      ph[0] += vep * nei * EPT[i * nk + k0];
      ph[1] += vep * (1.0 - nei) * EP[i * nk + k0];
      ph[2] += vhp * nhi * HPT[i * nk + k0];
      ph[3] += vhp * (1.0 - nhi) * HP[i * nk + k0];
    }
    rate_block_sum<4>(ph, red);
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] = acc[q] + ph[q];
  }
  double rsp = 0.0;
  if (v.mb.recomb) {
    // SpontEmission (emission.py:94-131) from the level the right-hand side
    // reads (SBEs.py:5237-5238): Ec (emission.py:133-172) with Re n and the
    // screened V, Ek = gap + Ee + Eh + Ec, then SpontIntegral
    // (emission.py:174-199): sum_n x rho0(x) square_n dhw, x = HOmega_n + Ek,
    // rho0(x) = x^2 / (c0^3 pi^2 hbar^3)
    const double2* C2 = v.L + n2;
    const double2* D2 = v.L + 2 * n2;
    const double veh0 = v.V3[0], vee0 = v.V3[nk], vhh0 = v.V3[2 * nk];
    double ec[2] = {0.0, 0.0};
    for (int i = threadIdx.x; i < nk; i += kRateThreads) {
      const int d = i > k0 ? i - k0 : k0 - i;
      const double ne = C2[i * nk + i].x, nh = D2[i * nk + i].x;
      ec[0] += ne * (vee0 - v.V3[nk + d]) + nh * (vhh0 - v.V3[2 * nk + d]);
      const double id = i == k0 ? 0.0 : 1.0;
      ec[1] += ne * veh0 * id - nh * veh0 * id;
    }
    rate_block_sum<2>(ec, red);
    const double ek = ((v.gap + v.Ee[k0]) + v.Eh[k0]) + ((ec[0] + ec[1]) - veh0);
    const double* hw = v.mb.emis;
    const double* sq = hw + v.mb.n_hw;
    double it[1] = {0.0};
    for (int n = threadIdx.x; n < v.mb.n_hw; n += kRateThreads) {
      const double x = hw[n] + ek;
      it[0] += x * (x * x / v.mb.rho0_den) * sq[n];
    }
    rate_block_sum<1>(it, red);
    rsp = it[0] * v.mb.dhw;
  }
  if (threadIdx.x == 0) {
    v.rates[k0] = acc[0];
    v.rates[nk + k0] = acc[1];
    v.rates[2 * nk + k0] = acc[2];
    v.rates[3 * nk + k0] = acc[3];
    if (v.mb.recomb) v.rates[4 * nk + k0] = rsp;
  }
}

// n <- exp(-W dt) ((-1 + exp(W dt) + n) Win + n Wout) / (W + small), W = Win
// + Wout, on the diagonal of C3 and D3 (SBEs.py:5322-5331).
__global__ void mb_relax_kernel(MBView v0, double dt) {
  const MBView v = at_wire(v0);
  const int nk = v.nk, k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nk) return;
  const int n2 = nk * nk;
  const double small = 1e-200;
  for (int b = 0; b < 2; ++b) {
    const double win = v.rates[2 * b * nk + k], wout = v.rates[(2 * b + 1) * nk + k];
    const double W = win + wout;
    double2* c = v.X3 + (1 + b) * n2 + k * nk + k;
    const double2 n = *c;
    const double em = exp(-W * dt), ep = exp(W * dt);
    const double2 s1 = make_double2((-1.0 + ep) + n.x, n.y);
    const double2 s = make_double2(s1.x * win + n.x * wout, s1.y * win + n.y * wout);
    const double den = W + small;
    *c = make_double2(em * s.x / den, em * s.y / den);
  }
  if (v.mb.recomb) {
    // n_e *= exp(-Rsp n_h dt), then n_h *= exp(-Rsp n_e dt) with the new
    // n_e (SBEs.py:5335-5337), complex as the reference's ne3, nh3
    const double r = v.rates[4 * nk + k];
    double2* ce = v.X3 + n2 + k * nk + k;
    double2* ch = v.X3 + 2 * n2 + k * nk + k;
    auto cexp_ = [](double x, double y) {
      const double m = exp(x);
      return make_double2(m * cos(y), m * sin(y));
    };
    const double2 nh = *ch;
    const double2 ne = cm(*ce, cexp_(-r * nh.x * dt, -r * nh.y * dt));
    *ce = ne;
    *ch = cm(nh, cexp_(-r * ne.x * dt, -r * ne.y * dt));
  }
}

// DC transport (Transport, dcfield.py:1213-1247): ShiftN1D / ShiftN2D move
// a vector or matrix in k by fft -> times exp(-i Y dk) -> ifft
// (dcfield.py:1169-1211), i.e. a circular convolution with
//   s[d] = (1/nk) sum_m exp(-i Y_m dk) exp(2 pi i m d / nk),
// applied along both indices of each matrix (lf) or to its diagonal.
// One CTA per wire: the phases exp(-i Y_m dk) and the roots of nk in shared
// memory, thread d sums over m (64 wires of Nk 114: 0.01 ms; 0.06 with both
// evaluated per (m, d)).
constexpr int kShThreads = 128;
__global__ void __launch_bounds__(kShThreads) mb_shift_kernel(MBView v0) {
  const MBView v = at_wire(v0);
  const int nk = v.nk;
  extern __shared__ double2 shs[];  // [nk] phases, [nk] roots
  for (int i = threadIdx.x; i < nk; i += kShThreads) {
    sincos(-v.mb.Y[i] * v.mb.dc_dk, &shs[i].y, &shs[i].x);
    sincospi(2.0 * i / nk, &shs[nk + i].y, &shs[nk + i].x);
  }
  __syncthreads();
  for (int d = threadIdx.x; d < nk; d += kShThreads) {
    double re = 0.0, im = 0.0;
    int r = 0;  // m d mod nk
    for (int m = 0; m < nk; ++m) {
      const double cy = shs[m].x, sy = shs[m].y, cw = shs[nk + r].x, sw = shs[nk + r].y;
      re += fma(cy, cw, -__dmul_rn(sy, sw));  // (rounding: see cm_rn)
      im += fma(cy, sw, __dmul_rn(sy, cw));
      r += d;
      if (r >= nk) r -= nk;
    }
    v.shift[d] = make_double2(re / nk, im / nk);
  }
}

// The complex product with its rounding spelled out: a caller's charge density
// is the difference of two densities of the shifted C and D and cancels to the
// last digits, so their bits stay.
__device__ __forceinline__ double2 cm_rn(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -__dmul_rn(a.y, b.y)), fma(a.y, b.x, __dmul_rn(a.x, b.y)));
}

// The two circulant products of the shift, tiled: one CTA per 32 x 32 block of
// one matrix (x) of one wire, a warp per 8 rows, a lane per column; per chunk
// of kST summation indices the block's operand tile and the coefficients s[(j -
// b) mod nk] it needs sit in shared memory, and a lane's eight sums share the
// operand that varies along the columns (the other is a broadcast).  Bound by
// the FP64 pipe.  Each element sums with the summation index ascending.
// 64 wires of Nk 114: 0.16 ms each, 0.23 with one element per thread.
constexpr int kST = 16, kSB = 32, kSR = 8, kSThreads = kSB / kSR * 32;

// ROWS: T[x][a][j] = sum_b X3[x][a][b] s[(j - b) mod nk], into tr;
// else X3[x][i][j] = sum_a s[(i - a) mod nk] T[x][a][j], into X3
template <bool ROWS>
__global__ void __launch_bounds__(kSThreads) mb_shift_mat_kernel(MBView v0) {
  const MBView v = at_wire(v0);
  const int nk = v.nk, n2 = nk * nk, nb = (nk + kSB - 1) / kSB;
  const int x = blockIdx.x / (nb * nb), t = blockIdx.x % (nb * nb);
  const int I0 = (t / nb) * kSB, J0 = (t % nb) * kSB;
  const int tid = threadIdx.x, lane = tid & 31, r0 = (tid >> 5) * kSR;
  __shared__ double2 xt[ROWS ? kSB : kST][ROWS ? kST + 1 : kSB + 1];
  __shared__ double2 sv[kSB + kST - 1];
  const double2* X = (ROWS ? v.X3 : v.tr) + (size_t)x * n2;
  double2 acc[kSR];
#pragma unroll
  for (int r = 0; r < kSR; ++r) acc[r] = make_double2(0.0, 0.0);
  const int S0 = ROWS ? J0 : I0;  // output index the coefficients run over
  for (int b0 = 0; b0 < nk; b0 += kST) {
    for (int e = tid; e < kSB * kST; e += kSThreads) {
      const int er = ROWS ? e / kST : e / kSB, ec = ROWS ? e % kST : e % kSB;
      const int r = (ROWS ? I0 : b0) + er, c = (ROWS ? b0 : J0) + ec;
      xt[er][ec] = (r < nk && c < nk) ? X[r * nk + c] : make_double2(0.0, 0.0);
    }
    for (int u = tid; u < kSB + kST - 1; u += kSThreads) {
      // sv[u] = s[(S0 - b0 - (kST - 1) + u) mod nk]
      int d = (S0 - b0 - (kST - 1) + u) % nk;
      if (d < 0) d += nk;
      sv[u] = v.shift[d];
    }
    __syncthreads();
    const int bn = min(kST, nk - b0);
    if (I0 + r0 < nk)
      for (int bb = 0; bb < bn; ++bb) {
        if (ROWS) {
          const double2 c = sv[lane - bb + kST - 1];
#pragma unroll
          for (int r = 0; r < kSR; ++r) acc[r] = ca(acc[r], cm_rn(xt[r0 + r][bb], c));
        } else {
          const double2 c = xt[bb][lane];
#pragma unroll
          for (int r = 0; r < kSR; ++r) acc[r] = ca(acc[r], cm_rn(sv[r0 + r - bb + kST - 1], c));
        }
      }
    __syncthreads();
  }
  double2* out = (ROWS ? v.tr : v.X3) + (size_t)x * n2;
#pragma unroll
  for (int r = 0; r < kSR; ++r) {
    const int i = I0 + r0 + r, j = J0 + lane;
    if (i < nk && j < nk) out[i * nk + j] = acc[r];
  }
}

// without lf only the diagonals move: T[x][a] = sum_n s[(a - n) mod nk] X3[x][n][n]
__global__ void mb_shift_diag_kernel(MBView v0) {
  const MBView v = at_wire(v0);
  const int nk = v.nk, n2 = nk * nk, e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 3 * nk) return;
  const int x = e / nk, a = e % nk;
  const double2* X = v.X3 + (size_t)x * n2;
  double2 acc = make_double2(0.0, 0.0);
  for (int n = 0; n < nk; ++n) {
    const int d = a - n < 0 ? a - n + nk : a - n;
    acc = ca(acc, cm(v.shift[d], X[n * nk + n]));
  }
  v.tr[e] = acc;
}

__global__ void mb_shift_diag_store_kernel(MBView v0) {
  const MBView v = at_wire(v0);
  const int nk = v.nk, e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 3 * nk) return;
  const int x = e / nk, a = e % nk;
  v.X3[(size_t)x * nk * nk + a * nk + a] = v.tr[e];
}

// CalcMBArrays (coulomb.py:367-499) on the (nk+1)^3 grid the reference
// allocates (index 0 unused); UnDel(i, j) = 0 on row/column 0 and the
// diagonal, else 1 (coulomb.py:336-366).  One thread per entry.
__global__ void mb_tables_kernel(int nk, const double* Ee, const double* Eh, double ge,
                                 double gh, double hb, int lorentz, double* Ceh) {
  const int N1 = nk + 1;
  const size_t n3 = (size_t)N1 * N1 * N1;
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n3) return;
  double* Cee = Ceh + n3;
  double* Chh = Ceh + 2 * n3;
  const int a = (int)(e / ((size_t)N1 * N1)), bb = (int)((e / N1) % N1), c = (int)(e % N1);
  Ceh[e] = Cee[e] = Chh[e] = 0.0;
  if (a == 0 || bb == 0 || c == 0) return;
  const int k1 = a - 1, k2 = bb - 1, k4 = c - 1;
  auto undel = [&](int i, int j) { return (i == 0 || j == 0 || i == j) ? 0.0 : 1.0; };
  auto gdelta = [&](double x, double w) {
    if (fabs(w) < 1e-300) return 0.0;
    return 1.0 / (sqrt(kPi) * w) * exp(-((x / w) * (x / w)));
  };
  const double geh = (ge + gh) / 2.0;
  const double twopi = 2.0 * kPi;
  // Veh(k1, k2, k30, k4), k30 = k3[k4, k2, k1]
  int r = (k4 + 1) + (k2 + 1) - (k1 + 1);
  if (r >= 1 && r <= nk) {
    const int k30 = r - 1;
    const double Ed = Ee[k1] + Eh[k2] - Eh[k30] - Ee[k4];
    if (lorentz) {
      const double h2 = (hb * geh) * (hb * geh);
      Ceh[e] = 2.0 * geh * undel(a, c) * undel(bb, r) / (Ed * Ed + h2);
    } else {
      Ceh[e] = twopi / hb * undel(a, c) * undel(bb, r) * gdelta(Ed, hb * geh);
    }
  }
  // Vee / Vhh(k1, k2, k30, k4), k30 = k3[k1, k2, k4]
  r = (k1 + 1) + (k2 + 1) - (k4 + 1);
  if (r >= 1 && r <= nk) {
    const int k30 = r - 1;
    const double Ede = Ee[k1] + Ee[k2] - Ee[k30] - Ee[k4];
    const double Edh = Eh[k1] + Eh[k2] - Eh[k30] - Eh[k4];
    if (lorentz) {
      Cee[e] = 2.0 * ge * undel(a, c) * undel(bb, r) / (Ede * Ede + (hb * ge) * (hb * ge));
      Chh[e] = 2.0 * gh * undel(a, c) * undel(bb, r) / (Edh * Edh + (hb * gh) * (hb * gh));
    } else {
      Cee[e] = twopi / hb * undel(a, c) * undel(bb, r) * gdelta(Ede, hb * ge);
      Chh[e] = twopi / hb * undel(a, c) * undel(bb, r) * gdelta(Edh, hb * gh);
    }
  }
}

// Screening of a batch (CalcScreenedArrays, coulomb.py:1195-1230), one CTA
// per wire: n1D from the diagonals of the level the right-hand side reads,
// eps(q; n1D) of the grid's table block and V3 = V0 / eps.  The n1D sum
// has psb_screen_f64's thread mapping and tree, so a wire's V3 is the same
// bits as the one-wire path's.
constexpr int kScrThreads = 256;
__global__ void __launch_bounds__(kScrThreads) screen_batch_kernel(Step s0, const double* tab,
                                                                   double L, double dens_max,
                                                                   double* eps, double* V3) {
  const Step s = at_wire(s0);
  const int nk = s.nk, n2 = nk * nk;
  const int64_t w = blockIdx.y;
  eps = bump(eps, w * s.st_v3);
  V3 = bump(V3, w * s.st_v3);
  const double2* C = s.L3 + n2;
  const double2* D = s.L3 + 2 * n2;
  double t = 0.0;
  for (int k = threadIdx.x; k < nk; k += kScrThreads) t += C[k * nk + k].x + D[k * nk + k].x;
  __shared__ double red[kScrThreads / 32];
  __shared__ double n1d_s;
  t = warp_sum(t);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
  __syncthreads();
  if (threadIdx.x == 0) {
    double u = 0.0;
    for (int i = 0; i < kScrThreads / 32; ++i) u += red[i];
    const double n1d = u / 2.0 / L;
    n1d_s = n1d < dens_max ? n1d : dens_max;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < nk; q += kScrThreads) {
    const double e = eps1d(tab, nk, q, n1d_s);
    eps[q] = e;
    V3[q] = tab[q] / e;
    V3[nk + q] = tab[nk + q] / e;
    V3[2 * nk + q] = tab[2 * nk + q] / e;
  }
}

}  // namespace full
}  // namespace psb

using namespace psb;

extern "C" int64_t psb_full_work_bytes(int nk) {
  if (nk < 2 || nk > PSB_MAX_NK) return set_error(PSB_ERR_SIZE, "nk %d out of range", nk);
  return (int64_t)7 * nk * nk * 16;
}

namespace {
// scratch of the many-body terms: GamE, GamH, De, Dh, OffP, X3, rates
// (+ Rsp), the DC-shift kernel and intermediate
struct MBScratch {
  size_t gam, de, dh, offp, x3, rates, shift, tr, total;
  explicit MBScratch(int nk) {
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    const size_t n = (size_t)nk, n2 = n * n, nd = (2 * n + 1) * n;
    gam = 0;
    de = al(gam + 2 * n * 8);
    dh = al(de + nd * 8);
    offp = al(dh + nd * 8);
    x3 = al(offp + n2 * 16);
    rates = al(x3 + 3 * n2 * 16);
    shift = al(rates + 5 * n * 8);
    tr = al(shift + n * 16);
    total = al(tr + 3 * n2 * 16);
  }
};
}  // namespace

extern "C" int64_t psb_full_mb_scratch_bytes(int nk) {
  if (nk < 2 || nk > PSB_MAX_NK) return set_error(PSB_ERR_SIZE, "nk %d out of range", nk);
  return (int64_t)MBScratch(nk).total;
}

extern "C" int psb_mb_tables_f64(int nk, const double* d_Ee, const double* d_Eh, double ge,
                                 double gh, double hbar, int lorentz, double* d_C,
                                 void* stream) {
  if (!d_Ee || !d_Eh || !d_C) return set_error(PSB_ERR_INVALID, "psb_mb_tables_f64: null pointer");
  if (nk < 2 || nk > PSB_MAX_NK) return set_error(PSB_ERR_SIZE, "psb_mb_tables_f64: nk %d", nk);
  if (!(hbar > 0.0)) return set_error(PSB_ERR_INVALID, "hbar must be > 0");
  const size_t n3 = (size_t)(nk + 1) * (nk + 1) * (nk + 1);
  const int th = 256;
  const unsigned bl = (unsigned)((n3 + th - 1) / th);
  full::mb_tables_kernel<<<bl, th, 0, (cudaStream_t)stream>>>(nk, d_Ee, d_Eh, ge, gh, hbar,
                                                               lorentz ? 1 : 0, d_C);
  return check_cuda("psb_mb_tables_f64");
}

namespace {
// per-wire work of a batch: seven matrices' room (the occupations' sums in the
// first, H in the next three, X1 + 2 dt dX in the last three), then the screened
// V3 and eps
struct BatchWork {
  size_t v3, eps, total;
  explicit BatchWork(int nk) {
    auto al = [](size_t x) { return (x + 255) & ~(size_t)255; };
    v3 = al((size_t)7 * nk * nk * 16);
    eps = al(v3 + 3 * (size_t)nk * 8);
    total = al(eps + (size_t)nk * 8);
  }
};

// one full-matrix step of nw wires of one grid (nw = 1: the one-wire entry)
struct Launch {
  int nw, nk, nr, nq0;
  const double* V3;
  int64_t st_v3;         // bytes between wires' V3 (0: shared)
  const double* Ee;
  const double* Eh;
  const double* fields;  // [nw][3][nr] complex
  const PsbFullParams* params;
  const double* wpar;    // [nw][4] or null
  const PsbFullMB* mb;
  double* L1;
  double* L2;
  double* L3;
  void* work;
  int64_t st_wk;         // bytes between wires' work
  const double* tab;     // screened batch: the grid's table block, else null
  double L, dens_max;
};

int check_mb(const PsbFullMB* mb, bool deph, bool relax, bool dct) {
  if (!(deph || relax || dct)) return PSB_OK;
  if (!mb->scratch) return set_error(PSB_ERR_INVALID, "PsbFullMB.scratch is null");
  if (mb->diag_dph && (!mb->maps || !mb->iq || !mb->xe || !mb->xh))
    return set_error(PSB_ERR_INVALID, "PsbFullMB: dephasing tables missing");
  if ((mb->ehs && !mb->C) || (mb->phonon && !mb->ph))
    return set_error(PSB_ERR_INVALID, "PsbFullMB: relaxation tables missing");
  if (relax && mb->recomb && (!mb->emis || mb->n_hw < 2 || !(mb->rho0_den > 0.0)))
    return set_error(PSB_ERR_INVALID, "PsbFullMB: emission tables missing");
  if (dct && !mb->Y) return set_error(PSB_ERR_INVALID, "PsbFullMB: DC wavenumbers missing");
  return PSB_OK;
}

template <int TM>
int launch_derivs_tm(const full::Step& s, int nw, cudaStream_t st) {
  constexpr size_t sm = (size_t)full::kDStages * full::kDStage<TM> * sizeof(double2);
  const int n = (s.nk + TM - 1) / TM, rc = allow_smem(full::derivs_kernel<TM>, sm, sm);
  if (rc != PSB_OK) return rc;
  full::derivs_kernel<TM><<<dim3(n, nw, n), TM * 8, sm, st>>>(s);
  return PSB_OK;
}
// Blocks of 32 x 32 elements once they fill the GPU twice over, else of
// 16 x 16: 64 wires of Nk 114 have 1024 blocks of 32, one wire 16 (64 of 16).
int launch_derivs(const full::Step& s, int nw, cudaStream_t st) {
  const int n32 = (s.nk + 31) / 32;
  return (int64_t)n32 * n32 * nw >= 592 ? launch_derivs_tm<32>(s, nw, st)
                                        : launch_derivs_tm<16>(s, nw, st);
}

// mb_offd_kernel with 8 wires per CTA where the batch has them
int launch_offd(const full::MBView& v, int nk, int nw, cudaStream_t st) {
  const int W = nw >= 4 ? 8 : 1, th = 128;
  auto kern = W == 8 ? full::mb_offd_kernel<8> : full::mb_offd_kernel<1>;
  const size_t per_k = (2 + 2 * (size_t)W) * 8, sm = nk * per_k;
  const int rc = allow_smem(kern, sm, PSB_MAX_NK * per_k);
  if (rc != PSB_OK) return rc;
  const int nd = (2 * nk + 1) * nk;
  kern<<<dim3((nd + th - 1) / th, (nw + W - 1) / W), th, sm, st>>>(v, nw);
  return PSB_OK;
}

// mb_scatter_kernel for batches of up to 64 wires a CTA
template <int NT>
int launch_scatter_nt(const full::MBView& v, int nk, int nw, cudaStream_t st) {
  const size_t sm = (size_t)full::kScK * full::sc_ld(NT) * 8;
  const int rc = allow_smem(full::mb_scatter_kernel<NT>, sm, sm);
  if (rc != PSB_OK) return rc;
  full::mb_scatter_kernel<NT>
      <<<dim3(2 * nk - 1, 4, (nw + 8 * NT - 1) / (8 * NT)), 32 * full::kScWarps, sm, st>>>(v, nw);
  return PSB_OK;
}
int launch_scatter(const full::MBView& v, int nk, int nw, cudaStream_t st) {
  if (nw <= 8) return launch_scatter_nt<1>(v, nk, nw, st);
  if (nw <= 16) return launch_scatter_nt<2>(v, nk, nw, st);
  if (nw <= 32) return launch_scatter_nt<4>(v, nk, nw, st);
  return launch_scatter_nt<8>(v, nk, nw, st);
}

int full_launch(const Launch& a, cudaStream_t st) {
  const int nk = a.nk, nw = a.nw, n2 = nk * nk;
  const PsbFullMB* mb = a.mb;
  const bool deph = mb && (mb->diag_dph || mb->offdiag_dph);
  const bool relax = mb && (mb->ehs || mb->phonon);
  const bool dct = mb && mb->dctrans;
  int rc_ = check_mb(mb, deph, relax, dct);
  if (rc_ != PSB_OK) return rc_;
  full::Step s{};
  s.nk = nk;
  s.nr = a.nr;
  s.nq0 = a.nq0;
  s.V3 = a.V3;
  s.Ee = a.Ee;
  s.Eh = a.Eh;
  s.E = reinterpret_cast<const double2*>(a.fields);
  s.prm = *a.params;
  s.L1 = reinterpret_cast<double2*>(a.L1);
  s.L2 = reinterpret_cast<double2*>(a.L2);
  s.L3 = reinterpret_cast<double2*>(a.L3);
  double2* w = reinterpret_cast<double2*>(a.work);
  s.fac = reinterpret_cast<double*>(w);
  s.H = w + n2;
  s.X3 = w + 4 * n2;
  s.st_x3 = a.st_wk;
  s.st_v3 = a.st_v3;
  s.st_e = (int64_t)3 * a.nr * 16;
  s.st_lv = (int64_t)3 * n2 * 16;
  s.st_wk = a.st_wk;
  s.st_sc = (int64_t)MBScratch(nk).total;
  s.wpar = a.wpar;
  const dim3 one(1, nw);
  const double* eps = mb ? mb->eps : nullptr;
  int64_t st_eps = 0;
  if (a.tab) {
    // each wire's V3 and eps from its own densities, into its work
    const BatchWork bw(nk);
    double* v3w = reinterpret_cast<double*>(reinterpret_cast<uint8_t*>(a.work) + bw.v3);
    double* epsw = reinterpret_cast<double*>(reinterpret_cast<uint8_t*>(a.work) + bw.eps);
    s.V3 = v3w;
    s.st_v3 = a.st_wk;
    full::screen_batch_kernel<<<one, full::kScrThreads, 0, st>>>(s, a.tab, a.L, a.dens_max,
                                                                  epsw, v3w);
    eps = epsw;
    st_eps = a.st_wk;
  }
  full::MBView v{};
  if (deph || relax || dct) {
    const MBScratch L(nk);
    uint8_t* sc = reinterpret_cast<uint8_t*>(mb->scratch);
    v.nk = nk;
    v.V3 = s.V3;
    v.Ee = a.Ee;
    v.Eh = a.Eh;
    v.L = s.L3;
    v.hbar = a.params->hbar;
    v.mb = *mb;
    v.mb.eps = eps;
    v.GamE = reinterpret_cast<double*>(sc + L.gam);
    v.GamH = v.GamE + nk;
    v.De = reinterpret_cast<double*>(sc + L.de);
    v.Dh = reinterpret_cast<double*>(sc + L.dh);
    v.OffP = reinterpret_cast<double2*>(sc + L.offp);
    v.X3 = reinterpret_cast<double2*>(sc + L.x3);
    v.rates = reinterpret_cast<double*>(sc + L.rates);
    v.shift = reinterpret_cast<double2*>(sc + L.shift);
    v.tr = reinterpret_cast<double2*>(sc + L.tr);
    v.gap = a.params->gap;
    v.lf = a.params->lf;
    v.st_v3 = s.st_v3;
    v.st_lv = s.st_lv;
    v.st_sc = s.st_sc;
    v.st_eps = st_eps;
    v.wpar = a.wpar;
  }
  const int th = 128;
  const dim3 bl((n2 + th - 1) / th, nw), blk((nk + th - 1) / th, nw);
  if (relax || dct) {
    // X3 goes where the relaxation and the shift find it
    s.X3 = v.X3;
    s.st_x3 = s.st_sc;
  }
  {
    // two CTAs per SM where that leaves several diagonals in one
    constexpr size_t most = 110 * 1024;  // (one diagonal of the largest grid fits)
    int nd = full::kHDiags;
    while (nd > 1 && full::h_smem(nk, nd) > most) nd /= 2;
    const size_t sm = full::h_smem(nk, nd);
    rc_ = allow_smem(full::calch_kernel, sm, most);
    if (rc_ != PSB_OK) return rc_;
    full::calch_kernel<<<dim3((2 * nk - 1 + nd - 1) / nd, nw), 32 * nd, sm, st>>>(s);
  }
  // dephasing from the level the right-hand side reads (SBEs.py:5225-5232)
  if (mb && mb->diag_dph) {
    full::mb_gamma_kernel<<<dim3((nk + full::kGamWarps - 1) / full::kGamWarps, nw),
                            32 * full::kGamWarps, 0, st>>>(v);
    s.GamE = v.GamE;
    s.GamH = v.GamH;
  }
  if (mb && mb->offdiag_dph) {
    rc_ = launch_offd(v, nk, nw, st);
    if (rc_ != PSB_OK) return rc_;
    const int nb = (nk + full::kOT - 1) / full::kOT;
    full::mb_offp_kernel<<<dim3(nb * nb, nw), 256, 0, st>>>(v);
    s.OffP = v.OffP;
  }
  rc_ = launch_derivs(s, nw, st);
  if (rc_ != PSB_OK) return rc_;
  if (relax || dct) {
    // X3's occupations relaxed (SBEs.py:5688-5695) and shifted by the DC field
    // (SBEs.py:5698-5702), then the rescale
    if (relax) {
      if (mb->ehs) {
        full::mb_occ_kernel<<<blk, th, 0, st>>>(v);
        rc_ = launch_scatter(v, nk, nw, st);
        if (rc_ != PSB_OK) return rc_;
      }
      full::mb_rates_kernel<<<dim3(nk, nw), full::kRateThreads, 0, st>>>(v);
      full::mb_relax_kernel<<<blk, th, 0, st>>>(v, a.params->dt);
    }
    if (dct) {
      full::mb_shift_kernel<<<one, full::kShThreads, (size_t)2 * nk * 16, st>>>(v);
      if (a.params->lf) {
        const int nb = (nk + full::kSB - 1) / full::kSB;
        const dim3 bt(3 * nb * nb, nw);
        full::mb_shift_mat_kernel<true><<<bt, full::kSThreads, 0, st>>>(v);
        full::mb_shift_mat_kernel<false><<<bt, full::kSThreads, 0, st>>>(v);
      } else {
        const dim3 bd((3 * nk + th - 1) / th, nw);
        full::mb_shift_diag_kernel<<<bd, th, 0, st>>>(v);
        full::mb_shift_diag_store_kernel<<<bd, th, 0, st>>>(v);
      }
    }
  }
  full::occ_sums_kernel<<<one, full::kLfThreads, 0, st>>>(s);
  const dim3 b3((3 * n2 + full::kLfThreads - 1) / full::kLfThreads, nw);
  full::leapfrog_kernel<<<b3, full::kLfThreads, 0, st>>>(s);
  return PSB_OK;
}
}  // namespace

extern "C" int psb_full_step_mb_f64(int nk, int nr, int nq0, const double* d_V3,
                                    const double* d_Ee, const double* d_Eh,
                                    const double* d_fields, const PsbFullParams* params,
                                    const PsbFullMB* mb, double* d_L1, double* d_L2,
                                    double* d_L3, void* d_work, int64_t n_work_bytes,
                                    void* stream) {
  if (!d_V3 || !d_Ee || !d_Eh || !d_fields || !params || !d_L1 || !d_L2 || !d_L3 || !d_work)
    return set_error(PSB_ERR_INVALID, "psb_full_step_f64: null pointer");
  if (nk < 2 || nk > PSB_MAX_NK || nr < 1 || nq0 < 0 || nq0 >= nr)
    return set_error(PSB_ERR_SIZE, "psb_full_step_f64: nk %d / nr %d / nq0 %d out of range", nk,
                     nr, nq0);
  if (n_work_bytes < psb_full_work_bytes(nk))
    return set_error(PSB_ERR_SIZE, "psb_full_step_f64: work needs psb_full_work_bytes(nk)");
  if (!(params->hbar > 0.0)) return set_error(PSB_ERR_INVALID, "hbar must be > 0");
  Launch a{};
  a.nw = 1;
  a.nk = nk;
  a.nr = nr;
  a.nq0 = nq0;
  a.V3 = d_V3;
  a.Ee = d_Ee;
  a.Eh = d_Eh;
  a.fields = d_fields;
  a.params = params;
  a.mb = mb;
  a.L1 = d_L1;
  a.L2 = d_L2;
  a.L3 = d_L3;
  a.work = d_work;
  const int rc = full_launch(a, (cudaStream_t)stream);
  if (rc != PSB_OK) return rc;
  return check_cuda("psb_full_step_f64");
}

extern "C" int psb_full_step_f64(int nk, int nr, int nq0, const double* d_V3, const double* d_Ee,
                                 const double* d_Eh, const double* d_fields,
                                 const PsbFullParams* params, double* d_L1, double* d_L2,
                                 double* d_L3, void* d_work, int64_t n_work_bytes,
                                 void* stream) {
  return psb_full_step_mb_f64(nk, nr, nq0, d_V3, d_Ee, d_Eh, d_fields, params, nullptr, d_L1,
                              d_L2, d_L3, d_work, n_work_bytes, stream);
}

extern "C" int64_t psb_full_batch_work_bytes(int nw, int nk) {
  if (nk < 2 || nk > PSB_MAX_NK) return set_error(PSB_ERR_SIZE, "nk %d out of range", nk);
  if (nw < 1 || nw > PSB_FULL_MAX_WIRES) return set_error(PSB_ERR_SIZE, "nw %d out of range", nw);
  return (int64_t)nw * (int64_t)BatchWork(nk).total;
}

extern "C" int psb_full_step_batch_f64(int nw, int nk, int nr, int nq0, const double* d_tab,
                                       double L, double dens_max, int screened,
                                       const double* d_fields, const PsbFullParams* params,
                                       const double* d_wpar, const PsbFullMB* mb, double* d_L1,
                                       double* d_L2, double* d_L3, void* d_work,
                                       int64_t n_work_bytes, void* stream) {
  if (!d_tab || !d_fields || !params || !d_wpar || !d_L1 || !d_L2 || !d_L3 || !d_work)
    return set_error(PSB_ERR_INVALID, "psb_full_step_batch_f64: null pointer");
  if (nk < 2 || nk > PSB_MAX_NK || nr < 1 || nq0 < 0 || nq0 >= nr || nw < 1 ||
      nw > PSB_FULL_MAX_WIRES)
    return set_error(PSB_ERR_SIZE, "psb_full_step_batch_f64: nw %d / nk %d / nr %d / nq0 %d", nw,
                     nk, nr, nq0);
  if (n_work_bytes < psb_full_batch_work_bytes(nw, nk))
    return set_error(PSB_ERR_SIZE, "psb_full_step_batch_f64: work needs "
                                   "psb_full_batch_work_bytes(nw, nk)");
  if (!(params->hbar > 0.0)) return set_error(PSB_ERR_INVALID, "hbar must be > 0");
  if (screened && !(L > 0.0)) return set_error(PSB_ERR_INVALID, "screening needs L > 0");
  Launch a{};
  a.nw = nw;
  a.nk = nk;
  a.nr = nr;
  a.nq0 = nq0;
  a.V3 = d_tab;  // V_eh, V_ee, V_hh rows of the table block, shared when unscreened
  a.Ee = d_tab + 3 * (size_t)nk;
  a.Eh = d_tab + 4 * (size_t)nk;
  a.fields = d_fields;
  a.params = params;
  a.wpar = d_wpar;
  a.mb = mb;
  a.L1 = d_L1;
  a.L2 = d_L2;
  a.L3 = d_L3;
  a.work = d_work;
  a.st_wk = (int64_t)BatchWork(nk).total;
  if (screened) {
    a.tab = d_tab;
    a.L = L;
    a.dens_max = dens_max;
  }
  const int rc = full_launch(a, (cudaStream_t)stream);
  if (rc != PSB_OK) return rc;
  return check_cuda("psb_full_step_batch_f64");
}

namespace {
// both source kernels for nw wires; CTAs of the polarisation until the GPU has
// about one each
int launch_sources(int nw, int nk, int nr, const double* kr, const double* r,
                   const double* window, double L, double dcv, double yw, double sgnw,
                   const double* wpar, const double* lev, double* out, cudaStream_t st) {
  // 8 positions per CTA of the densities once that leaves two CTAs per SM
  const bool wide = (int64_t)(nr + 7) / 8 * nw >= 296;
  const int R = wide ? 8 : 4;
  auto dens = wide ? full::densities_kernel<8> : full::densities_kernel<4>;
  const size_t sp = (size_t)2 * (2 * nk - 1) * 16, sd = (size_t)R * nk * 16;
  int rc = allow_smem(full::polarisation_kernel, sp, (size_t)2 * (2 * PSB_MAX_NK - 1) * 16);
  if (rc == PSB_OK) rc = allow_smem(dens, sd, (size_t)R * PSB_MAX_NK * 16);
  if (rc != PSB_OK) return rc;
  const double2* lv = reinterpret_cast<const double2*>(lev);
  double2* o = reinterpret_cast<double2*>(out);
  const int nb = nw >= 148 ? 1 : (148 / nw < 16 ? 148 / nw : 16);
  dens<<<dim3((nr + R - 1) / R, nw), full::kSrcThreads, sd, st>>>(nk, nr, kr, r, window, L, dcv, yw,
                                                                 sgnw, wpar, lv, o);
  full::polarisation_kernel<<<dim3(nb, nw), full::kPolThreads, sp, st>>>(
      nk, nr, kr, r, window, dcv, yw, sgnw, wpar, lv, o);
  return check_cuda("sources kernels");
}
}  // namespace

extern "C" int psb_full_sources_f64(int nk, int nr, const double* d_kr, const double* d_r,
                                    const double* d_window, double L, double dcv, double yw,
                                    double sgnw, const double* d_level, double* d_out,
                                    void* stream) {
  if (!d_kr || !d_r || !d_window || !d_level || !d_out)
    return set_error(PSB_ERR_INVALID, "psb_full_sources_f64: null pointer");
  if (nk < 2 || nk > PSB_MAX_NK || nr < 1)
    return set_error(PSB_ERR_SIZE, "psb_full_sources_f64: nk %d / nr %d out of range", nk, nr);
  return launch_sources(1, nk, nr, d_kr, d_r, d_window, L, dcv, yw, sgnw, nullptr, d_level, d_out,
                        (cudaStream_t)stream);
}

extern "C" int psb_full_sources_batch_f64(int nw, int nk, int nr, const double* d_kr,
                                          const double* d_r, const double* d_window, double L,
                                          double dcv, const double* d_wpar,
                                          const double* d_levels, double* d_out, void* stream) {
  if (!d_kr || !d_r || !d_window || !d_wpar || !d_levels || !d_out)
    return set_error(PSB_ERR_INVALID, "psb_full_sources_batch_f64: null pointer");
  if (nk < 2 || nk > PSB_MAX_NK || nr < 1 || nw < 1 || nw > PSB_FULL_MAX_WIRES)
    return set_error(PSB_ERR_SIZE, "psb_full_sources_batch_f64: nw %d / nk %d / nr %d", nw, nk,
                     nr);
  return launch_sources(nw, nk, nr, d_kr, d_r, d_window, L, dcv, 0.0, 0.0, d_wpar, d_levels,
                        d_out, (cudaStream_t)stream);
}
