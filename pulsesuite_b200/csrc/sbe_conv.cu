// sbe_conv.cu -- the FP64 SBE step (right-hand side, RK4, leapfrog) of one
// quantum wire per CTA, with the exchange sums by fast convolution, sm_100a.
//
// The exchange sums of a right-hand side (pulsesuite/PSTD3D/SBEs.py:896-921)
// are three Toeplitz products with the real, even tables V(|k - k'|):
//   Omega_k += sum_k' Veh p_k'   Se_k -= sum Vee ne   Sh_k -= sum Vhh nh
// i.e. 8 Nk FP64 flops per point when summed directly.  As cyclic
// convolutions of length M >= 2 Nk of the complex signals p and ne + i nh
// (zero beyond Nk) they take one forward and one inverse transform each, four
// of 5 M log2 M flops: 40 log2 M per point at M = 2 Nk.  A real, even table has
// a real spectrum, so with one shared table both signals are multiplied by the
// same real numbers; with distinct Vee and Vhh the second signal's product
// is Z (Vee + Vhh)/2 + conj(Z(-f)) (Vee - Vhh)/2.
//
// Rounding.  All in FP64, as the direct sums, but the error is relative to the
// largest sum of a signal, about 2^-53 3 log2 M (4e-15) of it at most, not to
// each sum: sums far from the carriers that are small beside it have fewer
// digits.  The two parts of a complex signal share it too, n_h's sums that of
// n_e's; a step adds these up, and CalcH, which returns them, brings the parts
// to one size first.  Whole passes are as close to 64-bit references as with
// direct sums (1e-16 to 1e-15 of the largest value).
//
// Transform.  M = 16 q, q = 8 L with L = 1, 2, 4, 8, 16 lanes (Nk <= 64 L);
// T = 32 L threads with 8 complex points each:
//   A   thread (signal, half, a): the 8 points x[a + q r] (the upper 8 of 16
//       are zero padding and cost nothing); a 16-point transform over r
//       splits into two of 8 points, the even outputs and (after the roots
//       of 16) the odd ones; times exp(-2 pi i a g / M), into row g column a;
//   B   row (signal, g), q points over L lanes of one warp: 8 points per
//       lane, the roots of q, then L points (between the two lanes by
//       shuffles for L = 2, by a transposition inside the row above), times the
//       spectrum, and back;
//   A'  the inverse of A, of whose 16 outputs the 8 wanted ones are formed.
// So a stage takes four CTA barriers.  The row stride keeps the column and
// the row accesses of 16-byte elements free of bank conflicts.  8 points per
// thread and not 16: with 16 (half the threads, fewer shared-memory passes)
// the state and a transform did not fit 168 registers, and a lone wire's stage
// took 1.5 to 2 times as long.  Lengths between the powers of two (rows of 5,
// 6, 7 points per lane) gained at most 10 % at Nk <= 192 and nothing above:
// the same instructions with fewer active lanes.
//
// The elementwise right-hand side, RK4 combination and sums follow in the
// same kernel; each thread keeps the base state and the RK accumulator of
// its (at most 2) points in registers for the whole call.  A wire's
// arithmetic depends on its own Nk only (a launch takes the wires of its own
// L), so its result never depends on the other wires of a launch.
//
// What bounds it: shared-memory traffic, about 460 wavefronts per warp and
// stage (86 % of the pipe at Nk 512), with the FP64 pipe at 54 % beside it; a
// lone wire is bound by the latency of its stages.  Measured
// on B200 against the direct sums it replaces (us per wire-stage and SM, 3552
// wires; in brackets us per stage of one wire):
//   Nk     direct       screened       transforms    screened
//   64     1.42 (2.07)  2.01 (3.31)    0.20 (1.45)   0.39 (3.11)
//   128    1.97 (2.68)  2.83 (4.24)    0.50 (1.71)   0.88 (3.46)
//   256    4.49 (5.45)  5.65 (7.59)    1.08 (2.05)   1.76 (4.03)
//   512    14.9 (16.2)  16.9 (21.3)    2.37 (3.12)   3.91 (6.79)
//   1024   60.0 (59.9)  58.8 (58.4)    6.21 (6.01)   10.1 (9.89)
#include <math.h>

#include "fft64.cuh"
#include "sbe_f64.cuh"

namespace psb {
namespace conv {

using fft::Dft;
using fft::mulw;

constexpr int kEpt = 2;    // points of k per thread
constexpr int kDrive = 8;  // steps whose drive is evaluated at once

// Lanes of a row.
__host__ __device__ constexpr int lanes_of(int nk) {
  return nk <= 64 ? 1 : (nk <= 128 ? 2 : (nk <= 256 ? 4 : (nk <= 512 ? 8 : 16)));
}
// Row stride (16-byte elements): the residue modulo 8 that spreads the 8 / L
// rows of a quarter warp over the banks, and from L = 4 room for the
// transposed row, whose element (l, f) lies at l + (L + 1) f.
__host__ __device__ constexpr int stride_of(int L) {
  return L == 1 ? 9 : (L == 2 ? 18 : (L == 4 ? 44 : 8 * L + 7));
}

// What a wire's steps need besides its points (shared memory).
struct Par {
  double gamma, gap, pscale, half_l, dens_max, hm;  // 1 / (2 L), mscale / hbar
  double pulse[2][4];  // t0, 1 / fwhm, -mscale amp (cos, sin)(phase) / hbar
  double2 drive[kDrive + 1][2];  // M / hbar at t + h/2, t + h of kDrive steps; M(t)
  int64_t p_off;
  double red[2][4][16];  // partial sums [parity][value][warp]
};

// Shared memory of one wire (bytes) with NT tables.
template <int L>
struct Lay {
  static constexpr int q = 8 * L, np = 8 * q, rs = stride_of(L), T = 32 * L;
  // pass B's second transform, of L points: over H lanes by shuffles, D = L /
  // H points in each; lane l holds f = l % D + D it and the frequencies
  // g + 16 (f + 8 (H i + b)), b the lane's place among the H, whose spectra
  // lie at (it D + i) 16 L + g L + l
  static constexpr int H = L == 16 || L == 2 ? 2 : 1, D = L / H, nf = 8 / D;
  static constexpr int LS = L >= 4 ? L + 1 : L;  // stride of f in the transposed row
  static constexpr int sl = 16 * q;
  static constexpr uint32_t yp = 32u * rs * 16u;   // after E, [32 rows][rs] complex: p,
  static constexpr uint32_t yn = yp + np * 16u;    // ne + i nh of the stage point
  static constexpr uint32_t twa = yn + np * 16u;   // exp(-2 pi i a 2^s / M), [4][q]
  static constexpr uint32_t twb = twa + 4u * q * 16u;  // exp(-2 pi i l 2^s / q), [3][L]
  static constexpr uint32_t par = twb + 3u * L * 16u;
  static constexpr uint32_t s = par + (uint32_t)sizeof(Par);  // spectra [NT][sl]
  // The tables on their way to S: one table fits the rows of the second
  // signal, which its transform leaves free; three follow the spectra.
  static constexpr uint32_t vq1 = 16u * rs * 16u, vq3 = s + 3u * sl * 8u;
  static constexpr uint32_t total1 = s + sl * 8u, total3 = vq3 + 3u * np * 8u;
};

// Barrier over the CTA.
template <int L>
__device__ __forceinline__ void cta_sync() {
  if constexpr (L == 1)
    __syncwarp();
  else
    __syncthreads();
}

// The roots exp(-2 pi i a (2 f + half) / M), f = 4 b + c, as t[c] (v: b = 1).
template <int q>
__device__ __forceinline__ void roots_a(const double2* tw, bool half, double2 (&t)[4],
                                        double2& v) {
  const double2 u1 = tw[q];
  t[0] = half ? tw[0] : make_double2(1.0, 0.0);
  t[1] = mulw<-1>(t[0], u1);
  const double2 u2 = tw[2 * q];
  t[2] = mulw<-1>(t[0], u2);
  t[3] = mulw<-1>(t[1], u2);
  v = tw[3 * q];
}

// Pass A on the 8 points in x: output f to o[2 f rs] (row 2 f + half of the
// signal, column a); tw points at column a of the roots.
template <int q, int rs>
__device__ __forceinline__ void pass_a(double2 (&x)[8], double2* o, const double2* tw,
                                       bool half) {
  if (half)
    fft::unroll<8>([&](auto R) {
      constexpr int r = decltype(R)::value;
      x[r] = fft::rot16<r, -1>(x[r]);
    });
  Dft<8, -1>::run(x);
  double2 t[4], v;
  roots_a<q>(tw, half, t, v);
#pragma unroll
  for (int f = 0; f < 8; ++f) {
    double2 z = x[f];
    if (f >= 4) z = mulw<-1>(z, v);
    o[2 * f * rs] = mulw<-1>(z, t[f & 3]);
  }
}

// Pass A': this half's share of the 8 points a + q r, into its own slots.
template <int q, int rs>
__device__ __forceinline__ void pass_a_inv(double2* o, const double2* tw, bool half) {
  double2 x[8], t[4], v;
  roots_a<q>(tw, half, t, v);
#pragma unroll
  for (int f = 0; f < 8; ++f) {
    double2 z = mulw<1>(o[2 * f * rs], t[f & 3]);
    if (f >= 4) z = mulw<1>(z, v);
    x[f] = z;
  }
  Dft<8, 1>::run(x);
  if (half)
    fft::unroll<8>([&](auto R) {
      constexpr int r = decltype(R)::value;
      x[r] = fft::rot16<r, 1>(x[r]);
    });
#pragma unroll
  for (int r = 0; r < 8; ++r) o[2 * r * rs] = x[r];
}

// x[f] times the roots exp(SG 2 pi i l f / q) of lane l.
template <int L, int SG>
__device__ __forceinline__ void roots_b(double2 (&x)[8], const double2* twb) {
  const double2 w1 = twb[0], w2 = twb[L], w4 = twb[2 * L];
  x[1] = mulw<SG>(x[1], w1);
  x[2] = mulw<SG>(x[2], w2);
  x[4] = mulw<SG>(x[4], w4);
  x[5] = mulw<SG>(x[5], mulw<-1>(w1, w4));
  x[6] = mulw<SG>(x[6], mulw<-1>(w2, w4));
  const double2 w3 = mulw<-1>(w1, w2);
  x[3] = mulw<SG>(x[3], w3);
  x[7] = mulw<SG>(x[7], mulw<-1>(w3, w4));
}

// What pass B does with a row.
enum RowOp {
  kTables = 0,    // forward only, of the even tables: Veh in signal 0 (its
                  // spectrum, the real part, into S[0]) and Vee + i Vhh in
                  // signal 1 (half sum and half difference into S[1], S[2])
  kOneTable = 1,  // times S[0], and back
  kDistinct = 2   // p times S[0]; ne + i nh with S[1], S[2], and back
};

template <int L>
__device__ __forceinline__ void pass_b(RowOp op, bool one, double2* E, double* S,
                                       const double2* twb, double scale) {
  using Y = Lay<L>;
  constexpr int H = Y::H, D = Y::D, NF = Y::nf, SL = Y::sl, LS = Y::LS;
  const int row = (int)threadIdx.x / L, l = (int)threadIdx.x % L, g = row & 15;
  const int f0 = l % D, b = l / D;
  double2* R = E + row * Y::rs;
  double2 z[NF][D];
  // a radix-2 step between lanes `mask` apart: sums below, differences above
  auto step = [&](double2& v, int mask) {
    const double sg = (l & mask) ? -1.0 : 1.0;
    const double ox = __shfl_xor_sync(0xffffffffu, v.x, mask);
    const double oy = __shfl_xor_sync(0xffffffffu, v.y, mask);
    v = make_double2(fma(sg, v.x, ox), fma(sg, v.y, oy));
  };
  {
    double2 x[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) x[r] = R[l + L * r];
    Dft<8, -1>::run(x);
    if constexpr (L > 1) roots_b<L, -1>(x, twb + l);
    if constexpr (D == 1) {
#pragma unroll
      for (int f = 0; f < 8; ++f) {
        if constexpr (L == 2) step(x[f], 1);
        z[f][0] = x[f];
      }
    } else {
      __syncwarp();
#pragma unroll
      for (int f = 0; f < 8; ++f) R[l + LS * f] = x[f];
      __syncwarp();
#pragma unroll
      for (int it = 0; it < NF; ++it) {
#pragma unroll
        for (int i = 0; i < D; ++i) z[it][i] = R[i + D * b + LS * (f0 + D * it)];
        if constexpr (H == 2) {
#pragma unroll
          for (int i = 0; i < D; ++i) step(z[it][i], 8);
          if (b)
            fft::unroll<D>([&](auto I) {
              constexpr int i = decltype(I)::value;
              z[it][i] = fft::rot16<i, -1>(z[it][i]);
            });
        }
        Dft<D, -1>::run(z[it]);
      }
    }
  }
  double* Sg = S + g * L + l;
  if (op == kTables) {
    if (row >= 16 && one) return;
    double* d = Sg + (row < 16 ? 0 : SL);
#pragma unroll
    for (int it = 0; it < NF; ++it)
#pragma unroll
      for (int i = 0; i < D; ++i) {
        const double2 c = z[it][i];
        const int o = (it * D + i) * 16 * L;
        d[o] = row < 16 ? c.x * scale : 0.5 * scale * (c.x + c.y);
        if (row >= 16) d[SL + o] = 0.5 * scale * (c.x - c.y);
      }
    return;
  }
  if (op == kOneTable || row < 16) {
#pragma unroll
    for (int it = 0; it < NF; ++it)
#pragma unroll
      for (int i = 0; i < D; ++i) {
        const double v = Sg[(it * D + i) * 16 * L];
        z[it][i].x *= v;
        z[it][i].y *= v;
      }
  }
  if (op == kDistinct) {
    // the second signal's product needs its mirrored frequency, which
    // another row holds; it travels through E
    __syncwarp();
    if (row >= 16) {
#pragma unroll
      for (int it = 0; it < NF; ++it)
#pragma unroll
        for (int i = 0; i < D; ++i) R[H * i + b + LS * (f0 + D * it)] = z[it][i];
    }
    cta_sync<L>();
    if (row >= 16) {
      // frequency g + 16 j, j = f + 8 k; its mirror is row -g, index
      // q - 1 - j (row 0: q - j, modulo q)
      const double2* M = E + (16 + ((16 - g) & 15)) * Y::rs;
#pragma unroll
      for (int it = 0; it < NF; ++it) {
        const int f = f0 + D * it;
        const int fm = g != 0 ? 7 - f : (f > 0 ? 8 - f : 0);
#pragma unroll
        for (int i = 0; i < D; ++i) {
          const int k = H * i + b, im = g == 0 && f == 0 ? (L - k) % L : L - 1 - k;
          const double2 m = M[im + LS * fm];
          const double sp = Sg[SL + (it * D + i) * 16 * L];
          const double sm = Sg[2 * SL + (it * D + i) * 16 * L];
          z[it][i] = make_double2(fma(m.x, sm, z[it][i].x * sp), fma(-m.y, sm, z[it][i].y * sp));
        }
      }
    }
    cta_sync<L>();
  }
  double2 x[8];
  if constexpr (D == 1) {
#pragma unroll
    for (int f = 0; f < 8; ++f) {
      x[f] = z[f][0];
      if constexpr (L == 2) step(x[f], 1);
    }
  } else {
#pragma unroll
    for (int it = 0; it < NF; ++it) {
      Dft<D, 1>::run(z[it]);
      if constexpr (H == 2) {
        if (b)
          fft::unroll<D>([&](auto I) {
            constexpr int i = decltype(I)::value;
            z[it][i] = fft::rot16<i, 1>(z[it][i]);
          });
#pragma unroll
        for (int i = 0; i < D; ++i) step(z[it][i], 8);
      }
#pragma unroll
      for (int i = 0; i < D; ++i) R[i + D * b + LS * (f0 + D * it)] = z[it][i];
    }
    __syncwarp();
#pragma unroll
    for (int f = 0; f < 8; ++f) x[f] = R[l + LS * f];
    __syncwarp();
  }
  if constexpr (L > 1) roots_b<L, 1>(x, twb + l);
  Dft<8, 1>::run(x);
#pragma unroll
  for (int r = 0; r < 8; ++r) R[l + L * r] = x[r];
}

// log |a / b| with one division: with x = |a| 2^-e, y = |b|, x / y in
// [0.7, 1.42], it is e log 2 + 2 atanh((x - y) / (x + y)), the inverse
// hyperbolic tangent by its Taylor series (|argument| < 0.172: the terms left
// out are below 3e-17 of it).  far: a or b is zero, not finite or near the
// ends of the range, and the result is not it.
__device__ __forceinline__ double log_ratio(double a, double b, bool& far) {
  double x = fabs(a);
  const double y = fabs(b);
  far |= !(x > 1e-290 && y > 1e-290 && x < 1e290 && y < 1e290);
  int e = (__double2hiint(x) >> 20) - (__double2hiint(y) >> 20);
  x = __hiloint2double(__double2hiint(x) - e * (1 << 20), __double2loint(x));  // x / y in (1/2, 2)
  const int up = x > 1.41 * y ? 1 : (x < 0.705 * y ? -1 : 0);
  x = __hiloint2double(__double2hiint(x) - up * (1 << 20), __double2loint(x));
  e += up;
  const double s = (x - y) / (x + y), s2 = s * s;
  double p = 1.0 / 19.0;
#pragma unroll
  for (int k = 8; k >= 1; --k) p = fma(p, s2, 1.0 / (2 * k + 1));
  return fma((double)e, 0.69314718055994530942, fma(2.0 * s * s2, p, 2.0 * s));
}

// CTAs per SM the registers are limited for: 16 warps of 128 registers, the
// best of 16, 20 and 24 for L = 1, 2, 16; 20 of 96 for L = 4 (Nk 256: 1.08
// against 1.15 us per wire-stage and SM); 24 of 80 for L = 8, as fast as 16 on
// full waves and with a third more wires in flight on short ones.
__host__ __device__ constexpr int ctas_of(int L) {
  return L == 16 ? 1 : (L == 4 ? 5 : (L == 8 ? 3 : 16 / L));
}

// Sums over the CTA in a fixed order: a warp's K = 2 or 4 sums at once (each
// step of the butterfly halves the values a lane carries, so K values take K + 2
// or so shuffles of a double, not 5 K) into red[v][warp].
template <int K>
__device__ __forceinline__ void put_sums(double (&v)[K], double (*red)[16], int lane, int warp) {
  int o = 16;
#pragma unroll
  for (int c = K / 2; c >= 1; c /= 2, o /= 2) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < c; ++i) {
      const double send = up ? v[i] : v[i + c], keep = up ? v[i + c] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  for (; o >= 1; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  // lane bits from 16 down chose the value
  constexpr int S = 32 / K;
  if (lane % S == 0) red[lane / S][warp] = v[0];
}
template <int L>
__device__ __forceinline__ double get_sum(const double (*red)[16], int v) {
  double t = red[v][0];
#pragma unroll
  for (int i = 1; i < L; ++i) t += red[v][i];
  return t;
}

// All steps of one wire whose descriptor and table have been checked.  ONCE:
// one right-hand side or CalcH (mode), else RK4 or leapfrog steps (MODE).
template <int L, int MODE>
__device__ __forceinline__ void wire_steps(const Batch& bt, int mode, bool scr, uint8_t* smem,
                                           int wi, const PsbTable& tb) {
  using Y = Lay<L>;
  constexpr int q = Y::q, np = Y::np, rs = Y::rs, T = Y::T;
  constexpr bool ONCE = MODE == kRhs;
  PsbWire* wp = bt.wires + wi;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nk = tb.nk;
  const int64_t off = wp->off;
  const bool one = (tb.flags & PSB_TAB_SHARED_V) != 0;  // one table for all columns
  const bool exc = (tb.flags & PSB_TAB_EXCITONS) != 0;
  scr = scr && exc && (tb.flags & PSB_TAB_SCREENED) != 0;
  double2* E = reinterpret_cast<double2*>(smem);
  double2* yp = reinterpret_cast<double2*>(smem + Y::yp);
  double2* yn = reinterpret_cast<double2*>(smem + Y::yn);
  double2* twa = reinterpret_cast<double2*>(smem + Y::twa);
  double2* twb = reinterpret_cast<double2*>(smem + Y::twb);
  double* S = reinterpret_cast<double*>(smem + Y::s);
  Par& par = *reinterpret_cast<Par*>(smem + Y::par);
  const double* blk = bt.tabdata + tb.off;

  // ---- roots, parameters, state ----------------------------------------------
  if (exc) {
    for (int i = tid; i < 4 * q; i += T) {
      double sn, cs;
      sincospi(2.0 / (16 * q) * (double)((i % q) << (i / q)), &sn, &cs);
      twa[i] = make_double2(cs, -sn);
    }
    for (int i = tid; i < 3 * L; i += T) {
      double sn, cs;
      sincospi(2.0 / q * (double)((i % L) << (i / L)), &sn, &cs);
      twb[i] = make_double2(cs, -sn);
    }
  }
  const double ih = 1.0 / bt.hbar;
  if (tid < 2) {
    // the drive is a sum of Gaussian pulses (SBEs drive, E(t))
    double* pc = par.pulse[tid];
    pc[0] = pc[1] = pc[2] = pc[3] = 0.0;
    if (tid < wp->npulse && MODE != kLeapfrog) {
      double sn, cs;
      sincos(wp->phase[tid], &sn, &cs);
      const double am = -wp->mscale * wp->amp[tid] * ih;
      pc[0] = wp->t0[tid];
      pc[1] = 1.0 / wp->fwhm[tid];
      pc[2] = am * cs;
      pc[3] = am * sn;
    }
    if (tid == 0) {
      par.gamma = wp->gamma;
      par.gap = wp->gap;
      par.pscale = wp->pscale;
      par.half_l = 1.0 / (2.0 * tb.L);
      par.dens_max = tb.dens_max;
      par.hm = wp->mscale * ih;
      par.p_off = wp->p_off;
    }
  }
  // pass A: signal (p, ne + i nh), half, column
  const int grp = tid / (8 * L), col = tid - grp * 8 * L, sig = grp >> 1;
  const bool half = (grp & 1) != 0;
  double2* ea = E + (16 * sig + half) * rs + col;  // rows 2 f further
  double yb[kEpt][4];   // base state / leapfrog X1
  double acc[kEpt][3];  // RK accumulator of p and of n (dn_e/dt = dn_h/dt)
  double ekh[kEpt];     // (Ee + Eh + gap) / hbar
  double nsum = 0.0;    // sum of n_e + n_h over this thread's points
  {
    const double2* y2 = reinterpret_cast<const double2*>(bt.y + 4 * off);
    const double2* y1 = reinterpret_cast<const double2*>(bt.y1 + 4 * off);
    const double gap = wp->gap;
#pragma unroll
    for (int e = 0; e < kEpt; ++e) {
      const int k = tid + e * T;
      double2 a = make_double2(0.0, 0.0), b = a;
      ekh[e] = 0.0;
      if (k < nk) {
        a = y2[2 * k];
        b = y2[2 * k + 1];
        ekh[e] = (blk[3 * nk + k] + gap + blk[4 * nk + k]) * ih;
        nsum += b.x + b.y;
      }
      yp[k] = a;
      yn[k] = b;
      if (MODE == kLeapfrog && k < nk) {
        a = y1[2 * k];
        b = y1[2 * k + 1];
      }
      yb[e][0] = a.x;
      yb[e][1] = a.y;
      yb[e][2] = b.x;
      yb[e][3] = b.y;
      acc[e][0] = acc[e][1] = acc[e][2] = 0.0;
    }
  }
  const double h = bt.dt, h2 = h / 2.0, h6 = h / 6.0;
  double t = wp->t;
  const int steps0 = wp->steps, nst = ONCE ? 1 : bt.nsteps;
  // warp 0: the drive of steps s .. s + kDrive - 1, whose first begins at t
  // (t advances by repeated addition, as the steps' t does); lane bits: pulse,
  // t + h/2 or t + h, step.  M(t) of step s, the last value before, moves to
  // the end of the table.
  auto drive_ahead = [&](double t0) {
    const int j = lane >> 2;
    for (int i = 0; i < kDrive - 1; ++i)
      if (i < j) t0 = t0 + h;
    const double* pc = par.pulse[lane & 1];
    const double u = ((lane & 2 ? t0 + h : t0 + h2) - pc[0]) * pc[1];
    const double env = exp(-4.0 * 0.69314718055994530942 * u * u);
    double vr = pc[2] * env, vi = pc[3] * env;
    vr += __shfl_xor_sync(0xffffffffu, vr, 1);
    vi += __shfl_xor_sync(0xffffffffu, vi, 1);
    if (lane == 0) par.drive[kDrive][0] = par.drive[kDrive - 1][1];
    __syncwarp();
    if ((lane & 1) == 0) par.drive[j][(lane >> 1) & 1] = make_double2(vr, vi);
  };
  __syncwarp();
  if (MODE != kLeapfrog && warp == 0) {
    // M(t) of the first step
    if (lane == 0) {
      double2 m = make_double2(0.0, 0.0);
      for (int j = 0; j < 2; ++j) {
        const double* pc = par.pulse[j];
        const double u = (t - pc[0]) * pc[1];
        const double env = exp(-4.0 * 0.69314718055994530942 * u * u);
        m.x += pc[2] * env;
        m.y += pc[3] * env;
      }
      par.drive[kDrive - 1][1] = m;
    }
    __syncwarp();
  }
  double ntot = 0.0;  // sum of n_e + n_h of the stage point, for its screening
  int par_red = 0;    // parity of the partial sums: read one barrier after they are put
  if (scr) {
    double v[2] = {nsum, 0.0};
    put_sums<2>(v, par.red[0], lane, warp);
  }
  // CalcH returns the two sums of a signal (of Re p and Im p, of n_e and n_h) as
  // numbers of their own: the second is brought to the size of the first by a
  // power of two on its way through the transforms, whose rounding error is that
  // of the larger one, and the sum of a column of zeros is zero.
  const bool apart = ONCE && exc && mode == kCalcH;
  int up[2] = {0, 0};         // of Im p, of n_h
  bool some[4] = {1, 1, 1, 1};  // the column is not all zeros
  if (apart) {
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      double top = 0.0;
#pragma unroll
      for (int e = 0; e < kEpt; ++e) {
        const double x = fabs(yb[e][v]);
        top = fmax(top, isfinite(x) ? x : HUGE_VAL);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
      if (lane == 0) par.red[1][v][warp] = top;
    }
  }
  cta_sync<L>();
  if (apart) {
    double top[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      top[v] = par.red[1][v][0];
      for (int i = 1; i < L; ++i) top[v] = fmax(top[v], par.red[1][v][i]);
      some[v] = top[v] > 0.0;
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
      if (some[2 * c] && some[2 * c + 1] && isfinite(top[2 * c]) && isfinite(top[2 * c + 1]))
        up[c] = ilogb(top[2 * c]) - ilogb(top[2 * c + 1]);
#pragma unroll
    for (int e = 0; e < kEpt; ++e) {
      const int k = tid + e * T;
      yp[k].y = ldexp(yb[e][1], up[0]);
      yn[k].y = ldexp(yb[e][3], up[1]);
    }
    // (read by others after the barrier behind the tables)
  }

  for (int s = 0; s < nst; ++s) {
    double2 m_lf = make_double2(0.0, 0.0);
    if (MODE == kLeapfrog) {
      const int64_t fi = (int64_t)wi * bt.field_stride + 2 * ((int64_t)steps0 + s);
      if (bt.field && fi >= 0 && fi + 1 < bt.n_field)
        m_lf = make_double2(-par.hm * bt.field[fi], -par.hm * bt.field[fi + 1]);
    } else if (s % kDrive == 0) {
      // read by all after the next barrier
      if (warp == 0) drive_ahead(t);
      if (!exc) cta_sync<L>();
    }
    for (int st = 0; st < (MODE == kRk4 ? 4 : 1); ++st) {
      if (exc) {
        // the stage's tables: once per call, or screened by the stage point
        // (coulomb.py:1218-1230) every time
        const bool build = scr || (s == 0 && st == 0);
        double* vq = reinterpret_cast<double*>(smem + (one ? Y::vq1 : Y::vq3));
        if (build) {
          double n1d = 0.0;
          if (scr) {
            if (MODE != kLeapfrog || s == 0) ntot = get_sum<L>(par.red[par_red], 0);
            n1d = ntot * par.half_l;
            n1d = n1d < par.dens_max ? n1d : par.dens_max;
          }
          double ie[kEpt];
          bool far = false;
          // eps(q; n1D) of Eps1D (coulomb.py:1185-1190)
          auto eps = [&](int d, double le, double lh) {
            return (1.0 - 2.0 * blk[5 * nk + d] * le) - 2.0 * blk[6 * nk + d] * lh;
          };
#pragma unroll
          for (int e = 0; e < kEpt; ++e) {
            const int d = min(tid + e * T, nk - 1);
            ie[e] = 1.0;
            if (scr) {
              const double qe = blk[7 * nk + d], qh = blk[8 * nk + d];
              const double le = log_ratio(qe - kPi * n1d, qe + n1d, far);
              const double lh = log_ratio(qh - kPi * n1d, qh + n1d, far);
              ie[e] = 1.0 / eps(d, le, lh);
            }
          }
          if (far) {
#pragma unroll 1
            for (int e = 0; e < kEpt; ++e) {
              const int d = min(tid + e * T, nk - 1);
              const double qe = blk[7 * nk + d], qh = blk[8 * nk + d];
              const double v = 1.0 / eps(d, log(fabs((qe - kPi * n1d) / (qe + n1d))),
                                         log(fabs((qh - kPi * n1d) / (qh + n1d))));
              if (e == 0) ie[0] = v;
              else ie[kEpt - 1] = v;
            }
          }
#pragma unroll
          for (int e = 0; e < kEpt; ++e) {
            const int d = tid + e * T;
            for (int n = 0; n < (one ? 1 : 3); ++n)
              vq[n * np + d] = d > 0 && d < nk ? blk[n * nk + d] * ie[e] : 0.0;
          }
          cta_sync<L>();
        }
        // rounds: the tables' spectra, the stage point
        for (int rnd = build ? 0 : 1; rnd < 2; ++rnd) {
          if (rnd == 1 || sig == 0 || !one) {
            double2 x[8];
            if (rnd == 1) {
              const double2* src = (sig == 0 ? yp : yn) + col;
#pragma unroll
              for (int r = 0; r < 8; ++r) x[r] = src[q * r];
            } else {
              // the even table c[d] = c[M - d] = V(d): the points a + q r and
              // a + q (r + 8), added (even outputs) or subtracted
              const double* v0 = vq + (sig == 0 ? 0 : np);
              const double* v1 = vq + 2 * np;
              const double sg = half ? -1.0 : 1.0;
#pragma unroll
              for (int r = 0; r < 8; ++r) {
                const int d = col + q * r, dm = np - d;  // M - (d + np); np: no such point
                x[r] = make_double2(fma(sg, dm < np ? v0[dm] : 0.0, v0[d]), 0.0);
                if (sig) x[r].y = fma(sg, dm < np ? v1[dm] : 0.0, v1[d]);
              }
            }
            pass_a<q, rs>(x, ea, twa + col, half);
          }
          cta_sync<L>();
          pass_b<L>(rnd == 0 ? kTables : (one ? kOneTable : kDistinct), one, E, S, twb,
                    ih * (1.0 / (16 * q)));
          cta_sync<L>();
        }
        pass_a_inv<q, rs>(ea, twa + col, half);
        cta_sync<L>();
      }
      // M(t), M(t + h/2) twice, M(t + h)
      const int sd = s % kDrive;
      const double2 m = MODE == kLeapfrog ? m_lf
                        : st == 0         ? (sd == 0 ? par.drive[kDrive][0] : par.drive[sd - 1][1])
                                          : par.drive[sd][st == 3 ? 1 : 0];
      const double gamma = par.gamma;
      // sums over k: Re p, Im p, and n_e + n_h or n_e, n_h
      double v[4] = {0.0, 0.0, 0.0, 0.0};
      // (points beyond Nk go through the same arithmetic and stay zero)
#pragma unroll
      for (int e = 0; e < kEpt; ++e) {
        const int k = tid + e * T;
        const bool in = k < nk;
        double2 om = m;
        double xe = 0.0, xh = 0.0;
        if (exc) {
          // k = a + q r: rows 2 r and 2 r + 1, column a
          const double2* o = E + 2 * (k / q) * rs + k % q;
          const double2 p0 = o[0], p1 = o[rs], n0 = o[16 * rs], n1 = o[17 * rs];
          double2 dp = make_double2(p0.x + p1.x, p0.y + p1.y);
          xe = n0.x + n1.x;
          xh = n0.y + n1.y;
          if (apart) {
            dp = make_double2(some[0] ? dp.x : 0.0, some[1] ? ldexp(dp.y, -up[0]) : 0.0);
            xe = some[2] ? xe : 0.0;
            xh = some[3] ? xh : 0.0;
          }
          om.x += dp.x;
          om.y += dp.y;
        }
        if (ONCE && mode == kCalcH) {
          // renormalised H diagonals (CalcH, SBEs.py:819-935): Heh (Rabi
          // frequency), Hee, Hhh in the slots of dy
          if (in) {
            const double hb = bt.hbar;
            double2* d2 = reinterpret_cast<double2*>(bt.dy + 4 * off);
            d2[2 * k] = make_double2(om.x * hb, om.y * hb);
            d2[2 * k + 1] = make_double2((blk[3 * nk + k] + par.gap) - xe * hb,
                                         blk[4 * nk + k] - ldexp(xh * hb, -up[1]));
          }
          continue;
        }
        // diagonal of dpdt, dCdt, dDdt (SBEs.py:1962-1975, 2325-2337,
        // 2623-2636), everything over hbar
        const double2 p = yp[k], n = yn[k];
        const double sh = ekh[e] - (xe + xh), nn = n.x + n.y - 1.0;
        const double f0 = sh * p.y - om.y * nn - gamma * p.x;
        const double f1 = om.x * nn - sh * p.x - gamma * p.y;
        const double f2 = 2.0 * (om.y * p.x - om.x * p.y);
        if (ONCE) {
          if (in) {
            double2* d2 = reinterpret_cast<double2*>(bt.dy + 4 * off);
            d2[2 * k] = make_double2(f0, f1);
            d2[2 * k + 1] = make_double2(f2, f2);
          }
          continue;
        }
        double2 zp, zn;
        if (MODE == kRk4) {
          // stages of integrator.py:143-157; acc = k1 + 2 k2 + 2 k3, and at
          // the last stage k1 + 2 k2 + 2 k3 + k4
          const double w = st == 1 || st == 2 ? 2.0 : 1.0;
          acc[e][0] = fma(w, f0, st == 0 ? 0.0 : acc[e][0]);
          acc[e][1] = fma(w, f1, st == 0 ? 0.0 : acc[e][1]);
          acc[e][2] = fma(w, f2, st == 0 ? 0.0 : acc[e][2]);
          const double c = st == 2 ? h : (st == 3 ? h6 : h2);
          const double g0 = st == 3 ? acc[e][0] : f0, g1 = st == 3 ? acc[e][1] : f1;
          const double g2 = st == 3 ? acc[e][2] : f2;
          zp = make_double2(fma(c, g0, yb[e][0]), fma(c, g1, yb[e][1]));
          zn = make_double2(fma(c, g2, yb[e][2]), fma(c, g2, yb[e][3]));
        } else {
          // leapfrog X3 = X1 + 2 dt f(X2) (SBEs.py:5685-5687) and the
          // occupations |n| for the rescale (SBEs.py:5704-5711)
          zp = make_double2(yb[e][0] + f0 * h * 2.0, yb[e][1] + f1 * h * 2.0);
          zn = make_double2(fabs(yb[e][2] + f2 * h * 2.0), fabs(yb[e][3] + f2 * h * 2.0));
        }
        if (!in) zp = zn = make_double2(0.0, 0.0);
        yp[k] = zp;
        yn[k] = zn;
        if (MODE == kRk4 && st == 3) {
          yb[e][0] = zp.x;
          yb[e][1] = zp.y;
          yb[e][2] = zn.x;
          yb[e][3] = zn.y;
        }
        v[0] += zp.x;
        v[1] += zp.y;
        v[2] += MODE == kRk4 ? zn.x + zn.y : zn.x;
        v[3] += zn.y;
      }
      if (ONCE) return;
      par_red ^= 1;
      if (MODE == kRk4) {
        // sums: n1D for the next stage's screening, P(t) after the last stage
        if (st == 3) {
          double u[4] = {v[2], v[0], v[1], 0.0};
          put_sums<4>(u, par.red[par_red], lane, warp);
        } else if (scr) {
          double u[2] = {v[2], 0.0};
          put_sums<2>(u, par.red[par_red], lane, warp);
        }
        cta_sync<L>();
      } else {
        double u[4] = {v[2], v[0], v[1], v[3]};
        put_sums<4>(u, par.red[par_red], lane, warp);
        cta_sync<L>();
        const double te = get_sum<L>(par.red[par_red], 0), th = get_sum<L>(par.red[par_red], 3);
        const double total = (te + th) / 2.0, small = 1e-200;
        const double ce = total / (te + small), ch = total / (th + small);
#pragma unroll
        for (int e = 0; e < kEpt; ++e) {
          const int k = tid + e * T;
          const double2 zp = yp[k];
          double2 zn = yn[k];
          zn = make_double2(zn.x * ce, zn.y * ch);
          yn[k] = zn;
          yb[e][0] = (yb[e][0] + zp.x) / 2.0;
          yb[e][1] = (yb[e][1] + zp.y) / 2.0;
          yb[e][2] = (yb[e][2] + zn.x) / 2.0;
          yb[e][3] = (yb[e][3] + zn.y) / 2.0;
        }
        ntot = te * ce + th * ch;
        cta_sync<L>();
      }
    }
    t = t + h;
    // P(t) record (qwoptics.py:815-946, diagonal: pscale * sum_k p_k)
    if (tid == 0 && bt.P && bt.p_stride > 0 && (s + 1) % bt.p_stride == 0) {
      const int r = (s + 1) / bt.p_stride - 1;
      const int64_t po = par.p_off;
      if (r < bt.p_cap && po >= 0 && po + r < bt.n_P) {
        bt.P[2 * (po + r)] = par.pscale * get_sum<L>(par.red[par_red], 1);
        bt.P[2 * (po + r) + 1] = par.pscale * get_sum<L>(par.red[par_red], 2);
      }
    }
  }
  if (ONCE) return;

  // Write the state back; flag non-finite wires.
  bool bad = false;
  double2* yo = reinterpret_cast<double2*>(bt.y + 4 * off);
  double2* y1o = reinterpret_cast<double2*>(bt.y1 + 4 * off);
#pragma unroll
  for (int e = 0; e < kEpt; ++e) {
    const int k = tid + e * T;
    if (k >= nk) continue;
    const double2 a = yp[k], b = yn[k];
    yo[2 * k] = a;
    yo[2 * k + 1] = b;
    bad |= !(isfinite(a.x) && isfinite(a.y) && isfinite(b.x) && isfinite(b.y));
    if (MODE == kLeapfrog) {
      y1o[2 * k] = make_double2(yb[e][0], yb[e][1]);
      y1o[2 * k + 1] = make_double2(yb[e][2], yb[e][3]);
      bad |= !(isfinite(yb[e][0]) && isfinite(yb[e][1]) && isfinite(yb[e][2]) &&
               isfinite(yb[e][3]));
    }
  }
  bad = L == 1 ? __any_sync(0xffffffffu, bad) : (bool)__syncthreads_or(bad);
  if (tid == 0) {
    wp->t = t;
    wp->steps = steps0 + nst;
    if (bad && wp->status == PSB_OK) wp->status = PSB_ERR_NONFINITE;
  }
}

// A launch covers the wires of its grid whose own Nk takes L lanes; the others
// are another launch's, unless the caller said that there are none (strict).
// check: this launch reports bad descriptors.
template <int L, int MODE>
__device__ __forceinline__ void wire_of_cta(const Batch& bt, int mode, bool screened, bool shared,
                                            bool check, bool strict, uint8_t* smem) {
  const int wi = bt.order ? bt.order[blockIdx.x] : (int)blockIdx.x;
  if (wi < 0 || wi >= bt.nw) return;
  PsbWire* wp = bt.wires + wi;
  const int table = wp->table;
  int bad = PSB_OK;
  PsbTable tb{};
  if (table < 0 || table >= bt.ntab) {
    bad = PSB_ERR_INVALID;
  } else {
    tb = bt.tables[table];
    const int64_t off = wp->off;
    if (tb.nk < 2 || tb.nk > bt.nk_limit || off < 0 || off + tb.nk > bt.n_state || tb.off < 0 ||
        tb.off + 9 * (int64_t)tb.nk > bt.n_tabdata || (strict && lanes_of(tb.nk) != L))
      bad = PSB_ERR_SIZE;
    else if (shared && (tb.flags & PSB_TAB_SHARED_V) == 0)
      bad = PSB_ERR_INVALID;
  }
  if (bad != PSB_OK) {
    if (check && threadIdx.x == 0) wp->status = bad;
    return;
  }
  if (lanes_of(tb.nk) == L) wire_steps<L, MODE>(bt, mode, screened, smem, wi, tb);
}

// The launches of one call over several classes follow one another on the
// stream, but their wires are different ones: each lets the next start once its
// CTAs have, and a chained one reads nothing that the one before writes.  Its
// first CTA stays until the launch before is complete, so that what follows on
// the stream finds the whole call done.  One RK4 step of 192 wires of Nk 64, 128
// and 256: 46 us one after another, 21 chained (31 with direct sums in one
// launch).
template <int L, int MODE>
__global__ void __launch_bounds__(32 * L, ctas_of(L))
    sbe_conv_kernel(Batch bt, int mode, bool screened, bool shared, bool check, bool strict,
                    bool chained) {
  extern __shared__ __align__(16) uint8_t smem[];
  asm volatile("griddepcontrol.launch_dependents;");
  wire_of_cta<L, MODE>(bt, mode, screened, shared, check, strict, smem);
  if (chained && blockIdx.x == 0) asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <int L>
uint32_t smem_of(bool shared) {
  return shared ? Lay<L>::total1 : Lay<L>::total3;
}

template <int L, int MODE>
int launch_lanes(const Batch& bt, int mode, int grid, bool screened, bool shared, bool check,
                 bool strict, bool chained, cudaStream_t st) {
  const uint32_t smem = smem_of<L>(shared);
  const int rc = allow_smem(sbe_conv_kernel<L, MODE>, smem, Lay<L>::total3);
  if (rc != PSB_OK) return rc;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(32 * L);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = chained ? 1 : 0;
  cudaLaunchKernelEx(&cfg, sbe_conv_kernel<L, MODE>, bt, mode, screened, shared, check, strict,
                     chained);
  return check_cuda("sbe_conv_kernel");
}

// One launch per width from that of nkmax down to that of nkmin + 1 (a single
// right-hand side: of the widths above the direct kernel's only).
template <int L, int MODE>
int launch_down(const Batch& bt, int mode, int grid, int nkmax, int nkmin, bool screened,
                bool shared, bool one_class, cudaStream_t st) {
  const int top = lanes_of(nkmax);
  if (L <= top && L >= lanes_of(nkmin + 1)) {
    const int rc = launch_lanes<L, MODE>(bt, mode, grid, screened, shared, L == top, one_class,
                                         L < top, st);
    if (rc != PSB_OK || one_class) return rc;
  }
  if constexpr (L > (MODE == kRhs ? lanes_of(kDirectNk + 1) : 1))
    return launch_down<L / 2, MODE>(bt, mode, grid, nkmax, nkmin, screened, shared, one_class, st);
  return PSB_OK;
}

}  // namespace conv

size_t conv_smem_bytes(int nk, bool shared) {
  switch (conv::lanes_of(nk)) {
    case 1: return conv::smem_of<1>(shared);
    case 2: return conv::smem_of<2>(shared);
    case 4: return conv::smem_of<4>(shared);
    case 8: return conv::smem_of<8>(shared);
    default: return conv::smem_of<16>(shared);
  }
}

int launch_sbe_conv(const Batch& bt, int mode, int grid, int nkmax, int nkmin, bool screened,
                    bool shared, bool one_class, cudaStream_t st) {
  if (mode == kRk4)
    return conv::launch_down<16, kRk4>(bt, mode, grid, nkmax, nkmin, screened, shared, one_class,
                                       st);
  if (mode == kLeapfrog)
    return conv::launch_down<16, kLeapfrog>(bt, mode, grid, nkmax, nkmin, screened, shared,
                                            one_class, st);
  return conv::launch_down<16, kRhs>(bt, mode, grid, nkmax, nkmin, screened, shared, one_class,
                                     st);
}

}  // namespace psb
