// fft64.cuh -- small FP64 discrete Fourier transforms (2, 4 or 8 points) held
// in one thread's registers, the building blocks of the exchange sums' fast
// convolution (sbe_conv.cu).
#pragma once

namespace psb {
namespace fft {

// cos and sin of pi k / 8, k = 0 .. 4
constexpr double kCos16[5] = {1.0, 0.9238795325112867, 0.7071067811865476, 0.3826834323650898,
                              0.0};

template <int I>
struct Int {
  static constexpr int value = I;
};
template <int N, int I = 0, class F>
__device__ __forceinline__ void unroll(F&& f) {
  if constexpr (I < N) {
    f(Int<I>{});
    unroll<N, I + 1>(f);
  }
}

__device__ __forceinline__ double2 add(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 sub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
// a w (SG = -1) or a conj(w) (SG = +1) for a forward root w = c - i s
template <int SG>
__device__ __forceinline__ double2 mulw(double2 a, double2 w) {
  return SG < 0 ? make_double2(fma(a.x, w.x, -(a.y * w.y)), fma(a.x, w.y, a.y * w.x))
                : make_double2(fma(a.x, w.x, a.y * w.y), fma(a.y, w.x, -(a.x * w.y)));
}
// a exp(SG 2 pi i K / 16), K = 0 .. 7
template <int K, int SG>
__device__ __forceinline__ double2 rot16(double2 a) {
  constexpr double r = kCos16[2];
  if constexpr (K == 0) {
    return a;
  } else if constexpr (K == 4) {
    return SG < 0 ? make_double2(a.y, -a.x) : make_double2(-a.y, a.x);
  } else if constexpr (K == 2) {
    return SG < 0 ? make_double2(r * (a.x + a.y), r * (a.y - a.x))
                  : make_double2(r * (a.x - a.y), r * (a.x + a.y));
  } else if constexpr (K == 6) {
    return SG < 0 ? make_double2(r * (a.y - a.x), -r * (a.x + a.y))
                  : make_double2(-r * (a.x + a.y), r * (a.x - a.y));
  } else {
    constexpr double c = K < 4 ? kCos16[K < 4 ? K : 0] : -kCos16[K < 4 ? 0 : 8 - K];
    constexpr double s = K < 4 ? kCos16[K < 4 ? 4 - K : 0] : kCos16[K < 4 ? 0 : K - 4];
    return SG < 0 ? make_double2(fma(a.x, c, a.y * s), fma(a.y, c, -(a.x * s)))
                  : make_double2(fma(a.x, c, -(a.y * s)), fma(a.y, c, a.x * s));
  }
}

template <int N, int SG>
struct Dft;

template <int SG>
struct Dft<2, SG> {
  static __device__ __forceinline__ void run(double2 (&x)[2]) {
    const double2 a = x[0];
    x[0] = add(a, x[1]);
    x[1] = sub(a, x[1]);
  }
};

template <int SG>
struct Dft<4, SG> {
  static __device__ __forceinline__ void run(double2 (&x)[4]) {
    const double2 t0 = add(x[0], x[2]), t1 = sub(x[0], x[2]);
    const double2 t2 = add(x[1], x[3]), t3 = sub(x[1], x[3]);
    x[0] = add(t0, t2);
    x[2] = sub(t0, t2);
    // t1 + SG i t3, t1 - SG i t3
    const double2 it = SG < 0 ? make_double2(t3.y, -t3.x) : make_double2(-t3.y, t3.x);
    x[1] = add(t1, it);
    x[3] = sub(t1, it);
  }
};

// two transforms of 4 points, the roots of 8, the pairs
template <int SG>
struct Dft<8, SG> {
  static __device__ __forceinline__ void run(double2 (&x)[8]) {
    double2 e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
    Dft<4, SG>::run(e);
    Dft<4, SG>::run(o);
    o[1] = rot16<2, SG>(o[1]);
    o[2] = rot16<4, SG>(o[2]);
    o[3] = rot16<6, SG>(o[3]);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = add(e[k], o[k]);
      x[k + 4] = sub(e[k], o[k]);
    }
  }
};
template <int SG>
struct Dft<1, SG> {
  static __device__ __forceinline__ void run(double2 (&)[1]) {}
};

}  // namespace fft
}  // namespace psb
