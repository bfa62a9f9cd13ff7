// Transforms held in registers: a line of N = R1 * R2 complex values is
// transformed in two steps, an R1-point and an R2-point DFT that one thread
// each computes on values in its registers, with a single exchange through
// shared memory between them.
//
//   N = R1 R2, n = n1 R2 + n2, k = k1 + R1 k2:
//   step A, thread n2 < R2: DFT of length R1 over n1, times W_N^(n2 k1)
//   exchange
//   step B, thread k1 < R1: DFT of length R2 over n2 -> k2
//
// The lengths are template parameters, so every shared-memory address is a
// base plus an immediate and the index arithmetic that bound the run-time
// radix stages of fft_core.cuh (about 250 instructions per output element,
// ncu) is gone.  The stages of fft_core.cuh stay for every other length.
#pragma once
#include "fft_core.cuh"

namespace lesgo {

// cos and sin of 2 pi m / R for the composite butterflies' inner twiddles
// (the 9- and 16-point ones; the others are prime-factor products).
__host__ __device__ constexpr double root_cos(int m, int R) {
  m %= R;
  if (2 * m > R) m = R - m;
  const int t = 144 * m / R;   // in units of 2.5 degrees (R divides 144)
  return t == 4 ? 0.98480775301220805937 : t == 8 ? 0.93969262078590838405 : t == 9 ? 0.92387953251128675613
       : t == 16 ? 0.76604444311897803520 : t == 18 ? 0.70710678118654752440 : t == 20 ? 0.64278760968653932632
       : t == 27 ? 0.38268343236508977173 : t == 28 ? 0.34202014332566873304 : t == 32 ? 0.17364817766693034885
       : -root_cos(72 - t, 144);
}
__host__ __device__ constexpr double root_sin(int m, int R) {
  // sin(x) = cos(x - pi/2), m / R of a turn -> 144ths
  const int t = 144 * (m % R) / R;
  return root_cos((t + 108) % 144, 144);
}

// a table value in the arithmetic A (double-word: hi and the rounded rest)
template <typename A> __host__ __device__ constexpr A root_const(double v) {
  if constexpr (std::is_same<A, df64>::value) return df64{(float)v, (float)(v - (double)(float)v)};
  else return (A)v;
}

// a * exp(-2 pi i M / R), or its conjugate rotation with INV
template <int M, int R, bool INV, typename T2>
__device__ __forceinline__ T2 mul_root(T2 a) {
  using A = decltype(a.x);
  constexpr int m = M % R;
  if constexpr (m == 0) return a;
  else if constexpr (4 * m == R) return INV ? mul_pi(a) : mul_mi(a);
  else if constexpr (2 * m == R) return mkc(-a.x, -a.y);
  else if constexpr (4 * m == 3 * R) return INV ? mul_mi(a) : mul_pi(a);
  else if constexpr (8 * m == R || 8 * m == 3 * R || 8 * m == 5 * R || 8 * m == 7 * R) {
    constexpr double cd = root_cos(m, R), sd = INV ? root_sin(m, R) : -root_sin(m, R);
    constexpr A c = root_const<A>(cd);   // +- sqrt(1/2)
    if constexpr (std::is_same<T2, dfc>::value)
      return cscale((cd > 0) == (sd > 0) ? csub(a, mul_mi(a)) : cadd(a, mul_mi(a)), c);
    else if constexpr ((cd > 0) == (sd > 0)) return mkc(c * (a.x - a.y), c * (a.x + a.y));
    else return mkc(c * (a.x + a.y), c * (a.y - a.x));
  } else {
    constexpr A c = root_const<A>(root_cos(m, R));
    constexpr A s = root_const<A>(INV ? root_sin(m, R) : -root_sin(m, R));
    if constexpr (std::is_same<T2, dfc>::value) return cmul(a, mkc(c, s));
    else return mkc(a.x * c - a.y * s, a.x * s + a.y * c);
  }
}

template <int V> struct IntC { static constexpr int value = V; };
template <int B, int E, typename F>
__device__ __forceinline__ void static_for(F&& f) {
  if constexpr (B < E) {
    f(IntC<B>{});
    static_for<B + 1, E>(f);
  }
}

// In-register DFT of R values, natural order in and out.
template <typename T2, bool INV, int R> struct Dft;
template <typename T2, bool INV> struct Dft<T2, INV, 1> {
  __device__ static __forceinline__ void run(T2*) {}
};
template <typename T2, bool INV> struct Dft<T2, INV, 2> {
  __device__ static __forceinline__ void run(T2* v) { bfly2<T2, INV>(v[0], v[1]); }
};
template <typename T2, bool INV> struct Dft<T2, INV, 3> {
  __device__ static __forceinline__ void run(T2* v) { bfly3<T2, INV>(v[0], v[1], v[2]); }
};
template <typename T2, bool INV> struct Dft<T2, INV, 4> {
  __device__ static __forceinline__ void run(T2* v) { bfly4<T2, INV>(v[0], v[1], v[2], v[3]); }
};
template <typename T2, bool INV> struct Dft<T2, INV, 8> {
  __device__ static __forceinline__ void run(T2* v) { bfly8<T2, INV>(v); }
};
// A * B with inner twiddles (Cooley-Tukey)
template <typename T2, bool INV, int A, int B> struct DftCT {
  __device__ static __forceinline__ void run(T2* v) {
    constexpr int R = A * B;
    T2 t[R];
    static_for<0, B>([&](auto n2) {
      T2 u[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) u[n1] = v[B * n1 + n2.value];
      Dft<T2, INV, A>::run(u);
      static_for<0, A>([&](auto k1) {
        t[k1.value * B + n2.value] = mul_root<n2.value * k1.value, R, INV>(u[k1.value]);
      });
    });
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      Dft<T2, INV, B>::run(t + k1 * B);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = t[k1 * B + k2];
    }
  }
};
// A * B with A and B coprime: no inner twiddles (Good 1958, Thomas 1963)
__host__ __device__ constexpr int inv_mod(int a, int m) {
  for (int x = 1; x < m; ++x)
    if (a * x % m == 1) return x;
  return 1;
}
template <typename T2, bool INV, int A, int B> struct DftPF {
  __device__ static __forceinline__ void run(T2* v) {
    constexpr int R = A * B;
    constexpr int ea = B * inv_mod(B % A, A), eb = A * inv_mod(A % B, B);
    T2 t[R];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      T2 u[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) u[n1] = v[(B * n1 + A * n2) % R];
      Dft<T2, INV, A>::run(u);
#pragma unroll
      for (int k1 = 0; k1 < A; ++k1) t[k1 * B + n2] = u[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      Dft<T2, INV, B>::run(t + k1 * B);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) v[(ea * k1 + eb * k2) % R] = t[k1 * B + k2];
    }
  }
};
template <typename T2, bool INV> struct Dft<T2, INV, 6> : DftPF<T2, INV, 2, 3> {};
template <typename T2, bool INV> struct Dft<T2, INV, 9> : DftCT<T2, INV, 3, 3> {};
template <typename T2, bool INV> struct Dft<T2, INV, 12> : DftPF<T2, INV, 4, 3> {};
template <typename T2, bool INV> struct Dft<T2, INV, 16> : DftCT<T2, INV, 4, 4> {};
template <typename T2, bool INV> struct Dft<T2, INV, 18> : DftPF<T2, INV, 2, 9> {};
template <typename T2, bool INV> struct Dft<T2, INV, 24> : DftPF<T2, INV, 8, 3> {};

__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int odd_up(int a) { return a | 1; }

// v *= W^(k1 n2) (forward) or its conjugate (INV); tw[k1 * R2 + n2]
template <bool INV, typename T2> __device__ __forceinline__ T2 mul_tw(T2 a, const T2* w) {
  const T2 t = ldt(w);
  return INV ? cmulconj(a, t) : cmul(a, t);
}

// i k a, and a + i k b
template <typename T2, typename A> __device__ __forceinline__ T2 mul_ik(A k, T2 a) {
  if constexpr (std::is_same<T2, dfc>::value) return cscale(mul_pi(a), k);
  else return mkc(-k * a.y, k * a.x);
}
template <typename T2, typename A> __device__ __forceinline__ T2 add_ik(T2 a, A k, T2 b) {
  if constexpr (std::is_same<T2, dfc>::value) return cadd(a, mul_ik(k, b));
  else return mkc(a.x - k * b.y, a.y + k * b.x);
}

// The factors of a length, chosen at compile time from a list; the host
// asks the same list (rx_factors, ry_factors, rxb_factors) to build the
// twiddle table.
template <int A, int B> struct Len {
  static constexpr int R1 = A, R2 = B, N = A * B;
};

}  // namespace lesgo
