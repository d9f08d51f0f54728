// Short complex DFTs held entirely in registers (device code): every index
// and twiddle is a compile-time constant.  Additions and real-by-complex
// products run as packed f32x2 instructions (one issue slot for the real and
// the imaginary part, each rounded to nearest as the scalar instruction
// rounds it).
#pragma once

#include "common.cuh"

namespace avx {

AVX_D unsigned long long f2_bits(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
AVX_D float2 f2_of(unsigned long long r) {
  float2 a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
  return a;
}
AVX_D float2 add2(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)));
  return f2_of(r);
}
// a b + c, component by component
AVX_D float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(b)), "l"(f2_bits(c)));
  return f2_of(r);
}
AVX_D float2 sub2(float2 a, float2 b) { return fma2(b, make_float2(-1.f, -1.f), a); }
AVX_D float2 scale2(float2 a, float s) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_bits(a)), "l"(f2_bits(make_float2(s, s))));
  return f2_of(r);
}
// a + i s b for s = +1 / -1
template <int S>
AVX_D float2 add_i(float2 a, float2 b) {
  return S > 0 ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, a.y - b.x);
}

// cos and sin of 2 pi k / n as constants: the angle is reduced to the first
// octant, where the Taylor series to degree 17 is exact to double precision.
struct CosSin {
  double c, s;
};
constexpr CosSin cossin_octant(double a) {
  double c = 1.0, s = a, tc = 1.0, ts = a;
  for (int i = 1; i <= 8; ++i) {
    tc *= -a * a / ((2 * i - 1) * (2 * i));
    ts *= -a * a / ((2 * i) * (2 * i + 1));
    c += tc;
    s += ts;
  }
  return CosSin{c, s};
}
constexpr CosSin root_of_unity(int k, int n) {
  k %= n;
  if (k < 0) k += n;
  if (8 * k > 4 * n) {  // conjugate half
    const CosSin r = root_of_unity(n - k, n);
    return CosSin{r.c, -r.s};
  }
  if (8 * k > 2 * n) {  // second quadrant: pi - a, with a = pi (1 - 2 k / n)
    const CosSin r = root_of_unity(n - 2 * k, 2 * n);
    return CosSin{-r.c, r.s};
  }
  if (8 * k > n) {  // second octant: pi / 2 - a
    const CosSin r = cossin_octant(6.283185307179586476925 * (n - 4 * k) / (4.0 * n));
    return CosSin{r.s, r.c};
  }
  return cossin_octant(6.283185307179586476925 * k / n);
}

// v * exp(SIGN 2 pi i K / N)
template <int K, int N, int SIGN>
AVX_D float2 mul_root(float2 v) {
  if constexpr (K % N == 0) {
    return v;
  } else if constexpr (4 * K == N) {
    return SIGN > 0 ? make_float2(-v.y, v.x) : make_float2(v.y, -v.x);
  } else if constexpr (2 * K == N) {
    return make_float2(-v.x, -v.y);
  } else if constexpr (8 * K == N || 8 * K == 3 * N) {
    constexpr float h = 0.70710678118654752440f;
    constexpr float s = SIGN > 0 ? h : -h;
    if constexpr (8 * K == N)
      return SIGN > 0 ? make_float2(h * (v.x - v.y), h * (v.y + v.x)) : make_float2(h * (v.x + v.y), h * (v.y - v.x));
    else
      return make_float2(fmaf(-s, v.y, -h * v.x), fmaf(s, v.x, -h * v.y));
  } else {
    constexpr CosSin r = root_of_unity(K, N);
    constexpr float c = (float)r.c, s = (float)(SIGN > 0 ? r.s : -r.s);
    return make_float2(fmaf(-s, v.y, c * v.x), fmaf(s, v.x, c * v.y));
  }
}

constexpr int first_radix(int n) {
  for (int r : {4, 2, 3, 5, 7, 11, 13})
    if (n % r == 0) return r;
  return n;
}

template <int N, int SIGN>
AVX_D void reg_dft(float2 (&v)[N]);

template <int N, int SIGN, int R, int M, int B>
AVX_D void reg_columns(float2 (&v)[N]) {
  if constexpr (B < M) {
    float2 a[R];
#pragma unroll
    for (int i = 0; i < R; ++i) a[i] = v[M * i + B];
    reg_dft<R, SIGN>(a);
#pragma unroll
    for (int i = 0; i < R; ++i) v[M * i + B] = a[i];
    reg_columns<N, SIGN, R, M, B + 1>(v);
  }
}
template <int N, int SIGN, int R, int M, int C, int B>
AVX_D void reg_twiddle_row(float2 (&a)[M]) {
  if constexpr (B < M) {
    a[B] = mul_root<B * C, N, SIGN>(a[B]);
    reg_twiddle_row<N, SIGN, R, M, C, B + 1>(a);
  }
}
template <int N, int SIGN, int R, int M, int C>
AVX_D void reg_rows(const float2 (&v)[N], float2 (&out)[N]) {
  if constexpr (C < R) {
    float2 a[M];
#pragma unroll
    for (int i = 0; i < M; ++i) a[i] = v[M * C + i];
    reg_twiddle_row<N, SIGN, R, M, C, 1>(a);
    reg_dft<M, SIGN>(a);
#pragma unroll
    for (int i = 0; i < M; ++i) out[C + R * i] = a[i];
    reg_rows<N, SIGN, R, M, C + 1>(v, out);
  }
}
// odd prime N: X_q, X_{N-q} = v0 + sum_k cos(2 pi k q / N) (v_k + v_{N-k}) +- i SIGN sum_k sin(..) (v_k - v_{N-k})
template <int N, int SIGN, int Q, int K>
AVX_D void reg_prime_sum(const float2 (&t)[N], float2& m, float2& s) {
  if constexpr (K <= N / 2) {
    constexpr CosSin r = root_of_unity(K * Q, N);
    constexpr float c = (float)r.c, d = (float)r.s;
    m = fma2(t[K], make_float2(c, c), m);
    if constexpr (K == 1)
      s = scale2(t[N - K], d);
    else
      s = fma2(t[N - K], make_float2(d, d), s);
    reg_prime_sum<N, SIGN, Q, K + 1>(t, m, s);
  }
}
template <int N, int SIGN, int Q>
AVX_D void reg_prime(const float2 (&t)[N], float2 (&v)[N]) {
  if constexpr (Q <= N / 2) {
    float2 m = t[0], s;
    reg_prime_sum<N, SIGN, Q, 1>(t, m, s);
    v[Q] = add_i<SIGN>(m, s);
    v[N - Q] = add_i<-SIGN>(m, s);
    reg_prime<N, SIGN, Q + 1>(t, v);
  }
}

// v[k] <- sum_n v[n] exp(SIGN 2 pi i n k / N), natural order on both sides
template <int N, int SIGN>
AVX_D void reg_dft(float2 (&v)[N]) {
  if constexpr (N == 1) {
  } else if constexpr (N == 2) {
    const float2 a = v[0];
    v[0] = add2(a, v[1]);
    v[1] = sub2(a, v[1]);
  } else if constexpr (N == 4) {
    const float2 a0 = add2(v[0], v[2]), a1 = sub2(v[0], v[2]);
    const float2 b0 = add2(v[1], v[3]), b1 = sub2(v[1], v[3]);
    v[0] = add2(a0, b0);
    v[1] = add_i<SIGN>(a1, b1);
    v[2] = sub2(a0, b0);
    v[3] = add_i<-SIGN>(a1, b1);
  } else if constexpr (first_radix(N) == N) {
    float2 t[N];
    t[0] = v[0];
    float2 sum = v[0];
#pragma unroll
    for (int k = 1; k <= N / 2; ++k) {
      t[k] = add2(v[k], v[N - k]);
      t[N - k] = sub2(v[k], v[N - k]);
      sum = add2(sum, t[k]);
    }
    reg_prime<N, SIGN, 1>(t, v);
    v[0] = sum;
  } else {
    constexpr int R = first_radix(N), M = N / R;
    float2 o[N];
    reg_columns<N, SIGN, R, M, 0>(v);
    reg_rows<N, SIGN, R, M, 0>(v, o);
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = o[i];
  }
}

}  // namespace avx
