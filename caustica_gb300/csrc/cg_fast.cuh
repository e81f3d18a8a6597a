// Size-specialised pencil FFTs: register DFT codelets with compile-time
// twiddles and a two-level ("four-step") transform with one shared-memory
// exchange per pencil transform (three levels and two exchanges on 125, 243, 250
// and 375 points, see fft3).
//
// A pencil of length N = A * B is held by B threads on input: thread s < B
// owns x[s + B a], a in [0, A). Phase 1 applies an A-point DFT in registers
// and the twiddle W_N^(s k1); the values go to shared memory as Y[k1][s];
// phase 2 thread s' < A reads Y[s'][n2], n2 in [0, B), and applies a B-point
// DFT, so thread s' ends up owning X[s' + A b], b in [0, B):
//   X[k1 + A k2] = sum_n2 W_N^(n2 k1) W_B^(n2 k2) sum_n1 x[B n1 + n2] W_A^(n1 k1).
// The output distribution of an (A, B) transform is the input distribution
// of a (B, A) transform, so a forward transform followed by an inverse one
// (or the reverse) needs no extra exchange.
//
// Register DFTs of composite size R = a b use the same decomposition inside
// one thread with compile-time twiddles W_R^m, evaluated by constexpr
// Taylor series of sin and cos (double precision, rounded once to float).
#pragma once

#include <stdlib.h>

#include <type_traits>
#include <utility>

#include "cg_common.cuh"

namespace cgf {

// ------------------------------------------------ compile-time sin/cos --
constexpr double kPi = 3.14159265358979323846264338327950288;

constexpr double ct_sin_series(double x) {
  double x2 = x * x, term = x, sum = x;
  for (int k = 1; k < 16; ++k) {
    term *= -x2 / ((2.0 * k) * (2.0 * k + 1.0));
    sum += term;
  }
  return sum;
}

constexpr double ct_cos_series(double x) {
  double x2 = x * x, term = 1.0, sum = 1.0;
  for (int k = 1; k < 16; ++k) {
    term *= -x2 / ((2.0 * k - 1.0) * (2.0 * k));
    sum += term;
  }
  return sum;
}

// cos(2 pi m / R) and sin(2 pi m / R), exact at multiples of pi/2
constexpr double ct_cos2pi(int m, int R) {
  int q = ((m % R) + R) % R;
  if ((4 * q) % R == 0) {
    int quad = (4 * q) / R;
    return quad == 0 ? 1.0 : (quad == 2 ? -1.0 : 0.0);
  }
  double x = 2.0 * kPi * (double)q / (double)R;
  if (x > kPi) x -= 2.0 * kPi;
  return ct_cos_series(x);
}

constexpr double ct_sin2pi(int m, int R) {
  int q = ((m % R) + R) % R;
  if ((4 * q) % R == 0) {
    int quad = (4 * q) / R;
    return quad == 1 ? 1.0 : (quad == 3 ? -1.0 : 0.0);
  }
  double x = 2.0 * kPi * (double)q / (double)R;
  if (x > kPi) x -= 2.0 * kPi;
  return ct_sin_series(x);
}

// ------------------------------------------------------ static loops --
template <int I, int N, class F>
__host__ __device__ __forceinline__ void static_for(F&& f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    static_for<I + 1, N>(f);
  }
}

// v * W_R^m, forward W = exp(-2 pi i m / R), inverse its conjugate
template <int R, int M, bool INV>
__host__ __device__ __forceinline__ float2 twiddle_ct(float2 v) {
  constexpr double c = ct_cos2pi(M, R);
  constexpr double s = INV ? ct_sin2pi(M, R) : -ct_sin2pi(M, R);
  constexpr float cf = (float)c, sf = (float)s;
  if constexpr (cf == 1.0f && sf == 0.0f) return v;
  if constexpr (cf == -1.0f && sf == 0.0f) return make_float2(-v.x, -v.y);
  if constexpr (cf == 0.0f && sf == 1.0f) return make_float2(-v.y, v.x);
  if constexpr (cf == 0.0f && sf == -1.0f) return make_float2(v.y, -v.x);
  return make_float2(f_fma(v.x, cf, -f_mul(v.y, sf)), f_fma(v.x, sf, f_mul(v.y, cf)));
}

template <bool INV>
__host__ __device__ __forceinline__ float2 rot(float2 a) {  // forward: -i a ; inverse: +i a
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

constexpr int ct_gcd(int a, int b) { return b == 0 ? a : ct_gcd(b, a % b); }
// Largest power of the smallest prime factor of R: coprime to the rest.
constexpr int ct_prime_power(int R) {
  const int p = R % 2 == 0 ? 2 : (R % 3 == 0 ? 3 : 5);
  int q = 1;
  while (R % p == 0) {
    q *= p;
    R /= p;
  }
  return q;
}
constexpr int ct_first_factor(int R) {
  const int q = ct_prime_power(R);
  return q < R ? q : ((R % 4 == 0 && R > 8) ? 4 : (R % 2 == 0 ? 2 : (R % 3 == 0 ? 3 : 5)));
}
// The k < A B with k = k1 mod A and k = k2 mod B (A, B coprime).
constexpr int ct_crt(int k1, int k2, int A, int B) {
  int k = k1;
  while (k % B != k2) k += A;
  return k;
}

// ------------------------------------------------------- DFT codelets --
// Composite sizes of coprime factors A, B by the prime-factor algorithm (Good
// 1958, Thomas 1963): n = (B n1 + A n2) mod R, k = k1 mod A = k2 mod B, an A x B
// transform without twiddles; the permutations are register names. Powers of
// one prime by Cooley and Tukey's, with twiddles in between. A step with twiddles
// everywhere -> as it is: 192x192x256 275.7 -> 274.6 us, 320^3 1182 -> 1165,
// 384^3 1946 -> 1895, 400^3 2173 -> 2111; the error of a round trip against 64
// bits 1.86e-7 -> 1.79e-7 at 180 points, 2.05e-7 -> 1.89e-7 at 400.
// FINE: the factors of 5 multiply by sin(2 pi/5) as a pair of floats (fft2).
template <int R, bool INV, bool FINE>
struct Dft {
  static constexpr int A = ct_first_factor(R), B = R / A;
  static constexpr bool COPRIME = ct_gcd(A, B) == 1;
  __host__ __device__ __forceinline__ static void run(float2* v) {
    if constexpr (COPRIME)
      run_coprime(v);
    else
      run_twiddled(v);
  }
  __host__ __device__ __forceinline__ static void run_coprime(float2* v) {
    float2 o[R];  // o[B k1 + n2], then o[B k1 + k2]
    static_for<0, B>([&](auto ni) {
      constexpr int n2 = decltype(ni)::value;
      float2 t[A];
      static_for<0, A>([&](auto mi) {
        constexpr int n1 = decltype(mi)::value;
        t[n1] = v[(B * n1 + A * n2) % R];
      });
      Dft<A, INV, FINE>::run(t);
      static_for<0, A>([&](auto ki) { o[B * decltype(ki)::value + n2] = t[decltype(ki)::value]; });
    });
    static_for<0, A>([&](auto ki) { Dft<B, INV, FINE>::run(o + B * decltype(ki)::value); });
    static_for<0, A>([&](auto k1i) {
      static_for<0, B>([&](auto k2i) {
        constexpr int k1 = decltype(k1i)::value, k2 = decltype(k2i)::value;
        constexpr int k = ct_crt(k1, k2, A, B);
        v[k] = o[B * k1 + k2];
      });
    });
  }
  __host__ __device__ __forceinline__ static void run_twiddled(float2* v) {
    static_for<0, B>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      float2 t[A];
      static_for<0, A>([&](auto ai) { t[decltype(ai)::value] = v[B * decltype(ai)::value + b]; });
      Dft<A, INV, FINE>::run(t);
      static_for<0, A>([&](auto ai) {
        constexpr int a = decltype(ai)::value;
        v[B * a + b] = twiddle_ct<R, a * b, INV>(t[a]);
      });
    });
    static_for<0, A>([&](auto ki) { Dft<B, INV, FINE>::run(v + B * decltype(ki)::value); });
    float2 o[R];
    static_for<0, A>([&](auto k1i) {
      static_for<0, B>([&](auto k2i) {
        constexpr int k1 = decltype(k1i)::value, k2 = decltype(k2i)::value;
        o[k1 + A * k2] = v[B * k1 + k2];
      });
    });
    static_for<0, R>([&](auto i) { v[decltype(i)::value] = o[decltype(i)::value]; });
  }
};

template <bool INV, bool FINE>
struct Dft<1, INV, FINE> {
  __host__ __device__ __forceinline__ static void run(float2*) {}
};

template <bool INV, bool FINE>
struct Dft<2, INV, FINE> {
  __host__ __device__ __forceinline__ static void run(float2* v) {
    float2 a = v[0], b = v[1];
    v[0] = c_add(a, b);
    v[1] = c_sub(a, b);
  }
};

template <bool INV, bool FINE>
struct Dft<3, INV, FINE> {
  __host__ __device__ __forceinline__ static void run(float2* v) {
    // sqrt(3)/2 as a pair of floats: the error of one, 1.6e-8, is the same in
    // every transform of every step and adds up (whole-field phasors of
    // 144x180x192 2.0e-6 -> 1.4e-6 from 64 bits)
    const float h = 0.86602540378443864676f, hl = (float)(0.86602540378443864676 - (double)h);
    float2 t = c_add(v[1], v[2]);
    float2 d = c_sub(v[1], v[2]);
    float2 m = c_fma(t, -0.5f, v[0]);
    float2 r = rot<INV>(c_fma(d, h, c_scale(d, hl)));
    v[0] = c_add(v[0], t);
    v[1] = c_add(m, r);
    v[2] = c_sub(m, r);
  }
};

template <bool INV, bool FINE>
struct Dft<4, INV, FINE> {
  __host__ __device__ __forceinline__ static void run(float2* v) {
    float2 t0 = c_add(v[0], v[2]);
    float2 t1 = c_sub(v[0], v[2]);
    float2 t2 = c_add(v[1], v[3]);
    float2 t3 = rot<INV>(c_sub(v[1], v[3]));
    v[0] = c_add(t0, t2);
    v[2] = c_sub(t0, t2);
    v[1] = c_add(t1, t3);
    v[3] = c_sub(t1, t3);
  }
};

template <bool INV, bool FINE>
struct Dft<5, INV, FINE> {
  __host__ __device__ __forceinline__ static void run(float2* v) {
    const float c1 = 0.30901699437494742410f, c2 = -0.80901699437494742410f;
    const float s1 = 0.95105651629515357212f, s2 = 0.58778525229247312917f;
    const float s1l = (float)(0.95105651629515357212 - (double)s1);
    float2 t1 = c_add(v[1], v[4]);
    float2 t2 = c_add(v[2], v[3]);
    float2 t3 = c_sub(v[1], v[4]);
    float2 t4 = c_sub(v[2], v[3]);
    float2 y0 = c_add(v[0], c_add(t1, t2));
    float2 b1 = c_fma(t2, c2, c_fma(t1, c1, v[0]));
    float2 b2 = c_fma(t2, c1, c_fma(t1, c2, v[0]));
    const float2 e1l = c_scale(t4, s2), e2l = c_scale(t3, s2);
    float2 e1 = c_fma(t3, s1, FINE ? c_fma(t3, s1l, e1l) : e1l);
    float2 e2 = c_fma(t4, -s1, FINE ? c_fma(t4, -s1l, e2l) : e2l);
    float2 r1 = rot<INV>(e1);
    float2 r2 = rot<INV>(e2);
    v[0] = y0;
    v[1] = c_add(b1, r1);
    v[4] = c_sub(b1, r1);
    v[2] = c_add(b2, r2);
    v[3] = c_sub(b2, r2);
  }
};

template <bool INV, bool FINE>
struct Dft<8, INV, FINE> {
  __host__ __device__ __forceinline__ static void run(float2* v) {
    const float r2 = 0.70710678118654752440f;
    float2 e[4] = {v[0], v[2], v[4], v[6]};
    float2 o[4] = {v[1], v[3], v[5], v[7]};
    Dft<4, INV, FINE>::run(e);
    Dft<4, INV, FINE>::run(o);
    // o[1] and o[3] without their factor r2, which the last sums apply
    o[1] = INV ? make_float2(o[1].x - o[1].y, o[1].x + o[1].y) : make_float2(o[1].x + o[1].y, o[1].y - o[1].x);
    o[2] = rot<INV>(o[2]);
    o[3] = INV ? make_float2(-(o[3].x + o[3].y), o[3].x - o[3].y) : make_float2(o[3].y - o[3].x, -(o[3].x + o[3].y));
    v[0] = c_add(e[0], o[0]);
    v[4] = c_sub(e[0], o[0]);
    v[1] = c_fma(o[1], r2, e[1]);
    v[5] = c_fma(o[1], -r2, e[1]);
    v[2] = c_add(e[2], o[2]);
    v[6] = c_sub(e[2], o[2]);
    v[3] = c_fma(o[3], r2, e[3]);
    v[7] = c_fma(o[3], -r2, e[3]);
  }
};

// ------------------------------------------------ two-level transform --
// Split of a pencil length N into (A, B): B = gcd(N, 16), A = N / B.
template <int N>
struct Split {
  static constexpr int B = ct_gcd(N, 16);
  static constexpr int A = N / B;
  static constexpr bool ok = (A <= 16);
};

// The most even split n = a b (a <= b) of a pencil; its smaller factor.
constexpr int ct_even_split(int n) {
  int best = 1;
  for (int a = 1; a * a <= n; ++a)
    if (n % a == 0) best = a;
  return best;
}

// Whether a split (a, b) is transformed in three levels: where the codelets of
// b points would leave most threads idle (a of b busy) on more than 20 values
// each, and b = c d with c and d factors of a (125, 243, 250 and 375 points: a
// step 251 -> 108 us at 125^3, 1207 -> 643 at 243^3, 3537 -> 2624 at 375^3).
constexpr int ct_three_d(int b) { return ct_even_split(b); }
constexpr bool ct_three(int a, int b) { return b > 20 && a % ct_three_d(b) == 0 && a % (b / ct_three_d(b)) == 0; }

// Whether the 5-point codelets of a split (a, b) take sin(2 pi/5) as a pair of
// floats. One float is 2.5e-8 too large, in every transform of every step; the
// twiddles inside a codelet of 8, 16 or 32 points (cos(pi/4), cos(pi/8)) are up
// to 2.9e-8 too small, and beside one of those the two make up for each other.
// Phasors from 64 bits (1e-6), pair / float: 100x125x135 0.91 / 1.9, 200^3 1.2 /
// 1.9, 125^3 1.2 / 1.9; beside 16 points 128x128x320 2.0 / 1.8, quiet phasors of
// 96x96x320 24.5 / 20.0.
constexpr bool ct_fine(int a, int b) { return a % 8 != 0 && b % 8 != 0; }

// Threads per pencil for a split whose larger factor is m: 8 or 16 (whole
// pencils per warp), else m rounded up to 4 so that 8 pencils fill whole warps.
constexpr int ct_tpp(int m) { return m <= 8 ? 8 : (m <= 16 ? 16 : (m + 3) / 4 * 4); }

// Pencil split of the size-specialised passes: (A, B) with B threads
// holding A values on input and A threads holding B values on output. The
// most even split: fewest instructions for the warp that waits on its
// longest codelet, and up to 400 points no thread holds more than 20 values
// except on 384 (24), the lengths of three levels included. Against 16 x (N / 16)
// for the multiples of 16: 64^3 33 -> 29 us a step, 96x96x128 54 -> 52,
// 32^3 25 -> 20.
template <int N>
struct PSplit {
  static constexpr int A = ct_even_split(N), B = N / A;
  static constexpr bool THREE = ct_three(A, B);
  static constexpr int OA = THREE ? B : A, OB = THREE ? A : B;  // threads and values after the transform
  static constexpr int TW = N + (THREE ? B : 0);                // entries of a twiddle table
  static constexpr int TPP = ct_tpp(A > B ? A : B);             // threads per pencil
};
template <>
struct PSplit<512> {
  static constexpr int A = 32, B = 16, OA = A, OB = B, TW = 512, TPP = 32;
  static constexpr bool THREE = false;
};
template <>
struct PSplit<640> {
  static constexpr int A = 32, B = 20, OA = A, OB = B, TW = 640, TPP = 32;
  static constexpr bool THREE = false;
};

// The split of the y-passes, whose threads read and write runs of a row: 16 x
// (N / 16) from 80 points on, for whole lines (Y_INV_GRAD on 96x96x128 9.8 us
// against 11.9 for 8 x 12), the most even one below (32^3 6.4 against 7.8).
template <int N>
struct YSplit {
  static constexpr bool LINES = N % 16 == 0 && N > 64 && N <= 256;
  static constexpr int A = LINES ? N / 16 : PSplit<N>::A, B = N / A;
  static constexpr int OA = LINES ? A : PSplit<N>::OA, OB = N / OA, TW = PSplit<N>::TW;
  static constexpr int TPP = ct_tpp(A > B ? A : B);
};

// Odd leading dimension >= n (bank-conflict-free strided access).
constexpr int ct_odd(int n) { return (n % 2) ? n : n + 1; }

// Exchange-buffer indexers. Row tiles: 16 pencils along threadIdx / 16, the
// within-pencil index s along the lanes. Column tiles: pencils along the
// lanes (threadIdx % 16).
// WARP: every thread of the pencil sits in one warp (threads per pencil
// divide 32 and pencils are consecutive in threadIdx), so the exchange of a
// pencil's own slab needs only a warp barrier. Hazards between pencils
// (staging buffers shared by a whole tile) keep their block barriers.
template <int A, int B, bool WARP = false>
struct RowEx {
  float2* base;  // this pencil's slab
  static constexpr int LD = ct_odd(B);
  static constexpr int SLAB = A * LD;
  static constexpr bool kWarp = WARP;
  __device__ __forceinline__ float2& at(int k1, int n2) const { return base[k1 * LD + n2]; }
};

template <int A, int B, int P = 16>
struct ColEx {
  float2* base;  // + lane pencil
  // below 16 columns a row is part of the banks: an odd row count puts the rows
  // s and s + 1 that a warp reads together on different ones
  static constexpr int LD = P < 16 ? ct_odd(B) : B;
  static constexpr int SLAB = A * LD * P;
  static constexpr bool kWarp = false;  // a column pencil spans the whole block
  __device__ __forceinline__ float2& at(int k1, int n2) const { return base[(k1 * LD + n2) * P]; }
};

template <class Ex>
__device__ __forceinline__ void ex_sync() {
  if constexpr (Ex::kWarp)
    __syncwarp();
  else
    __syncthreads();
}

// Twiddle table of an (A, B) transform in the order the threads read it:
// twt[k1 * B + s] = exp(-2 pi i s k1 / N) (lanes run over s: conflict free);
// behind it, for a three-level transform (R != B values per thread after it),
// exp(-2 pi i m / B).
template <int A, int B, int R = B>
__device__ __forceinline__ void fill_twt(float2* twt, const float2* __restrict__ tw_lin) {
  for (int i = threadIdx.x; i < A * B; i += blockDim.x) {
    const int k1 = i / B, s = i - k1 * B;
    twt[i] = tw_lin[s * k1];
  }
  if constexpr (R != B)
    for (int i = threadIdx.x; i < B; i += blockDim.x) twt[A * B + i] = tw_lin[A * i];
}

// Three-level transform of one pencil of V T points, T = C D: thread s (< T)
// holds v[a] = x[s + T a] before and w[a] = X[s + T a] after it. Level 1: V
// points per thread; level 2: C points of every (k1, d), each thread V / C of
// them, in the slots it read; level 3: D points of every m = k1 + V kc, m = s +
// T j. All T threads work in every level and hold V values.
template <int V, int T, bool INV, class Ex>
__device__ __forceinline__ void fft3(const float2 (&v_in)[V], float2 (&w)[V], int s, const float2* __restrict__ twt,
                                     const Ex& ex) {
  constexpr int D = ct_three_d(T), C = T / D, JC = V / C, JD = V / D;
  constexpr bool FINE = ct_fine(V, T);
  if (s < T) {
    float2 v[V];
    static_for<0, V>([&](auto i) { v[decltype(i)::value] = v_in[decltype(i)::value]; });
    Dft<V, INV, FINE>::run(v);
    static_for<0, V>([&](auto ki) {
      constexpr int k1 = decltype(ki)::value;
      float2 y = v[k1];
      if constexpr (k1 > 0) {
        float2 t = twt[k1 * T + s];
        if (INV) t.y = -t.y;
        y = c_mul(y, t);
      }
      ex.at(k1, s) = y;
    });
  }
  ex_sync<Ex>();
  if (s < T) {
    const int d = s % D, k0 = s / D;
    static_for<0, JC>([&](auto ji) {
      const int k1 = k0 + C * decltype(ji)::value;
      float2 q[C];
      static_for<0, C>([&](auto ci) { q[decltype(ci)::value] = ex.at(k1, D * decltype(ci)::value + d); });
      Dft<C, INV, FINE>::run(q);
      static_for<0, C>([&](auto ki) {
        constexpr int kc = decltype(ki)::value;
        if constexpr (kc > 0) {
          float2 t = twt[V * T + d * kc];
          if (INV) t.y = -t.y;
          q[kc] = c_mul(q[kc], t);
        }
        ex.at(k1, D * kc + d) = q[kc];
      });
    });
  }
  ex_sync<Ex>();
  if (s < T) {
    static_for<0, JD>([&](auto ji) {
      constexpr int j = decltype(ji)::value;
      const int m = s + T * j, kc = m / V, k1 = m - V * kc;
      float2 q[D];
      static_for<0, D>([&](auto di) { q[decltype(di)::value] = ex.at(k1, D * kc + decltype(di)::value); });
      Dft<D, INV, FINE>::run(q);
      static_for<0, D>([&](auto ki) { w[j + JD * decltype(ki)::value] = q[decltype(ki)::value]; });
    });
  }
  ex_sync<Ex>();
}

// (A, B) transform of one pencil: thread s (< B) holds v[a] = x[s + B a];
// afterwards thread s (< A) holds w[b] = X[s + A b], or, in three levels, s (<
// B) w[a] = X[s + B a]. `twt` is the table laid out by fill_twt, or (TR) that of
// the (B, A) transform. Every thread of the block calls it.
template <int A, int B, bool INV, bool TR = false, class Ex, int R>
__device__ __forceinline__ void fft2(const float2 (&v_in)[A], float2 (&w)[R], int s, const float2* __restrict__ twt,
                                     const Ex& ex) {
  if constexpr (R != B) {
    fft3<A, B, INV>(v_in, w, s, twt, ex);
    return;
  } else {
    constexpr bool FINE = ct_fine(A, B);
    if (s < B) {
      float2 v[A];
      static_for<0, A>([&](auto i) { v[decltype(i)::value] = v_in[decltype(i)::value]; });
      Dft<A, INV, FINE>::run(v);
      static_for<0, A>([&](auto ki) {
        constexpr int k1 = decltype(ki)::value;
        float2 y = v[k1];
        if constexpr (k1 > 0) {
          float2 t = twt[TR ? s * A + k1 : k1 * B + s];
          if (INV) t.y = -t.y;
          y = c_mul(y, t);
        }
        ex.at(k1, s) = y;
      });
    }
    ex_sync<Ex>();
    if (s < A) {
      static_for<0, B>([&](auto bi) { w[decltype(bi)::value] = ex.at(s, decltype(bi)::value); });
      Dft<B, INV, FINE>::run(w);
    }
    ex_sync<Ex>();
  }
}

// Asynchronous 16-byte global -> shared copy (L2 only), completed by
// cp_async_wait0 and made visible to the block by a following barrier.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Tensor-map (TMA) copies completed on a shared-memory mbarrier. One thread
// arms the barrier with the byte count it expects and issues the copies;
// every consumer waits on the barrier's phase parity.
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
// makes the initialised barriers visible to the asynchronous (TMA) proxy
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory"); }
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Waits for the phase with the given parity, giving up after `limit` polls
// (each poll may suspend the thread for a short while); false when it gave up.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity, int limit = 1 << 20) {
  for (int i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
// generic-proxy accesses of this thread before asynchronous-proxy ones after
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }
// A 3-D box of the tensor map at `map` (global memory) into shared memory at
// `dst` (aligned to the swizzle span), counted on `bar`.
__device__ __forceinline__ void tma_load_3d(void* dst, const void* map, unsigned long long* bar, int c0, int c1,
                                            int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];\n" ::"r"(smem_addr(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_addr(bar))
      : "memory");
}

// Contiguous copies between global and shared memory (16-byte aligned, sizes a
// multiple of 16): a load counted on bar, a store as one bulk group of the
// issuing thread, and the waits for its groups to have read shared memory or
// to be complete.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, const void* src, unsigned bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(dst), "r"(smem_addr(src)),
               "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory"); }
__device__ __forceinline__ void bulk_wait() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }

// A value that this pass reads once, kept out of the L1 and in program order.
__device__ __forceinline__ float2 ld_once(const float2* p) {
  float2 v;
  asm volatile("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}

// A read-only value, loaded in program order.
__device__ __forceinline__ float ld_ordered(const float* p) {
  float v;
  asm volatile("ld.global.nc.f32 %0, [%1];\n" : "=f"(v) : "l"(p) : "memory");
  return v;
}

// Starts the fetch of the line that holds *p into the L2.
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p)); }

// Programmatic dependent launch: a pass lets the next one launch as soon as
// all of its own CTAs are running (pdl_trigger), and waits for the previous
// pass to complete and its writes to be visible (pdl_wait) before its first
// access to any field or spectrum; only constant tables are read before.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// Whether a handle's launches are programmatic: unless CG_PDL=0 when it is created.
inline int pdl_default() {
  const char* e = getenv("CG_PDL");
  return (e && e[0] == '0') ? 0 : 1;
}
// Launch, with programmatic stream serialisation when `pdl` is set.
template <typename... KArgs, typename... Args>
inline void launch(int pdl, void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = pdl ? 1 : 0;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k, args...);
}

// SM count of the current device (cached; 152 on GB300 if the query fails).
inline int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        n < 1)
      n = 152;
  }
  return n;
}

}  // namespace cgf
