// Size-specialised y- and x-passes (axis length N known at compile time):
// kernels and per-length launchers. The launchers are instantiated by the
// cg_fast_yx_*.cu units (a few lengths each, so they compile in parallel)
// and dispatched by cg_fast_yx.cu.
//
// y-pass: rows (x, kz) of length ny, YP rows per CTA; thread (p, s) =
// (threadIdx / TPP, threadIdx % TPP) owns row p (TPP = threads per pencil: 8
// or 16, or 20..32 for the longer splits). x-pass: XP
// consecutive (kz, y) columns per CTA; thread (c, s) = (threadIdx % XP,
// threadIdx / XP) owns column c. Pencil data moves global -> registers -> one exchange per
// transform -> registers -> global (cg_fast.cuh).
#pragma once

#include "cg_fast.cuh"
#include "cg_kspace.cuh"

// resident CTAs per SM the register allocation targets (y: 4-row CTAs,
// ~102 registers per thread, no spills; x: 16-column CTAs, ~85 registers;
// both measured best on a 192^2 x 256 grid)
#ifndef CG_FAST_MINB_Y
#define CG_FAST_MINB_Y 10
#endif
#ifndef CG_FAST_MINB_X
#define CG_FAST_MINB_X 3
#endif
// the same for the x-pass modes other than X_DIV (the divergence pass parks
// a spectrum tile and needs the larger register budget)
#ifndef CG_FAST_MINB_XG
#define CG_FAST_MINB_XG CG_FAST_MINB_X
#endif
#ifndef CG_XP20
#define CG_XP20 8
#endif
// rows per y-CTA and columns per x-CTA (16 threads each)
#ifndef CG_YP20
#define CG_YP20 4  // rows per y-CTA on 20-thread pencils
#endif
#ifndef CG_YP
#define CG_YP 4
#endif
#ifndef CG_XP
#define CG_XP 16
#endif

using cgf::ColEx;
using cgf::PSplit;
using cgf::YSplit;
using cgf::RowEx;
using cgf::fft2;
using cgf::static_for;

// Threads and resident CTAs per SM of the y- and x-pass CTAs for length N.
// Splits with more than 16 threads a pencil take 8 columns per x-CTA, three
// CTAs to an SM, or four where no thread holds more than 16 and 20 values
// (X_GRAD / X_DIV us with four / three: 216^3 57 / 55 against 66 / 64, 320^3
// 155 / 166 against 176 / 166, 400^3 323 / 333 against 297 / 302; with two,
// 400^3 348 / 345), and five y-CTAs, or six up to 34 values (Y_INV_GRAD /
// Y_FWD_DIV with six / five: 288^3 106 / 109 against 107 / 129, 320^3 146 / 144
// against 129 / 133). Three-level pencils: four x- and eight y-CTAs up to ten
// values a thread, three and six above (250^3 with 4, 8 / 3, 6 / 2, 4 CTAs:
// X_GRAD 78 / 86 / 107, Y_INV_GRAD 81 / 82 / 88; 375^3 308 / 293 / 316 and 321 /
// 287 / 291).
template <int N>
struct YT {
  static constexpr int TPP = YSplit<N>::TPP, YP = TPP < 16 ? 2 * CG_YP : (TPP > 16 && TPP < 32 ? CG_YP20 : CG_YP);
  static constexpr int THREADS = TPP * YP;
  static constexpr int SUM = YSplit<N>::A + YSplit<N>::B, VALS = YSplit<N>::A;
  static constexpr bool THREE = PSplit<N>::THREE && !YSplit<N>::LINES;
  static constexpr int MINB = TPP <= 16 ? CG_FAST_MINB_Y : (TPP < 28 ? (SUM <= 34 ? 6 : 5) : (THREE ? (VALS <= 10 ? 8 : 6) : 4));
};
template <int N>
struct XT {
  static constexpr int TPP = PSplit<N>::TPP, XP = TPP > 16 ? CG_XP20 : CG_XP, THREADS = TPP * XP;
  using S = PSplit<N>;
  static constexpr int EX_F = ColEx<S::A, S::B, XP>::SLAB, EX_I = ColEx<S::OB, S::OA, XP>::SLAB;
  static constexpr int EX = EX_F > EX_I ? EX_F : EX_I;  // the exchange tile
  // the (OB, OA) twiddles: the (A, B) ones where the two orders are the same, or
  // read across (TR) unless the few rows s of a warp then share their banks
  // (with padded exchange rows, X_GRAD / X_DIV us: 400^3 285 / 294 -> 266 / 275,
  // 324^3 173 / 174 -> 162 / 164, 144x180x192 25.4 / 26.6 -> 25.0 / 24.6)
  static constexpr bool TR = S::A != S::OB && S::OB % 16 != 0;
  static constexpr int TABLES = S::A == S::OB || TR ? 1 : 2;
  // X_GRAD loops over one copy of its inverse transform, whose 32-value codelets
  // are long: two copies / one, 512x128x128 62 / 49 us, 640x128x128 76 / 65, 512^3
  // 709 / 603
  static constexpr bool LOOP = TPP == 32;
  static constexpr int minb(int mode) {
    if (TPP <= 16) return 16 / TPP * (mode != X_DIV ? CG_FAST_MINB_XG : CG_FAST_MINB_X);
    if (PSplit<N>::THREE) return PSplit<N>::A <= 10 ? 4 : 3;
    return TPP < 28 ? (PSplit<N>::A <= 16 && TPP == 20 ? 4 : 3) : 2;
  }
};

// One instantiation per mode keeps each kernel's code small enough for the
// instruction cache; the modes stay straight-line, where the compiler hoists
// the next input's loads above the current transform.
template <int N, int MODE>
__global__ void __launch_bounds__(YT<N>::THREADS, YT<N>::MINB) kf_ypass(Dims d, Tables t, float2* __restrict__ S0,
                                                                        float2* __restrict__ S1,
                                                                        float2* __restrict__ S2) {
  constexpr int A = YSplit<N>::A, B = YSplit<N>::B, OA = YSplit<N>::OA, OB = YSplit<N>::OB, TW = YSplit<N>::TW,
                TPP = YSplit<N>::TPP;
  using Ex = RowEx<A, B, (32 % TPP == 0)>;  // pencil-local exchange: warp barriers
  extern __shared__ float2 sm[];
  cgf::pdl_trigger();
  float2* tw = sm;  // (A, B) order
  // The first row loads while the twiddles are put in place (us, row first /
  // tables first: 400^3 Y_FWD 88 / 92, Y_INV_GRAD 221 / 227, 160x160x192 x 8
  // Y_FWD_DIV 129 / 134; a 100x125x135 step 94 / 99). Tables first, before the wait
  // for the pass before, where that pass is an x-pass and this one is launched
  // programmatically (y_pdl; 192x192x256 274.6 us a step against 276.3) and on
  // the smallest grids (64^3 27.6 against 29.3).
  constexpr bool FIRST = TPP > 16 || (TPP == 16 && (MODE == Y_FWD || MODE == Y_FWD_DIV || N > 192));
  if (!FIRST) cgf::fill_twt<A, B, OB>(tw, t.twy);
  cgf::pdl_wait();
  const int s = threadIdx.x % TPP, p = threadIdx.x / TPP;
  const Ex ex{sm + TW + p * Ex::SLAB};
  const long long nrows = (long long)d.nx * d.nzh;
  const long long row = (long long)blockIdx.x * YT<N>::YP + p;
  const bool valid = row < nrows;
  const long long off = (long long)blockIdx.y * d.nspec + row * N;
  float2 v[A], w[OB];
  auto load = [&](const float2* __restrict__ src) {
    static_for<0, A>([&](auto ai) {
      constexpr int a = decltype(ai)::value;
      v[a] = (valid && s < B) ? src[off + s + B * a] : make_float2(0.f, 0.f);
    });
  };
  auto store = [&](float2* __restrict__ dst) {
    if (valid && s < OA) static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      dst[off + s + OA * b] = w[b];
    });
  };
  if (!FIRST) __syncthreads();
  load(MODE == Y_FWD || MODE == Y_INV ? S0 : S1);
  if (FIRST) {
    cgf::fill_twt<A, B, OB>(tw, t.twy);
    __syncthreads();
  }
  if constexpr (MODE == Y_FWD || MODE == Y_INV) {
    fft2<A, B, MODE == Y_INV>(v, w, s, tw, ex);
    store(S0);
  } else if constexpr (MODE == Y_INV_GRAD) {
    // S1 <- IFFT(S1); S0 <- IFFT(i ky S2); S2 <- IFFT(S2)
    fft2<A, B, true>(v, w, s, tw, ex);
    store(S1);
    load(S2);
    float2 g[A];
    static_for<0, A>([&](auto ai) {
      constexpr int a = decltype(ai)::value;
      const float k = (s < B) ? t.ky[s + B * a] : 0.f;
      g[a] = c_muli(c_scale(v[a], k));
    });
    fft2<A, B, true>(g, w, s, tw, ex);
    store(S0);
    fft2<A, B, true>(v, w, s, tw, ex);
    store(S2);
  } else {
    // Y_FWD_DIV: S1 <- FFT(S1); S0 <- i ky FFT(S0) + FFT(S2)
    fft2<A, B, false>(v, w, s, tw, ex);
    store(S1);
    load(S0);
    fft2<A, B, false>(v, w, s, tw, ex);
    float2 h[OB];
    static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const float k = (s < OA) ? t.ky[s + OA * b] : 0.f;
      h[b] = c_muli(c_scale(w[b], k));
    });
    load(S2);
    fft2<A, B, false>(v, w, s, tw, ex);
    static_for<0, OB>([&](auto bi) { w[decltype(bi)::value] = c_add(w[decltype(bi)::value], h[decltype(bi)::value]); });
    store(S0);
  }
}

// The transverse chain of a grid of one x plane (2-D), where the x-transforms
// are the identity and k_x = 0: Y_FWD, X_GRAD, Y_INV_GRAD in one kernel
// (DIV = false: S0 <- IFFT(i ky q), S2 <- IFFT(q), S1 <- 0 q, q = kappa/N
// FFT(S0)) or Y_FWD_DIV, X_DIV, Y_INV (S0 <- IFFT(kappa/N (i ky FFT(S0) +
// FFT(S2 + 0 S1)))). The zero multiples carry a non-finite u_x or p over, as
// the products with k_x = 0 do. Bound: launch latency (a 135x192 step takes
// 34 us in eight launches, the arithmetic of one fits in two); four launches a
// step take 28 us. Rows as in the y-pass.
template <int N, bool DIV>
__global__ void __launch_bounds__(YT<N>::THREADS, 4) kf_plane(Dims d, Tables t, float kcoef, float invN,
                                                              float2* __restrict__ S0, float2* __restrict__ S1,
                                                              float2* __restrict__ S2) {
  constexpr int A = YSplit<N>::A, B = YSplit<N>::B, OA = YSplit<N>::OA, OB = YSplit<N>::OB, TW = YSplit<N>::TW,
                TPP = YSplit<N>::TPP;
  using ExF = RowEx<A, B, (32 % TPP == 0)>;
  using ExI = RowEx<OB, OA, (32 % TPP == 0)>;
  constexpr int SLAB = ExF::SLAB > ExI::SLAB ? ExF::SLAB : ExI::SLAB;
  extern __shared__ float2 sm[];
  cgf::pdl_trigger();
  float2* tw = sm;        // (A, B) order
  float2* twi = sm + TW;  // (OB, OA) order
  cgf::fill_twt<A, B, OB>(tw, t.twy);
  cgf::fill_twt<OB, OA, A>(twi, t.twy);
  // k_y | k_y^2, ready before the wait: a 135x192 step 32.7 -> 27.9 us, 64x96 16.4 -> 13.7
  float* kys = reinterpret_cast<float*>(sm + 2 * TW + YT<N>::YP * SLAB);
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    kys[i] = t.ky[i];
    kys[N + i] = t.ky2[i];
  }
  const int s = threadIdx.x % TPP, p = threadIdx.x / TPP;
  const ExF exf{sm + 2 * TW + p * SLAB};
  const ExI exi{sm + 2 * TW + p * SLAB};
  const int row = blockIdx.x * YT<N>::YP + p;  // kz
  const bool valid = row < d.nzh;
  const long long off = (long long)blockIdx.y * d.nspec + (long long)row * N;
  const float kz2 = valid ? t.kz2[row] : 0.f;
  cgf::pdl_wait();
  __syncthreads();
  float2 v[A], w[OB], z[A];
  auto load = [&](const float2* src) {
    static_for<0, A>([&](auto ai) {
      constexpr int a = decltype(ai)::value;
      v[a] = (valid && s < B) ? src[off + s + B * a] : make_float2(0.f, 0.f);
    });
  };
  auto store_z = [&](float2* dst) {
    if (valid && s < B) static_for<0, A>([&](auto ai) {
      constexpr int a = decltype(ai)::value;
      dst[off + s + B * a] = z[a];
    });
  };
  auto kappa = [&](int k) { return sinc_a2(kcoef * (kys[N + k] + kz2)) * invN; };
  if constexpr (!DIV) {
    load(S0);
    fft2<A, B, false>(v, w, s, tw, exf);
    float2 g[OB];
    static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int k = (s < OA) ? s + OA * b : 0;
      w[b] = c_scale(w[b], kappa(k));
      g[b] = c_muli(c_scale(w[b], kys[k]));
    });
    fft2<OB, OA, true>(g, z, s, twi, exi);
    store_z(S0);
    fft2<OB, OA, true>(w, z, s, twi, exi);
    store_z(S2);
    static_for<0, A>([&](auto ai) { z[decltype(ai)::value] = c_scale(z[decltype(ai)::value], 0.f); });
    store_z(S1);
  } else {
    load(S0);
    fft2<A, B, false>(v, w, s, tw, exf);
    float2 h[OB];
    static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int k = (s < OA) ? s + OA * b : 0;
      h[b] = c_muli(c_scale(w[b], kys[k]));
    });
    load(S2);
    static_for<0, A>([&](auto ai) {
      constexpr int a = decltype(ai)::value;
      if (valid && s < B) v[a] = c_add(v[a], c_scale(S1[off + s + B * a], 0.f));
    });
    fft2<A, B, false>(v, w, s, tw, exf);
    static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int k = (s < OA) ? s + OA * b : 0;
      w[b] = c_scale(c_add(w[b], h[b]), kappa(k));
    });
    fft2<OB, OA, true>(w, z, s, twi, exi);
    store_z(S0);
  }
}

template <int N>
static size_t smem_plane() {
  using F = RowEx<YSplit<N>::A, YSplit<N>::B>;
  using I = RowEx<YSplit<N>::OB, YSplit<N>::OA>;
  return sizeof(float2) * (2 * YSplit<N>::TW + YT<N>::YP * (F::SLAB > I::SLAB ? F::SLAB : I::SLAB)) +
         2 * sizeof(float) * N;  // + k_y, k_y^2
}

template <int N, int MODE>
__global__ void __launch_bounds__(XT<N>::THREADS, XT<N>::minb(MODE)) kf_xpass(Dims d, Tables t, float kcoef, float invN,
                                                                        float2* __restrict__ S0,
                                                                        float2* __restrict__ S1,
                                                                        float2* __restrict__ S2) {
  constexpr int A = PSplit<N>::A, B = PSplit<N>::B, OA = PSplit<N>::OA, OB = PSplit<N>::OB, TW = PSplit<N>::TW,
                XP = XT<N>::XP;
  extern __shared__ float2 sm[];
  cgf::pdl_trigger();
  constexpr bool TR = XT<N>::TR;
  constexpr int XB = XT<N>::TABLES * TW;  // behind the twiddles
  float2* tw = sm;                        // (A, B) order
  float2* twi = sm + (XB - TW);           // (OB, OA) order, or the one table
  float* kxs = reinterpret_cast<float*>(sm + XB + XT<N>::EX + N * XP);  // k_x | k_x^2
  cgf::fill_twt<A, B, OB>(tw, t.twx);
  if (XT<N>::TABLES == 2) cgf::fill_twt<OB, OA, A>(twi, t.twx);
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    kxs[i] = t.kx[i];
    kxs[N + i] = t.kx2[i];
  }
  cgf::pdl_wait();
  const int c = threadIdx.x % XP, s = threadIdx.x / XP;
  const ColEx<A, B, XP> exf{sm + XB + c};
  const ColEx<OB, OA, XP> exi{sm + XB + c};
  const long long ncol = (long long)d.nzh * d.ny;
  const long long col = (long long)blockIdx.x * XP + c;
  const bool valid = col < ncol;
  const long long base = (long long)blockIdx.y * d.nspec + col;
  float kyz2 = 0.f;
  {
    const unsigned cc = (unsigned)(valid ? col : ncol - 1);  // below 2^21: 32-bit division
    const int kz = (int)(cc / (unsigned)d.ny);
    const int ky = (int)(cc - (unsigned)kz * (unsigned)d.ny);
    kyz2 = t.ky2[ky] + t.kz2[kz];
  }
  float2 v[A], w[OB], z[A];
  auto load = [&](const float2* __restrict__ src) {
    static_for<0, A>([&](auto ai) {
      constexpr int a = decltype(ai)::value;
      const float2* g = src + (base + (long long)(s + B * a) * ncol);
      // in program order (X_GRAD / X_DIV us, plain against ordered: 192x192x256 41 /
      // 41 -> 39 / 39, 240^3 58 / 70 -> 55 / 59, 384^3 269 / 304 -> 267 / 282): the
      // compiler otherwise starts the divergence pass's second tile under the
      // first transform. It spills either way (X_DIV ordered, 192 / 240 points:
      // 44 / 92 bytes). 20 threads a pencil do better plain: 400^3 309 / 290 against
      // 309 / 298
      if constexpr (PSplit<N>::TPP == 20)
        v[a] = (valid && s < B) ? *g : make_float2(0.f, 0.f);
      else
        v[a] = (valid && s < B) ? cgf::ld_once(g) : make_float2(0.f, 0.f);
    });
  };
  // after an inverse (OB, OA) transform thread s < B owns z[a] = element s + B a
  auto store_z = [&](float2* __restrict__ dst) {
    if (valid && s < B) static_for<0, A>([&](auto ai) {
      constexpr int a = decltype(ai)::value;
      dst[base + (long long)(s + B * a) * ncol] = z[a];
    });
  };
  auto kappa = [&](int k) { return sinc_a2(kcoef * (kxs[N + k] + kyz2)) * invN; };
  // above 16 threads a pencil the first tile's loads need not wait for the tables
  if (XT<N>::TPP <= 16) __syncthreads();
  load(MODE == X_GRAD ? S0 : S1);
  if (XT<N>::TPP > 16) __syncthreads();
  if constexpr (MODE == X_GRAD) {
    // S2 <- IFFT(q); S1 <- IFFT(i kx q), q = kappa/N FFT(S0); q waits in shared
    // memory during the first inverse transform instead of in registers
    float2* qs = sm + XB + XT<N>::EX;
    fft2<A, B, false>(v, w, s, tw, exf);
    static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int k = (s < OA) ? s + OA * b : 0;
      w[b] = c_scale(w[b], kappa(k));
      if (s < OA) qs[(s + OA * b) * XP + c] = w[b];
    });
    auto times_ikx = [&]() {
      static_for<0, OB>([&](auto bi) {
        constexpr int b = decltype(bi)::value;
        const int k = (s < OA) ? s + OA * b : 0;
        w[b] = (s < OA) ? c_muli(c_scale(qs[(s + OA * b) * XP + c], kxs[k])) : make_float2(0.f, 0.f);
      });
    };
    if constexpr (XT<N>::LOOP) {
#pragma unroll 1
      for (int i = 0; i < 2; ++i) {
        if (i) times_ikx();
        fft2<OB, OA, true, TR>(w, z, s, twi, exi);
        store_z(i ? S1 : S2);
      }
    } else {
      fft2<OB, OA, true, TR>(w, z, s, twi, exi);
      store_z(S2);
      times_ikx();
      fft2<OB, OA, true, TR>(w, z, s, twi, exi);
      store_z(S1);
    }
  } else {
    // X_DIV: S0 <- IFFT(kappa/N (FFT(S0) + i kx FFT(S1))); FFT(S1) waits in shared memory
    float2* hs = sm + XB + XT<N>::EX;
    fft2<A, B, false>(v, w, s, tw, exf);
    if (s < OA) static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      hs[(s + OA * b) * XP + c] = w[b];
    });
    load(S0);
    fft2<A, B, false>(v, w, s, tw, exf);
    static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int k = (s < OA) ? s + OA * b : 0;
      const float2 h = (s < OA) ? hs[(s + OA * b) * XP + c] : make_float2(0.f, 0.f);
      w[b] = c_scale(c_add(w[b], c_muli(c_scale(h, kxs[k]))), kappa(k));
    });
    fft2<OB, OA, true, TR>(w, z, s, twi, exi);
    store_z(S0);
  }
}

// The x-transform alone: dst <- (I)FFT(src). src may be dst (a column is read
// whole before any of it is written), so neither is __restrict__.
template <int N, bool INV>
__global__ void __launch_bounds__(XT<N>::THREADS, XT<N>::minb(X_FWD)) kf_xhalf(Dims d, Tables t, const float2* src,
                                                                           float2* dst) {
  constexpr int A = PSplit<N>::A, B = PSplit<N>::B, OA = PSplit<N>::OA, OB = PSplit<N>::OB, XP = XT<N>::XP;
  extern __shared__ float2 sm[];
  cgf::pdl_trigger();
  cgf::fill_twt<A, B, OB>(sm, t.twx);  // (A, B) order
  cgf::pdl_wait();
  const int c = threadIdx.x % XP, s = threadIdx.x / XP;
  const ColEx<A, B, XP> ex{sm + PSplit<N>::TW + c};
  const long long ncol = (long long)d.nzh * d.ny;
  const long long col = (long long)blockIdx.x * XP + c;
  const bool valid = col < ncol;
  const long long base = (long long)blockIdx.y * d.nspec + col;
  if (XT<N>::TPP <= 16) __syncthreads();
  float2 v[A], w[OB];
  static_for<0, A>([&](auto ai) {
    constexpr int a = decltype(ai)::value;
    const float2* g = src + (base + (long long)(s + B * a) * ncol);
    if constexpr (XT<N>::TPP == 20)  // as in kf_xpass
      v[a] = (valid && s < B) ? *g : make_float2(0.f, 0.f);
    else
      v[a] = (valid && s < B) ? cgf::ld_once(g) : make_float2(0.f, 0.f);
  });
  if (XT<N>::TPP > 16) __syncthreads();
  fft2<A, B, INV>(v, w, s, sm, ex);
  if (valid && s < OA) static_for<0, OB>([&](auto bi) {
    constexpr int b = decltype(bi)::value;
    dst[base + (long long)(s + OA * b) * ncol] = w[b];
  });
}

// twiddles | exchange | (x: a parked spectrum tile, k_x, k_x^2)
template <int N>
static size_t smem_y() {
  return sizeof(float2) * (YSplit<N>::TW + YT<N>::YP * RowEx<YSplit<N>::A, YSplit<N>::B>::SLAB);
}
template <int N>
static size_t smem_x() {
  return sizeof(float2) * (XT<N>::TABLES * PSplit<N>::TW + XT<N>::EX + (size_t)N * XT<N>::XP) + 2 * sizeof(float) * N;  // + parked tile, k_x, k_x^2
}
template <int N>
static size_t smem_xhalf() {
  return sizeof(float2) * (PSplit<N>::TW + ColEx<PSplit<N>::A, PSplit<N>::B, XT<N>::XP>::SLAB);
}

// ------------------------------------------------ per-length launchers --
// Programmatic dependent launch of the y-passes. Not after a z-pass: a y-pass
// that starts while CTAs of a z-pass are still resident runs on the
// shared-memory carve-out of that pass, because an SM changes it only when
// empty, and the y-pass wants the L1 for its loads in flight. Per step with all
// passes / x and z only / none launched programmatically: 64^3 41 / 33 / 42 us,
// 160x160x192 161 / 162 / 170, 160x160x192 x 2 349 / 311 / 315, 240^3
// 480 / 438 / 446, 256x256x320 727 / 671 / 675. After an x-pass (the inverse
// y-passes) where 16-thread x-CTAs leave 64 KB of L1 (nx <= 192) and the grid
// is not so small that waiting CTAs delay the x-pass: with / without, 192x192x256
// 279 / 282 us, 128x128x160 96 / 100, 96x96x128 54 / 54, 64^3 36 / 33, 240^3
// 471 / 444, 300^3 1126 / 1114. On more x planes up to 2^23 cells in all (the
// three spectra, 100 MB, then fit the L2): 256x256x128 253 / 298, 320x128x128 186 /
// 200, 400x128x128 238 / 254, 512x128x128 324 / 342; not above: 240x240x180 329 /
// 317, 256x192x256 387 / 371, 512x160x160 515 / 476.
static inline int y_pdl(int mode, const Dims& d, int batch) {
  if (!d.pdl || (mode != Y_INV && mode != Y_INV_GRAD) || d.ncell < (1 << 20)) return 0;
  return d.nx <= 192 || d.ncell * batch <= (1 << 23);
}

template <int N>
bool yx_launch_y(int mode, const Dims& d, const Tables& t, float2* S0, float2* S1, float2* S2, int batch,
                 cudaStream_t st) {
  const dim3 grid((unsigned)((d.nx * (long long)d.nzh + YT<N>::YP - 1) / YT<N>::YP), batch);
  const dim3 block(YT<N>::THREADS);
  switch (mode) {
    case Y_FWD: cgf::launch(y_pdl(mode, d, batch), kf_ypass<N, Y_FWD>, grid, block, smem_y<N>(), st, d, t, S0, S1, S2); break;
    case Y_INV: cgf::launch(y_pdl(mode, d, batch), kf_ypass<N, Y_INV>, grid, block, smem_y<N>(), st, d, t, S0, S1, S2); break;
    case Y_INV_GRAD: cgf::launch(y_pdl(mode, d, batch), kf_ypass<N, Y_INV_GRAD>, grid, block, smem_y<N>(), st, d, t, S0, S1, S2); break;
    default: cgf::launch(y_pdl(mode, d, batch), kf_ypass<N, Y_FWD_DIV>, grid, block, smem_y<N>(), st, d, t, S0, S1, S2); break;
  }
  return true;
}

template <int N>
bool yx_launch_x(int mode, const Dims& d, const Tables& t, float kcoef, float invN, float2* S0, float2* S1,
                 float2* S2, int batch, cudaStream_t st) {
  const dim3 grid((unsigned)(((long long)d.nzh * d.ny + XT<N>::XP - 1) / XT<N>::XP), batch);
  const dim3 block(XT<N>::THREADS);
  switch (mode) {
    case X_GRAD: cgf::launch(d.pdl, kf_xpass<N, X_GRAD>, grid, block, smem_x<N>(), st, d, t, kcoef, invN, S0, S1, S2); break;
    case X_DIV: cgf::launch(d.pdl, kf_xpass<N, X_DIV>, grid, block, smem_x<N>(), st, d, t, kcoef, invN, S0, S1, S2); break;
    case X_FWD: cgf::launch(d.pdl, kf_xhalf<N, false>, grid, block, smem_xhalf<N>(), st, d, t, (const float2*)S1, S0); break;
    default: cgf::launch(d.pdl, kf_xhalf<N, true>, grid, block, smem_xhalf<N>(), st, d, t, (const float2*)S1, S0); break;
  }
  return true;
}

template <int N>
bool plane_launch(bool div, const Dims& d, const Tables& t, float kcoef, float invN, float2* S0, float2* S1,
                  float2* S2, int batch, cudaStream_t st) {
  const dim3 grid((unsigned)((d.nzh + YT<N>::YP - 1) / YT<N>::YP), batch);
  if (div)
    cgf::launch(d.pdl, kf_plane<N, true>, grid, dim3(YT<N>::THREADS), smem_plane<N>(), st, d, t, kcoef, invN, S0, S1, S2);
  else
    cgf::launch(d.pdl, kf_plane<N, false>, grid, dim3(YT<N>::THREADS), smem_plane<N>(), st, d, t, kcoef, invN, S0, S1, S2);
  return true;
}

template <typename K>
static bool yx_allow(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
}
template <int N>
int yx_prepare() {
  const size_t sy = smem_y<N>(), sx = smem_x<N>(), sh = smem_xhalf<N>(), sp = smem_plane<N>();
  return yx_allow(kf_ypass<N, Y_FWD>, sy) && yx_allow(kf_ypass<N, Y_INV>, sy) && yx_allow(kf_ypass<N, Y_INV_GRAD>, sy) &&
                 yx_allow(kf_ypass<N, Y_FWD_DIV>, sy) && yx_allow(kf_xpass<N, X_GRAD>, sx) &&
                 yx_allow(kf_xpass<N, X_DIV>, sx) && yx_allow(kf_xhalf<N, false>, sh) &&
                 yx_allow(kf_xhalf<N, true>, sh) && yx_allow(kf_plane<N, false>, sp) && yx_allow(kf_plane<N, true>, sp)
             ? 0
             : -1;
}

#define CG_YX_INSTANTIATE(n)                                                                                   \
  template bool yx_launch_y<n>(int, const Dims&, const Tables&, float2*, float2*, float2*, int, cudaStream_t); \
  template bool yx_launch_x<n>(int, const Dims&, const Tables&, float, float, float2*, float2*, float2*, int,   \
                               cudaStream_t);                                                                  \
  template bool plane_launch<n>(bool, const Dims&, const Tables&, float, float, float2*, float2*, float2*, int,   \
                                cudaStream_t);                                                                 \
  template int yx_prepare<n>();
