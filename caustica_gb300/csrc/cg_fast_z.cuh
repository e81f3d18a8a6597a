// Size-specialised z-passes (nz = N known at compile time): kernels and
// per-length launchers. The launchers are instantiated by the cg_fast_z_*.cu
// units (a few lengths each, so they compile in parallel) and dispatched by
// cg_fast_z.cu.
//
// Tile = (batch member, x, a run of consecutive y: 32, or 16 where that lets
// more CTAs share an SM). Real rows y0+2p and y0+2p+1
// form complex pencil p (p = threadIdx / TPP, TPP = threads per pencil: 8 or
// 16, or 20..32 for the longer splits); s = threadIdx % TPP runs
// along the pencil. The inverse (complex-to-real) transform is an (A, B) fft2, the
// forward one a (B, A) fft2, so the values produced by the inverse arrive in
// exactly the registers the forward transform reads; the pointwise update
// runs in between, on cells (x, y, s + A b) with coalesced row accesses.
// Half spectra are staged through shared memory in both directions (the
// spectral layout has y fastest, the real layout z fastest).
#pragma once

#include <string.h>

#include "cg_fast.cuh"
#include "cg_kspace.cuh"

// resident CTAs per SM the register allocation targets
#ifndef CG_FAST_MINB_Z
#define CG_FAST_MINB_Z 2
#endif
#define CG_FAST_MINB CG_FAST_MINB_Z

using cgf::RowEx;
using cgf::fft2;
using cgf::static_for;

// The pencil split with the larger factor first: after the inverse (A, B)
// transform A threads hold B cells each at n = s + A b, so the pointwise
// update runs on more lanes and every row access is a run of A floats.
// Smaller factor first on 192, 240 and 320 points, for accuracy: which codelet
// is next to the field decides how the rounding of the loud part of a field
// spreads to the quiet part. Error of phasors in a quiet middle of 96x96xN (1e-6
// of their norm, mean of three fields), larger first / smaller first: 192 16.2 /
// 13.5, 240 18.2 / 16.5, 320 24.0 / 20.5; within a tenth elsewhere: 160 12.0 / 12.3,
// 180 14.3 / 13.7, 216 13.5 / 13.1, 288 18.1 / 17.3, 300 16.2 / 18.0, 360 22.6 /
// 21.1, 384 21.2 / 22.9. It costs 160x160x192 x 8 1141 -> 1160 us a step,
// 192x192x320 370 -> 383 (128x128x240 137 -> 135).
template <int N>
struct ZSplit {
  using P = cgf::PSplit<N>;
  static constexpr bool SWAP = !P::THREE && P::A < P::B && N != 192 && N != 240 && N != 320;
  static constexpr int A = SWAP ? P::B : P::A, B = SWAP ? P::A : P::B;
  static constexpr int OA = SWAP ? P::OB : P::OA, OB = SWAP ? P::OA : P::OB, TW = P::TW;
  // three-level pencils fill a warp each, so that their three exchanges wait for
  // no other pencil (u-/p-pass us, 32 / 28 threads a pencil, two CTAs to an SM:
  // 250^3 242 / 95 against 254 / 103, 375^3 941 / 385 against 1303 / 667; three
  // CTAs of 32: 255 / 99, 1254 / 607)
  static constexpr int TPP = P::THREE ? 32 : P::TPP;
};

template <int N>
struct ZShape {
  static constexpr int A = ZSplit<N>::A, B = ZSplit<N>::B, OA = ZSplit<N>::OA, OB = ZSplit<N>::OB, NH = N / 2 + 1;
  static constexpr int EX_I = RowEx<A, B>::SLAB, EX_F = RowEx<OB, OA>::SLAB;
  static constexpr int EX = EX_I > EX_F ? EX_I : EX_F;
  static constexpr int STG = (NH * 34 > N * 17) ? NH * 34 : N * 17;  // float2 units
  // twiddles (two orders) | staging (aliased by xb) | exchange | material table | labels
  static constexpr size_t OFF_STG = 2 * N, OFF_EX = OFF_STG + STG, OFF_TAB = OFF_EX + (size_t)CG_TILE * EX;
  static constexpr size_t smem = sizeof(float2) * OFF_TAB + 256 * sizeof(float4) + (size_t)CG_ZROWS * N;
};

// Stage the half spectra of the tile: stg4[k * 17 + p] = (A_k, B_k) of pencil p,
// times i*mk[k] when mk is given; Im of the self-paired bins dropped.
template <int N>
__device__ __forceinline__ void z_stage(float4* stg4, const float2* __restrict__ S, const Dims& d, int x, int y0,
                                        const float* mk) {
  constexpr int NH = N / 2 + 1;
  constexpr int ITER = (NH * CG_TILE + CG_THREADS - 1) / CG_THREADS;
  const float2* base = S + (long long)x * NH * d.ny + y0;
  const bool even_ny = (d.ny & 1) == 0;
  float4 f[ITER];
  // every load of the tile is issued before the first shared-memory store
#pragma unroll
  for (int it = 0; it < ITER; ++it) {
    const int idx = threadIdx.x + it * CG_THREADS;
    const int k = idx >> 4, pp = idx & 15;
    const int ya = y0 + 2 * pp;
    const float2* q = base + (long long)k * d.ny + 2 * pp;
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (idx < NH * CG_TILE) {
      if (even_ny && ya + 1 < d.ny) {
        r = __ldg(reinterpret_cast<const float4*>(q));
      } else {
        if (ya < d.ny) {
          const float2 a = q[0];
          r.x = a.x;
          r.y = a.y;
        }
        if (ya + 1 < d.ny) {
          const float2 b = q[1];
          r.z = b.x;
          r.w = b.y;
        }
      }
    }
    f[it] = r;
  }
#pragma unroll
  for (int it = 0; it < ITER; ++it) {
    const int idx = threadIdx.x + it * CG_THREADS;
    if (idx >= NH * CG_TILE) break;
    const int k = idx >> 4, pp = idx & 15;
    float2 a = make_float2(f[it].x, f[it].y), b = make_float2(f[it].z, f[it].w);
    if (mk) {
      const float kk = mk[k];
      a = c_muli(c_scale(a, kk));
      b = c_muli(c_scale(b, kk));
    }
    if (k == 0 || 2 * k == N) {
      a.y = 0.f;
      b.y = 0.f;
    }
    stg4[k * 17 + pp] = make_float4(a.x, a.y, b.x, b.y);
  }
}

// The tile's material labels (32 rows x N bytes) and the material table in
// shared memory; returns false when the medium is dense (no labels).
template <int N>
__device__ __forceinline__ bool z_stage_labels(uint8_t* lab_s, float4* tab_s, const MediumDev& m, const Dims& d,
                                               int x, int y0) {
  if (!m.labels) return false;
  const int nyv = min(CG_ZROWS, d.ny - y0);
  const uint8_t* src = m.labels + ((long long)x * d.ny + y0) * N;
  const int nbytes = nyv * N;
  if ((N % 16) == 0) {
    const uint4* s4 = reinterpret_cast<const uint4*>(src);
    uint4* d4 = reinterpret_cast<uint4*>(lab_s);
    for (int i = threadIdx.x; i < nbytes / 16; i += blockDim.x) d4[i] = __ldg(s4 + i);
  } else {
    for (int i = threadIdx.x; i < nbytes; i += blockDim.x) lab_s[i] = src[i];
  }
  for (int i = threadIdx.x; i < 256; i += blockDim.x) tab_s[i] = m.ltab[i];
  return true;
}

// Phase-1 inputs of the inverse transform for thread (p, s): Z_n = A_n + i B_n
// with the Hermitian extension above N/2, n = s + B a.
template <int N>
__device__ __forceinline__ void z_inputs(float2 (&v)[ZSplit<N>::A], const float4* stg4, int p, int s) {
  constexpr int A = ZSplit<N>::A, B = ZSplit<N>::B;
  static_for<0, A>([&](auto ai) {
    constexpr int a = decltype(ai)::value;
    const int n = s + B * a;
    float2 z = make_float2(0.f, 0.f);
    if (s < B) {
      const bool hi = 2 * n > N;
      const float4 f = stg4[(hi ? N - n : n) * 17 + p];
      z = hi ? make_float2(f.x + f.w, f.z - f.y)   // conj(A) + i conj(B)
             : make_float2(f.x - f.w, f.y + f.z);  // A + i B
    }
    v[a] = z;
  });
}

// Slot of bin k of pencil p in the split-store buffer: rows of P pencils,
// permuted within the row so that 16 lanes holding consecutive k of one pencil
// or consecutive slots touch all banks once.
template <int P>
__device__ __forceinline__ int xb_at(int k, int p) {
  return k * P + (p ^ (P == 8 ? (k >> 1) & 7 : k & 15));
}

// After the forward transform thread (p, s < B) owns X[s + B a]; put them in
// the split-store buffer, then split each of the P pencils into its two half
// spectra and store them to S (x, k, y0 + 2p + {0, 1}), times i*mk[k] when
// given. CLOSE: a barrier after the last read of xb, for callers that write
// it again before their own next barrier.
template <int N, int P, bool CLOSE>
__device__ __forceinline__ void z_split_store(float2* xb, const float2 (&X)[ZSplit<N>::A], float2* __restrict__ S,
                                              const Dims& d, int x, int y0, int p, int s, const float* mk) {
  constexpr int A = ZSplit<N>::A, B = ZSplit<N>::B, NH = N / 2 + 1;
  // every pencil of the tile is done with the buffer (its exchange slab or
  // the staged spectrum) before any column lands in it
  __syncthreads();
  if (s < B) static_for<0, A>([&](auto ai) {
    constexpr int a = decltype(ai)::value;
    xb[xb_at<P>(s + B * a, p)] = X[a];
  });
  __syncthreads();
  float2* base = S + (long long)x * NH * d.ny + y0;
  const bool even_ny = (d.ny & 1) == 0;
  for (int idx = threadIdx.x; idx < NH * P; idx += blockDim.x) {
    const int k = idx / P, pp = idx % P;
    const int ya = y0 + 2 * pp;
    if (ya >= d.ny) continue;
    const float2 zk = xb[xb_at<P>(k, pp)];
    const float2 zm = c_conj(xb[xb_at<P>(k ? N - k : 0, pp)]);
    float2 a = c_scale(c_add(zk, zm), 0.5f);
    float2 b = c_scale(c_mulmi(c_sub(zk, zm)), 0.5f);
    if (mk) {
      a = c_muli(c_scale(a, mk[k]));
      b = c_muli(c_scale(b, mk[k]));
    }
    float2* q = base + (long long)k * d.ny + 2 * pp;
    if (even_ny && ya + 1 < d.ny) {
      *reinterpret_cast<float4*>(q) = make_float4(a.x, a.y, b.x, b.y);
    } else {
      q[0] = a;
      if (ya + 1 < d.ny) q[1] = b;
    }
  }
  if (CLOSE) __syncthreads();
}

template <int N>
__global__ void __launch_bounds__(CG_THREADS, CG_FAST_MINB) kf_zpass_u(Dims d, Tables t, MediumDev m, float* __restrict__ u,
                                                           float2* __restrict__ S0, float2* __restrict__ S1,
                                                           float2* __restrict__ S2) {
  using Z = ZShape<N>;
  constexpr int A = Z::A, B = Z::B, OA = Z::OA, OB = Z::OB;
  extern __shared__ float2 sm[];
  cgf::pdl_trigger();
  float2* tw = sm;        // (A, B) order: inverse transforms
  float2* twf = sm + N;   // (B, A) order: forward transforms
  float4* stg4 = reinterpret_cast<float4*>(sm + Z::OFF_STG);
  float2* xb = sm + Z::OFF_STG;
  cgf::fill_twt<A, B, OB>(tw, t.twz);
  cgf::fill_twt<OB, OA, A>(twf, t.twz);
  cgf::pdl_wait();
  const int s = threadIdx.x & 15, p = threadIdx.x >> 4;
  const RowEx<A, B, true> exi{sm + Z::OFF_EX + p * Z::EX};  // 16 threads per pencil: warp-local
  const RowEx<OB, OA, true> exf{sm + Z::OFF_EX + p * Z::EX};
  const int ytiles = (d.ny + CG_ZROWS - 1) / CG_ZROWS;
  const int x = blockIdx.x / ytiles;
  const int y0 = (blockIdx.x - x * ytiles) * CG_ZROWS;
  const int ya = y0 + 2 * p, yb = ya + 1;
  const bool va = ya < d.ny, vb = yb < d.ny;
  const int b_idx = blockIdx.y;
  const long long off = (long long)b_idx * d.nspec;
  const float spx = t.sx[x];
  const float spa = va ? spx * t.sy[ya] : 0.f, spb = vb ? spx * t.sy[yb] : 0.f;
  const long long rowa = ((long long)x * d.ny + ya) * N, rowb = rowa + N;
  // shared tables: tw | stg (aliased by xb) | exchange | material table | labels
  float4* tab_s = reinterpret_cast<float4*>(sm + Z::OFF_TAB);
  uint8_t* lab_s = reinterpret_cast<uint8_t*>(tab_s + 256);
  const bool lab = z_stage_labels<N>(lab_s, tab_s, m, d, x, y0);
  const uint8_t* la = lab_s + (2 * p) * N;
  const uint8_t* lb = la + N;
#pragma unroll 1
  for (int comp = 0; comp < 3; ++comp) {
    float2* S = (comp == 0 ? S1 : (comp == 1 ? S0 : S2)) + off;
    const float* mk = (comp == 2) ? t.kz : nullptr;
    float* uc = u + ((long long)comp * gridDim.y + b_idx) * d.ncell;
    z_stage<N>(stg4, S, d, x, y0, mk);
    // the velocities of this thread's cells load while the inverse transform runs
    float ua[OB], ub[OB];
    static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int n = s + OA * b;
      ua[b] = (s < OA && va) ? __ldg(uc + rowa + n) : 0.f;
      ub[b] = (s < OA && vb) ? __ldg(uc + rowb + n) : 0.f;
    });
    __syncthreads();
    float2 v[A], w[OB];
    z_inputs<N>(v, stg4, p, s);
    fft2<A, B, true>(v, w, s, tw, exi);
    // u <- (u - dt/rho g) * absorb * sponge   (engine.py:462-464)
    if (s < OA) static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int n = s + OA * b;
      const float sz = t.sz[n];
      float2 r = make_float2(0.f, 0.f);
      if (va) {
        const float4 cf = lab ? tab_s[la[n]] : cell_coef(m, rowa + n);
        float un = ua[b] - cf.x * w[b].x;
        un = un * cf.z;
        un = un * (spa * sz);
        uc[rowa + n] = un;
        r.x = un;
      }
      if (vb) {
        const float4 cf = lab ? tab_s[lb[n]] : cell_coef(m, rowb + n);
        float un = ub[b] - cf.x * w[b].y;
        un = un * cf.z;
        un = un * (spb * sz);
        uc[rowb + n] = un;
        r.y = un;
      }
      w[b] = r;
    });
    float2 X[A];
    fft2<OB, OA, false>(w, X, s, twf, exf);
    z_split_store<N, CG_TILE, true>(xb, X, S, d, x, y0, p, s, mk);
  }
}

// MODE 0: forward transform of p only; 1: full update
template <int N, int MODE>
__global__ void __launch_bounds__(CG_THREADS, CG_FAST_MINB) kf_zpass_p(Dims d, Tables t, MediumDev m, SourceDev src,
                                                           RecordDev rec, const long long* ctl, int n_local,
                                                           int record, float* __restrict__ p_all,
                                                           float2* __restrict__ S0) {
  using Z = ZShape<N>;
  constexpr int A = Z::A, B = Z::B, OA = Z::OA, OB = Z::OB;
  extern __shared__ float2 sm[];
  __shared__ unsigned int s_peak;
  float2* tw = sm;        // (A, B) order: inverse transforms
  float2* twf = sm + N;   // (B, A) order: forward transforms
  float4* stg4 = reinterpret_cast<float4*>(sm + Z::OFF_STG);
  float2* xb = sm + Z::OFF_STG;
  cgf::pdl_trigger();
  cgf::fill_twt<A, B, OB>(tw, t.twz);
  cgf::fill_twt<OB, OA, A>(twf, t.twz);
  cgf::pdl_wait();
  if (threadIdx.x == 0) s_peak = 0u;
  const int s = threadIdx.x & 15, p = threadIdx.x >> 4;
  const RowEx<A, B, true> exi{sm + Z::OFF_EX + p * Z::EX};  // 16 threads per pencil: warp-local
  const RowEx<OB, OA, true> exf{sm + Z::OFF_EX + p * Z::EX};
  const int ytiles = (d.ny + CG_ZROWS - 1) / CG_ZROWS;
  const int x = blockIdx.x / ytiles;
  const int y0 = (blockIdx.x - x * ytiles) * CG_ZROWS;
  const int ya = y0 + 2 * p, yb = ya + 1;
  const bool va = ya < d.ny, vb = yb < d.ny;
  const int b_idx = blockIdx.y;
  float2* S = S0 + (long long)b_idx * d.nspec;
  float* pb = p_all + (long long)b_idx * d.ncell;
  const long long rowa = ((long long)x * d.ny + ya) * N, rowb = rowa + N;
  __syncthreads();
  float2 w[OB];
  if constexpr (MODE == 0) {
    if (s < OA) static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int n = s + OA * b;
      w[b] = make_float2(va ? pb[rowa + n] : 0.f, vb ? pb[rowb + n] : 0.f);
    });
  } else {
    float4* tab_s = reinterpret_cast<float4*>(sm + Z::OFF_TAB);
    uint8_t* lab_s = reinterpret_cast<uint8_t*>(tab_s + 256);
    const bool lab = z_stage_labels<N>(lab_s, tab_s, m, d, x, y0);
    const uint8_t* la = lab_s + (2 * p) * N;
    const uint8_t* lb = la + N;
    z_stage<N>(stg4, S, d, x, y0, nullptr);
    // this thread's pressures load while the inverse transform runs
    float pa[OB], pbv[OB];
    static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int n = s + OA * b;
      pa[b] = (s < OA && va) ? __ldg(pb + rowa + n) : 0.f;
      pbv[b] = (s < OA && vb) ? __ldg(pb + rowb + n) : 0.f;
    });
    __syncthreads();
    float2 v[A];
    z_inputs<N>(v, stg4, p, s);
    fft2<A, B, true>(v, w, s, tw, exi);
    const long long n_step = ctl[0] + n_local;
    const float spx = t.sx[x];
    const float spa = va ? spx * t.sy[ya] : 0.f, spb = vb ? spx * t.sy[yb] : 0.f;
    // p <- (p - (rho c^2 dt [+ 2 beta dt p]) div u) * absorb * sponge   (engine.py:470-477)
    if (s < OA) static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int n = s + OA * b;
      const float sz = t.sz[n];
      float2 r = make_float2(0.f, 0.f);
      if (va) {
        const float4 cf = lab ? tab_s[la[n]] : cell_coef(m, rowa + n);
        const float po = pa[b];
        float pn = m.nonlinear ? po - (cf.y + cf.w * po) * w[b].x : po - cf.y * w[b].x;
        pn = pn * cf.z;
        r.x = __fmul_rn(pn, spa * sz);  // rounded here: see the persistent p-pass
      }
      if (vb) {
        const float4 cf = lab ? tab_s[lb[n]] : cell_coef(m, rowb + n);
        const float po = pbv[b];
        float pn = m.nonlinear ? po - (cf.y + cf.w * po) * w[b].y : po - cf.y * w[b].y;
        pn = pn * cf.z;
        r.y = __fmul_rn(pn, spb * sz);
      }
      w[b] = r;
    });
    // source (engine.py:478-482): entries of rows ya, yb owned by this thread
    if (src.S > 0 && n_step < src.n_drive && s < OA && va) {
      const float4 dr = src.drive[n_step];
      const int ra = x * d.ny + ya;
      const int e0 = src.row_ptr[ra], e1 = src.row_ptr[ra + 1], e2 = vb ? src.row_ptr[ra + 2] : e1;
      for (int e = e0; e < e2; ++e) {
        const int zz = src.zidx[e];
        if (zz % OA != s) continue;
        const int k2 = zz / OA;
        const float acv = src.ac[(long long)b_idx * src.S + e];
        const float asv = src.as[(long long)b_idx * src.S + e];
        const float add = dr.x * (dr.y * acv - dr.z * asv);
        const bool on_b = e >= e1;
        static_for<0, OB>([&](auto bi) {
          constexpr int b = decltype(bi)::value;
          if (k2 == b) {
            if (on_b) w[b].y += add;
            else w[b].x += add;
          }
        });
      }
    }
    // write p, convergence peak, record window
    unsigned int lpeak = 0u;
    const int m_bin = (int)(n_step % rec.spp);
    const long long Ry = rec.hi[1] - rec.lo[1], Rz = rec.hi[2] - rec.lo[2];
    const bool x_conv = x >= rec.clo[0] && x < rec.chi[0];
    const bool x_rec = record && x >= rec.lo[0] && x < rec.hi[0];
    float* bins = rec.bins + ((long long)b_idx * rec.spp + m_bin) * rec.nrec;
    float* comp = rec.comp + ((long long)b_idx * rec.spp + m_bin) * rec.nrec;
    float* pmax = rec.pmax + (long long)b_idx * rec.nrec;
    if (s < OA) static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int n = s + OA * b;
      for (int r = 0; r < 2; ++r) {
        const int y = r ? yb : ya;
        if (r ? !vb : !va) continue;
        const float pn = r ? w[b].y : w[b].x;
        pb[(r ? rowb : rowa) + n] = pn;
        const float apn = fabsf(pn);
        if (x_conv && y >= rec.clo[1] && y < rec.chi[1] && n >= rec.clo[2] && n < rec.chi[2])
          lpeak = max(lpeak, __float_as_uint(apn));
        if (x_rec && y >= rec.lo[1] && y < rec.hi[1] && n >= rec.lo[2] && n < rec.hi[2]) {
          const long long ri = ((long long)(x - rec.lo[0]) * Ry + (y - rec.lo[1])) * Rz + (n - rec.lo[2]);
          const float sv = bins[ri], cm0 = comp[ri];
          const float yk = pn - cm0;
          const float tk = sv + yk;
          comp[ri] = (tk - sv) - yk;
          bins[ri] = tk;
          const float pm = pmax[ri];
          pmax[ri] = (apn > pm || apn != apn) ? apn : pm;
        }
      }
    });
    lpeak = __reduce_max_sync(0xffffffffu, lpeak);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_peak, lpeak);
    __syncthreads();
    if (threadIdx.x == 0 && s_peak != 0u) {
      const long long per = n_step / rec.spp;
      if (per < rec.max_periods) atomicMax(&rec.peaks[(long long)b_idx * rec.max_periods + per], s_peak);
    }
  }
  float2 X[A];
  fft2<OB, OA, false>(w, X, s, twf, exf);
  z_split_store<N, CG_TILE, false>(xb, X, S, d, x, y0, p, s, nullptr);
}

// ---------------------------------------------------------------------------
// Persistent, pipelined z-passes. Each CTA walks every G-th item -- tiles in
// the p-pass, (tile, velocity component) pairs in the u-pass -- and the half
// spectrum and labels of the next item streams into shared memory -- by tensor-map box copies on an
// mbarrier (TMA instantiations, ny even) or by cp.async from every thread --
// while the current one is transformed. Both land in the same layout: boxes
// of 8 pencils by NH k rows of 128 bytes, a pencil's 16 bytes (A_k, B_k) of
// row k at chunk (p % 8) XOR (k % 8). An item's staging buffer is then reused
// as its exchange and split-store buffer.
//
// Bound: latency (barriers, shared-memory round trips) below about 256^3,
// HBM above. Resident warps, registers and the L1 that shared memory leaves
// for loads in flight pull against each other; measured (us, u-pass / p-pass):
//   8 pencils x 4 CTAs against 16 x 2 (16 threads a pencil): 160x160x192 x 8
//     378 / 148 against 403 / 156, 256x256x144 111 / 47 against 116 / 53, but
//     192x192x256 102 / 41 against 97 / 41 and 256^3 172 / 67 against 163 / 66
//   8 x 2 against 16 x 1 and 8 x 3 (20 threads): 400^3 706 / 289 against
//     755 / 305 and 817 / 337, 256x256x320 254 / 109 against 263 / 115, 316 / 126
//   16 x 1 against 8 x 2 (32 threads): 512^3 1786 / 671 against 1847 / 667
// (one line of spectrum per k row is 8 pencils). Before these tiles, with
// contiguous runs of 16-pencil tiles per CTA and the smaller split factor
// first: 400^3 768 / 322, 256x256x320 287 / 125, 160x160x192 x 8 433 / 182,
// 192x192x256 97 / 43.
constexpr size_t kSmBytes = 233472;  // shared memory of an SM; each CTA reserves 1 KB of it
constexpr size_t zp_fit(int ctas) {  // bytes a CTA may use when `ctas` share an SM
  return (kSmBytes / ctas < 232448 + 1024 ? kSmBytes / ctas : 232448 + 1024) - 1024 - 64;
}

template <int N>
struct ZPShape {
  static constexpr int A = ZSplit<N>::A, B = ZSplit<N>::B, OA = ZSplit<N>::OA, OB = ZSplit<N>::OB, NH = N / 2 + 1;
  static constexpr int TPP = ZSplit<N>::TPP;           // threads per pencil
  static constexpr int P = N == 256 || (TPP == 32 && !ZSplit<N>::P::THREE) ? 16 : 8;  // pencils per tile
  static constexpr int ROWS = 2 * P, THREADS = P * TPP, BOXES = P / 8;
  static constexpr bool WARP = (32 % TPP) == 0;  // a pencil's threads in one warp
  // the field values of a thread load before its inverse transform unless
  // the transform's A values per thread leave no registers for them
  static constexpr bool EARLY = A <= 20;
  static constexpr int EX_I = RowEx<A, B>::SLAB, EX_F = RowEx<OB, OA>::SLAB;
  static constexpr int EX = EX_I > EX_F ? EX_I : EX_F;
  // staged boxes, each on a 1024-byte boundary (the 128-byte swizzle repeats
  // every 8 rows), plus 1024 bytes to align the first one in the item buffer
  static constexpr bool TMA_OK = NH <= 256;
  static constexpr int BOXB = (NH * 128 + 1023) / 1024 * 1024;
  static constexpr int B_STG = (BOXES * BOXB + 1024) / 8, B_EX = P * EX, B_XB = N * P;  // float2 units
  static constexpr int B_MAX = B_STG > B_EX ? (B_STG > B_XB ? B_STG : B_XB) : (B_EX > B_XB ? B_EX : B_XB);
  static constexpr int BUF = (B_MAX + 1) / 2 * 2;  // even: float4-aligned
  // tensor-map instantiations of more than 16 threads a pencil move the tile's
  // field rows (contiguous) through shared memory by bulk copies instead of the
  // threads' loads and stores: runs of 18..25 floats straddle sectors, and the
  // registers that held the early loads are what these lengths lack. u- / p-pass
  // us, threads' loads -> bulk: 300^3 397 / 146 -> 357 / 142, 384^3 669 / 274 ->
  // 634 / 250, 400^3 705 / 278 -> 697 / 266, 256x256x200 222 / 92 -> 211 / 88;
  // with 16 threads 192x192x256 97 / 41 -> 99 / 43, 160x160x192 x 8 379 / 149 ->
  // 380 / 148.
  static constexpr bool BULK = N % 2 == 0 && TMA_OK && TPP > 16;
};

// Shared-memory layout of the u-pass (U) or the p-pass:
// twiddles (two orders, one where they are the same) | two item buffers | material table
// (u: (dt/rho, absorb); p: the four coefficients) | k_z (u) | z sponge | two
// label tiles | field rows (bulk copies) | mbarriers. Offsets in float2 units.
template <int N, bool U, bool TMA>
struct ZPLayout {
  using Z = ZPShape<N>;
  static constexpr bool BULK = TMA && Z::BULK;
  static constexpr int TW = ZSplit<N>::TW;
  static constexpr int TWF = Z::A == Z::OB ? 0 : TW;  // twiddles of the forward order
  static constexpr size_t OFF_BUF = Z::A == Z::OB ? TW + TW % 2 : 2 * TW;
  static constexpr size_t OFF_TAB = OFF_BUF + 2 * (size_t)Z::BUF;
  static constexpr size_t OFF_KZ = OFF_TAB + (U ? 256 : 512);
  static constexpr size_t LABB = 2 * ((size_t)Z::ROWS * N + 16);  // bytes, slots on multiples of 16
  static constexpr int KZ0 = U ? (Z::NH + 3) / 4 * 2 : 0, SZ0 = (N + 3) / 4 * 2;
  static constexpr size_t FLDB = BULK ? sizeof(float) * (size_t)Z::ROWS * N : 0;  // a multiple of 16
  static constexpr size_t CORE = sizeof(float2) * OFF_KZ + LABB + FLDB + 32;
  // resident CTAs per SM: up to 16 warps (two CTAs of the 20..28-thread
  // pencils, whose 18..27 values a thread want more than 128 registers), as
  // far as shared memory allows
  static constexpr int ctas() {
    int c = Z::TPP > 16 && Z::TPP < 32 ? 2 : 512 / Z::THREADS;
    while (c > 1 && CORE > zp_fit(c)) --c;
    return c;
  }
  static constexpr int MINB = ctas();
  // the k_z and sponge tables stay in shared memory where they cost no
  // resident CTA, else they are read through L1
  static constexpr bool TBL = CORE + sizeof(float2) * (KZ0 + SZ0) <= zp_fit(MINB);
  static constexpr size_t OFF_SZ = OFF_KZ + (TBL ? KZ0 : 0);
  static constexpr size_t OFF_LAB = OFF_SZ + (TBL ? SZ0 : 0);
  static constexpr size_t OFF_FLD = sizeof(float2) * OFF_LAB + LABB;  // bytes
  static constexpr size_t OFF_BAR = OFF_FLD + FLDB;                   // bytes
  static constexpr size_t smem = OFF_BAR + 4 * sizeof(unsigned long long);
  static_assert(smem <= zp_fit(1), "persistent z-pass tile does not fit shared memory");
};

// The forward-only pass holds no tables, labels or field rows: twiddles and two
// item buffers, 16 warps an SM. (Three CTAs instead of two of the 20-thread
// pencils: a 320^3 forward transform 191 -> 175 us, 300^3 165 -> 154. 24 warps of
// the 16-thread ones: 160x160x192 x 2 59 -> 57, but 100x120x135 x 2 32.5 -> 33.6
// and 256^3 83 -> 84.)
template <int N>
struct ZPFwd {
  using Z = ZPShape<N>;
  static constexpr size_t smem = sizeof(float2) * (ZPLayout<N, false, false>::OFF_BUF + 2 * (size_t)Z::BUF);
  static constexpr int ctas() {
    int c = 512 / Z::THREADS;
    while (c > 1 && smem > zp_fit(c)) --c;
    return c > 1 ? c : 1;
  }
  static constexpr int MINB = ctas();
};

// An item's place: velocity component comp (radix NC: 3 in the u-pass, 1 in
// the p-pass), member b, y-tile yt of plane x, the first fastest. CTA i takes
// items i, i + G, i + 2 G, ...: at any time the resident CTAs work on
// neighbouring tiles, whose spectrum rows and labels share lines and DRAM
// pages, and a grid of few tiles still fills the SMs. (A tile's components on
// three CTAs read its labels three times, once from DRAM; keeping them on one
// measured 0-3 % slower from 160x160x192 to 400^3.) Stepped by adding the
// digits of G: a CTA divides once, not once per item.
template <int NC>
struct ZCursor {
  int comp, b, yt, x;
  int dc, db, dyt, dx;  // digits of the stride
  __device__ __forceinline__ static void digits(unsigned i, int n_members, int ytiles, int& c, int& b, int& yt,
                                                int& x) {
    c = (int)(i % NC);
    i /= NC;
    b = (int)(i % (unsigned)n_members);
    i /= (unsigned)n_members;
    yt = (int)(i % (unsigned)ytiles);
    x = (int)(i / (unsigned)ytiles);
  }
  __device__ __forceinline__ ZCursor(int n_members, int ytiles) {
    digits(blockIdx.x, n_members, ytiles, comp, b, yt, x);
    digits(gridDim.x, n_members, ytiles, dc, db, dyt, dx);
  }
  __device__ __forceinline__ void next(int n_members, int ytiles) {
    comp += dc;
    b += db;
    yt += dyt;
    x += dx;
    if (comp >= NC) comp -= NC, ++b;
    if (b >= n_members) b -= n_members, ++yt;
    if (yt >= ytiles) yt -= ytiles, ++x;
  }
};

// First 1024-byte boundary of item buffer j.
template <int N, class L>
__device__ __forceinline__ char* zt_stage(float2* sm, int j) {
  char* b = reinterpret_cast<char*>(sm + L::OFF_BUF + (size_t)j * ZPShape<N>::BUF);
  const unsigned a = cgf::smem_addr(b);
  return b + (((a + 1023u) & ~1023u) - a);
}

// The half spectrum of tile (x, y0) of S into the staging boxes by cp.async
// (8-byte pieces on an odd ny; the missing second row of a last single row is
// zero, rows past it are left as they are: nothing of them is stored).
template <int N>
__device__ __forceinline__ void z_prefetch(char* stg, const float2* __restrict__ S, const Dims& d, int x, int y0) {
  using Z = ZPShape<N>;
  const float2* base = S + (long long)x * Z::NH * d.ny + y0;
  const int nyv = min(Z::ROWS, d.ny - y0);
  const bool even = (d.ny & 1) == 0;
  for (int idx = threadIdx.x; idx < Z::NH * Z::P; idx += Z::THREADS) {
    const int k = idx / Z::P, pp = idx % Z::P;
    char* dst = stg + (pp >> 3) * Z::BOXB + k * 128 + (((pp & 7) ^ (k & 7)) << 4);
    const float2* src = base + (long long)k * d.ny + 2 * pp;
    if (2 * pp + 1 < nyv) {
      if (even) {
        cgf::cp_async16(dst, src);
      } else {
        cgf::cp_async8(dst, src);
        cgf::cp_async8(dst + 8, src + 1);
      }
    } else if (2 * pp < nyv) {
      cgf::cp_async8(dst, src);
      *reinterpret_cast<float2*>(dst + 8) = make_float2(0.f, 0.f);
    }
  }
}

// The same by tensor-map box copies, counted on bar; issued by one thread.
template <int N>
__device__ __forceinline__ void zt_issue(char* stg, unsigned long long* bar, const CUtensorMap* map, const Dims& d,
                                         long long b, int x, int y0) {
  using Z = ZPShape<N>;
  const int c2 = (int)(b * d.nx + x);
  cgf::mbar_expect_tx(bar, (unsigned)Z::BOXES * Z::NH * 128u);
  cgf::tma_load_3d(stg, map, bar, 2 * y0, 0, c2);
  if constexpr (Z::BOXES == 2) cgf::tma_load_3d(stg + Z::BOXB, map, bar, 2 * y0 + 32, 0, c2);
}

// The tile's labels (ROWS rows of N bytes, contiguous) into lab_s +
// label_shift, asynchronously: 16 bytes at a time where every plane of ny N
// bytes starts on 16 (a tile starts a multiple of 16 N bytes into its plane, a
// slab on a plane), else the aligned 4-byte words that hold them; the last word
// of the volume, if it is not whole, byte by byte. The words before a tile's
// first byte are the volume's own: it starts on a multiple of 256.
template <int N>
__device__ __forceinline__ int label_shift(const MediumDev& m, const Dims& d, int x) {
  return (int)(((unsigned)(uintptr_t)m.labels + (unsigned)x * (unsigned)(d.ny * N)) & 3u);
}
template <int N>
__device__ __forceinline__ void z_prefetch_labels(uint8_t* lab_s, const MediumDev& m, const Dims& d, int x, int y0) {
  using Z = ZPShape<N>;
  const uint8_t* first = m.labels + ((long long)x * d.ny + y0) * N;
  const int nb = min(Z::ROWS, d.ny - y0) * N;
  if ((d.ny * N) % 16 == 0) {
    for (int i = 16 * threadIdx.x; i < nb; i += 16 * Z::THREADS) cgf::cp_async16(lab_s + i, first + i);
  } else {
    const int mis = label_shift<N>(m, d, x);
    const uint8_t* src = first - mis;
    const long long avail = m.labels_end - src;
    for (int i = 4 * threadIdx.x; i < nb + mis; i += 4 * Z::THREADS) {
      if (i + 4 <= avail)
        cgf::cp_async4(lab_s + i, src + i);
      else
        for (int k = i; k < avail; ++k) lab_s[k] = src[k];
    }
  }
}

// Phase-1 inputs of the inverse transform from the staged boxes: times
// i*mk[k] when mk is given, Im of the self-paired bins dropped, then the
// Hermitian extension (Z_n = A_n + i B_n, n = s + B a).
template <int N>
__device__ __forceinline__ void z_inputs_box(float2 (&v)[ZSplit<N>::A], const char* stg, int p, int s,
                                             const float* mk) {
  constexpr int A = ZSplit<N>::A, B = ZSplit<N>::B;
  const char* box = stg + (p >> 3) * ZPShape<N>::BOXB;
  const int c = p & 7;
  static_for<0, A>([&](auto ai) {
    constexpr int a = decltype(ai)::value;
    const int n = s + B * a;
    float2 z = make_float2(0.f, 0.f);
    if (s < B) {
      const bool hi = 2 * n > N;
      const int k = hi ? N - n : n;
      const float4 f = *reinterpret_cast<const float4*>(box + k * 128 + ((c ^ (k & 7)) << 4));
      float2 fa = make_float2(f.x, f.y), fb = make_float2(f.z, f.w);
      if (mk) {
        const float kk = mk[k];
        fa = c_muli(c_scale(fa, kk));
        fb = c_muli(c_scale(fb, kk));
      }
      if (k == 0 || 2 * k == N) {
        fa.y = 0.f;
        fb.y = 0.f;
      }
      z = hi ? make_float2(fa.x + fb.y, fb.x - fa.y)   // conj(A) + i conj(B)
             : make_float2(fa.x - fb.y, fa.y + fb.x);  // A + i B
    }
    v[a] = z;
  });
}

// Cells of a row that a thread reads at a time, of its B: all loads of a chunk
// before its first store, which the compiler will not move a load across. (A
// dense medium's coefficients, u- / p-pass us, a cell at a time -> in chunks:
// 192x192x256 170 / 67 -> 108 / 57, 150^3 76 / 39 -> 50 / 31.)
constexpr int z_chunk(int B) { return B % 4 == 0 ? 4 : (B % 5 == 0 ? 5 : (B % 3 == 0 ? 3 : (B % 2 == 0 ? 2 : 1))); }
// A dense medium's coefficients of the p-pass: (-, rho c^2 dt, absorb, 2 beta dt).
__device__ __forceinline__ float4 z_dense_p(const MediumDev& m, long long i) {
  return make_float4(0.f, __ldg(m.rc2 + i), __ldg(m.ab + i), m.b2 ? __ldg(m.b2 + i) : 0.f);
}

template <int N, bool U, bool TMA>
__device__ __forceinline__ void zp_tables(float2* sm, const Tables& t, const MediumDev& m) {
  using L = ZPLayout<N, U, TMA>;
  using Z = ZPShape<N>;
  cgf::fill_twt<Z::A, Z::B, Z::OB>(sm, t.twz);
  if (L::TWF) cgf::fill_twt<Z::OB, Z::OA, Z::A>(sm + L::TWF, t.twz);
  if (L::TBL) {
    if (U) {
      float* kz_s = reinterpret_cast<float*>(sm + L::OFF_KZ);
      for (int i = threadIdx.x; i < Z::NH; i += Z::THREADS) kz_s[i] = t.kz[i];
    }
    float* sz_s = reinterpret_cast<float*>(sm + L::OFF_SZ);
    for (int i = threadIdx.x; i < N; i += Z::THREADS) sz_s[i] = t.sz[i];
  }
  if (m.labels)
    for (int i = threadIdx.x; i < 256; i += Z::THREADS) {
      const float4 c = m.ltab[i];
      if (U)
        sm[L::OFF_TAB + i] = make_float2(c.x, c.z);
      else
        reinterpret_cast<float4*>(sm + L::OFF_TAB)[i] = c;
    }
}

// Waits for item buffer j's staging (tensor-map path); a wait that gives up
// raises the flag and the kernel carries on with whatever arrived.
__device__ __forceinline__ void zt_wait(unsigned long long* bars, unsigned& phase, int j, int* err) {
  if (!cgf::mbar_wait(bars + j, (phase >> j) & 1u)) atomicExch(err, 1);
  phase ^= 1u << j;
}

__device__ __forceinline__ void zt_init(unsigned long long* bars) {
  if (threadIdx.x == 0) {
    cgf::mbar_init(bars, 1);
    cgf::mbar_init(bars + 1, 1);
    cgf::mbar_init(bars + 2, 1);
    cgf::mbar_init_fence();
  }
  __syncthreads();
}

// TMA: the tile's half spectra arrive by tensor-map box copies (ztma: the
// descriptors, by value) instead of per-thread cp.async; the labels keep
// cp.async. Other instantiations ignore ztma.
// DENSE: the medium is maps, not labels. Instantiations of their own, for the
// registers: u- / p-pass us with labels, both in one kernel -> apart: 400^3 677 /
// 259 -> 637 / 240, 300^3 344 / 137 -> 330 / 132.
template <int N, bool TMA = false, bool DENSE = false>
__global__ void __launch_bounds__(ZPShape<N>::THREADS, ZPLayout<N, true, TMA>::MINB)
    kfp_zpass_u(Dims d, Tables t, MediumDev m, float* __restrict__ u, float2* __restrict__ S0,
                float2* __restrict__ S1, float2* __restrict__ S2, int n_members,
                const __grid_constant__ ZTma ztma) {
  using Z = ZPShape<N>;
  using L = ZPLayout<N, true, TMA>;
  constexpr int A = Z::A, B = Z::B, OA = Z::OA, OB = Z::OB;
  extern __shared__ float2 sm[];
  const int ytiles = (d.ny + Z::ROWS - 1) / Z::ROWS;  // the last tile may be ragged
  cgf::pdl_trigger();
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(sm) + L::OFF_BAR);
  unsigned phase = 0u;  // bit j: parity of item buffer j's next staging phase
  if constexpr (TMA) zt_init(bars);
  zp_tables<N, true, TMA>(sm, t, m);
  cgf::pdl_wait();
  const float* kz_s = L::TBL ? reinterpret_cast<const float*>(sm + L::OFF_KZ) : t.kz;
  const float* sz_s = L::TBL ? reinterpret_cast<const float*>(sm + L::OFF_SZ) : t.sz;
  const float2* tab2_s = sm + L::OFF_TAB;
  uint8_t* lab0 = reinterpret_cast<uint8_t*>(sm + L::OFF_LAB);
  constexpr bool lab = !DENSE;
  const int s = threadIdx.x % Z::TPP, p = threadIdx.x / Z::TPP;
  auto spec = [&](int comp, long long b) { return (comp == 0 ? S1 : (comp == 1 ? S0 : S2)) + b * d.nspec; };
  auto prefetch = [&](const ZCursor<3>& c, int j) {
    const int y0 = c.yt * Z::ROWS;
    char* stg = zt_stage<N, L>(sm, j);
    if constexpr (TMA) {
      if (threadIdx.x == 0) zt_issue<N>(stg, bars + j, &ztma.map[c.comp], d, c.b, c.x, y0);  // map order = comp order
    } else {
      z_prefetch<N>(stg, spec(c.comp, c.b), d, c.x, y0);
    }
    if constexpr (lab) z_prefetch_labels<N>(lab0 + j * (Z::ROWS * N + 16), m, d, c.x, y0);
    cgf::cp_async_commit();
  };
  ZCursor<3> cur(n_members, ytiles);
  int j = 0;
  // the item's velocity rows (BULK)
  float* fld = reinterpret_cast<float*>(reinterpret_cast<char*>(sm) + L::OFF_FLD);
  auto rows_of = [&](const ZCursor<3>& c) {
    return u + ((long long)c.comp * n_members + c.b) * d.ncell + ((long long)c.x * d.ny + c.yt * Z::ROWS) * N;
  };
  auto rows_bytes = [&](const ZCursor<3>& c) { return 4u * (unsigned)min(Z::ROWS, d.ny - c.yt * Z::ROWS) * N; };
  auto load_rows = [&](const ZCursor<3>& c) {
    if (threadIdx.x != 0) return;
    cgf::mbar_expect_tx(bars + 2, rows_bytes(c));
    cgf::bulk_load(fld, rows_of(c), rows_bytes(c), bars + 2);
  };
  prefetch(cur, 0);  // every CTA of the grid has an item
  if constexpr (L::BULK) load_rows(cur);
#pragma unroll 1
  for (; cur.x < d.nx; j ^= 1) {
    const int comp = cur.comp;
    const long long b_idx = cur.b;
    const int x = cur.x, y0 = cur.yt * Z::ROWS;
    const uint8_t* la = lab0 + j * (Z::ROWS * N + 16) + label_shift<N>(m, d, x) + (2 * p) * N;
    const uint8_t* lb = la + N;
    const int ya = y0 + 2 * p, yb = ya + 1;
    const bool va = ya < d.ny, vb = yb < d.ny;  // this pencil's rows exist
    const long long rowa = ((long long)x * d.ny + ya) * N, rowb = rowa + N;
    float* uc = u + ((long long)comp * n_members + b_idx) * d.ncell;
    // this thread's velocities load while the staged spectrum is transformed.
    // LATE: after it, where A-value registers would not leave room for them, a
    // chunk of cells at a time and in program order, from the L2, where the pencil
    // fetches its rows when the item starts. (The compiler otherwise moves each
    // load down to its use, a round trip to memory a cell. u-pass us, one block of
    // loads / in chunks / and fetched: 128x128x512 220 / 220 / 127, 512^3 3173 / 3166 /
    // 1733, 256x256x640 804 / 770 / 640, dense 128x128x640 273 / 242 / 222. One CTA
    // of 16 warps an SM: nothing else hides the latency.)
    constexpr bool LATE = !Z::EARLY && !L::BULK;
    float ua[OB], ub[OB];
    auto load_u = [&](auto first, auto count) {
      static_for<0, decltype(count)::value>([&](auto ji) {
        constexpr int b = decltype(first)::value + decltype(ji)::value;
        const int n = s + OA * b;
        if constexpr (LATE) {
          ua[b] = va ? cgf::ld_ordered(uc + rowa + n) : 0.f;
          ub[b] = vb ? cgf::ld_ordered(uc + rowb + n) : 0.f;
        } else {
          ua[b] = (s < OA && va) ? __ldg(uc + rowa + n) : 0.f;
          ub[b] = (s < OA && vb) ? __ldg(uc + rowb + n) : 0.f;
        }
      });
    };
    using All = std::integral_constant<int, OB>;
    using Zero = std::integral_constant<int, 0>;
    float* const rows = rows_of(cur);
    const unsigned bytes = rows_bytes(cur);
    // the sponge's x and y factors, read ahead of the transform (192x192x256 97.1 ->
    // 93.0 us, 160x160x192 x 8 375 -> 369; lengths of 20 threads the same)
    const float spx = t.sx[x], sya = va ? t.sy[ya] : 0.f, syb = vb ? t.sy[yb] : 0.f;
    if (Z::EARLY && !L::BULK) load_u(Zero{}, All{});
    if constexpr (LATE)
      for (int i = s; 32 * i < (va + vb) * N; i += Z::TPP) cgf::prefetch_l2(uc + rowa + 32 * i);
    // (tensor-map path) this thread's generic accesses to the buffer the
    // next copy fills are ordered before that copy
    if constexpr (TMA) cgf::fence_proxy_async();
    cgf::cp_async_wait0();
    __syncthreads();
    cur.next(n_members, ytiles);
    if (cur.x < d.nx) prefetch(cur, j ^ 1);
    float2* bufj = sm + L::OFF_BUF + (size_t)j * Z::BUF;
    float2 v[A], w[OB];
    if constexpr (TMA) zt_wait(bars, phase, j, ztma.err);
    z_inputs_box<N>(v, zt_stage<N, L>(sm, j), p, s, comp == 2 ? kz_s : nullptr);
    __syncthreads();  // the staging is read: the buffer becomes the exchange
    const RowEx<A, B, Z::WARP> exi{bufj + p * Z::EX};
    const RowEx<OB, OA, Z::WARP> exf{bufj + p * Z::EX};
    fft2<A, B, true>(v, w, s, sm, exi);
    if constexpr (L::BULK) {
      zt_wait(bars, phase, 2, ztma.err);
      static_for<0, OB>([&](auto bi) {
        constexpr int b = decltype(bi)::value;
        ua[b] = (s < OA) ? fld[2 * p * N + s + OA * b] : 0.f;
        ub[b] = (s < OA) ? fld[(2 * p + 1) * N + s + OA * b] : 0.f;
      });
    }
    const float spa = spx * sya, spb = spx * syb;
    // u <- (u - dt/rho g) * absorb * sponge   (engine.py:462-464)
    // ca, cb: (dt/rho, absorb) of cells n of the two rows
    auto update = [&](auto bi, float2 ca, float2 cb) {
      constexpr int b = decltype(bi)::value;
      const int n = s + OA * b;
      const float sz = sz_s[n];
      float una = ua[b] - ca.x * w[b].x;
      una = una * ca.y;
      una = una * (spa * sz);
      float unb = ub[b] - cb.x * w[b].y;
      unb = unb * cb.y;
      unb = unb * (spb * sz);
      if constexpr (L::BULK) {
        fld[2 * p * N + n] = una;
        fld[(2 * p + 1) * N + n] = unb;
      } else {
        if (va) uc[rowa + n] = una;
        if (vb) uc[rowb + n] = unb;
      }
      w[b] = make_float2(una, vb ? unb : 0.f);
    };
    constexpr int RC = z_chunk(OB);
    using Chunk = std::integral_constant<int, RC>;
    if constexpr (lab) {
      if (s < OA) static_for<0, OB / RC>([&](auto ci) {
        constexpr int c0 = decltype(ci)::value * RC;
        if constexpr (LATE) load_u(std::integral_constant<int, c0>{}, Chunk{});
        static_for<0, RC>([&](auto ji) {
          constexpr int b = c0 + decltype(ji)::value;
          const int n = s + OA * b;
          update(std::integral_constant<int, b>{}, tab2_s[la[n]], tab2_s[lb[n]]);
        });
      });
    } else if (s < OA) {
      static_for<0, OB / RC>([&](auto ci) {
        constexpr int c0 = decltype(ci)::value * RC;
        if constexpr (LATE) load_u(std::integral_constant<int, c0>{}, Chunk{});
        float2 ca[RC], cb[RC];
        static_for<0, RC>([&](auto ji) {
          constexpr int j = decltype(ji)::value;
          const int n = s + OA * (c0 + j);
          ca[j] = va ? make_float2(__ldg(m.dtr + rowa + n), __ldg(m.ab + rowa + n)) : make_float2(0.f, 0.f);
          cb[j] = vb ? make_float2(__ldg(m.dtr + rowb + n), __ldg(m.ab + rowb + n)) : make_float2(0.f, 0.f);
        });
        static_for<0, RC>([&](auto ji) {
          constexpr int j = decltype(ji)::value;
          update(std::integral_constant<int, c0 + j>{}, ca[j], cb[j]);
        });
      });
    }
    if constexpr (L::BULK) {
      cgf::fence_proxy_async();
      __syncthreads();
      if (threadIdx.x == 0) cgf::bulk_store(rows, fld, bytes);
    }
    float2 X[A];
    fft2<OB, OA, false>(w, X, s, sm + L::TWF, exf);
    if constexpr (L::BULK)
      if (threadIdx.x == 0 && cur.x < d.nx) {  // cur: the next item
        cgf::bulk_wait_read();
        load_rows(cur);
      }
    z_split_store<N, Z::P, false>(bufj, X, spec(comp, b_idx), d, x, y0, p, s, comp == 2 ? kz_s : nullptr);
  }
  if constexpr (L::BULK)
    if (threadIdx.x == 0) cgf::bulk_wait();
}

// REC: the step records into the phase bins (an instantiation without the
// record path keeps the non-recording steps' instruction stream short).
// FWD: only the closing forward transform, of the pressure as it is -- the
// spectrum a step leaves behind, rebuilt from a restored pressure field by
// the very code the step runs, so a restored run continues bit for bit.
// INV: only the opening inverse transform, its values to the pressure.
// TMA: the half spectra arrive by tensor-map box copies (as in the u-pass).
template <int N, bool REC, bool FWD = false, bool TMA = false, bool INV = false, bool DENSE = false>
__global__ void __launch_bounds__(ZPShape<N>::THREADS, FWD ? ZPFwd<N>::MINB : ZPLayout<N, false, TMA>::MINB)
    kfp_zpass_p(Dims d, Tables t, MediumDev m, SourceDev src, RecordDev rec, const long long* ctl, int n_local,
                int record, float* __restrict__ p_all, float2* __restrict__ S0, int n_members,
                const __grid_constant__ ZTma ztma) {
  using Z = ZPShape<N>;
  using L = ZPLayout<N, false, TMA>;
  constexpr int A = Z::A, B = Z::B, OA = Z::OA, OB = Z::OB;
  static_assert(!(FWD && (TMA || INV)), "the forward-only pass stages no spectrum");
  extern __shared__ float2 sm[];
  const int ytiles = (d.ny + Z::ROWS - 1) / Z::ROWS;  // the last tile may be ragged
  cgf::pdl_trigger();
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(reinterpret_cast<char*>(sm) + L::OFF_BAR);
  unsigned phase = 0u;  // bit j: parity of item buffer j's next staging phase
  if constexpr (TMA) zt_init(bars);
  if constexpr (FWD) {
    cgf::fill_twt<Z::OB, Z::OA, Z::A>(sm + L::TWF, t.twz);
    __syncthreads();
  } else if constexpr (INV) {
    cgf::fill_twt<Z::A, Z::B, Z::OB>(sm, t.twz);
  } else {
    zp_tables<N, false, TMA>(sm, t, m);
  }
  cgf::pdl_wait();
  const float* sz_s = L::TBL ? reinterpret_cast<const float*>(sm + L::OFF_SZ) : t.sz;
  const float4* tab_s = reinterpret_cast<const float4*>(sm + L::OFF_TAB);
  uint8_t* lab0 = reinterpret_cast<uint8_t*>(sm + L::OFF_LAB);
  constexpr bool lab = !INV && !DENSE;
  const int s = threadIdx.x % Z::TPP, p = threadIdx.x / Z::TPP;
  auto prefetch = [&](const ZCursor<1>& c, int j) {
    const int y0 = c.yt * Z::ROWS;
    char* stg = zt_stage<N, L>(sm, j);
    if constexpr (TMA) {
      if (threadIdx.x == 0) zt_issue<N>(stg, bars + j, &ztma.map[1], d, c.b, c.x, y0);  // map[1]: S0
    } else {
      z_prefetch<N>(stg, S0 + c.b * d.nspec, d, c.x, y0);
    }
    if constexpr (lab) z_prefetch_labels<N>(lab0 + j * (Z::ROWS * N + 16), m, d, c.x, y0);
    cgf::cp_async_commit();
  };
  ZCursor<1> cur(n_members, ytiles);
  if constexpr (FWD) {
    int jf = 0;
    for (; cur.x < d.nx; jf ^= 1, cur.next(n_members, ytiles)) {
      const long long b_idx = cur.b;
      const int x = cur.x, y0 = cur.yt * Z::ROWS;
      const int ya = y0 + 2 * p;
      const bool va = ya < d.ny, vb = ya + 1 < d.ny;
      const float* pb = p_all + b_idx * d.ncell;
      const long long rowa = ((long long)x * d.ny + ya) * N, rowb = rowa + N;
      float2 w[OB];
      if (s < OA) static_for<0, OB>([&](auto bi) {
        constexpr int b = decltype(bi)::value;
        const int n = s + OA * b;
        w[b] = make_float2(va ? __ldg(pb + rowa + n) : 0.f, vb ? __ldg(pb + rowb + n) : 0.f);
      });
      float2* bufj = sm + L::OFF_BUF + (size_t)jf * Z::BUF;
      const RowEx<OB, OA, Z::WARP> exf{bufj + p * Z::EX};
      float2 X[A];
      fft2<OB, OA, false>(w, X, s, sm + L::TWF, exf);
      z_split_store<N, Z::P, false>(bufj, X, S0 + b_idx * d.nspec, d, x, y0, p, s, nullptr);
    }
    return;
  }
  // the tile's pressure rows (BULK)
  float* fld = reinterpret_cast<float*>(reinterpret_cast<char*>(sm) + L::OFF_FLD);
  auto rows_of = [&](const ZCursor<1>& c) {
    return p_all + c.b * d.ncell + ((long long)c.x * d.ny + c.yt * Z::ROWS) * N;
  };
  auto rows_bytes = [&](const ZCursor<1>& c) { return 4u * (unsigned)min(Z::ROWS, d.ny - c.yt * Z::ROWS) * N; };
  auto load_rows = [&](const ZCursor<1>& c) {
    if (threadIdx.x != 0) return;
    cgf::mbar_expect_tx(bars + 2, rows_bytes(c));
    cgf::bulk_load(fld, rows_of(c), rows_bytes(c), bars + 2);
  };
  prefetch(cur, 0);
  if constexpr (L::BULK) load_rows(cur);
  const long long n_step = INV ? 0 : ctl[0] + n_local;
  const int m_bin = (int)(n_step % rec.spp);
  const long long per_log = n_step / rec.spp;
  unsigned int wpeak = 0u;
  int wmember = -1;
  const long long Ry = rec.hi[1] - rec.lo[1], Rz = rec.hi[2] - rec.lo[2];
  const bool drive_on = src.S > 0 && n_step < src.n_drive;
  const float4 dr = drive_on ? src.drive[n_step] : make_float4(0.f, 0.f, 0.f, 0.f);
  static_assert(OB <= 32, "one mask bit per cell of a thread");
  unsigned int zconv = 0u, zrec = 0u;  // bit b: this thread's cell z = s + A b is in the box
  if (s < OA) static_for<0, OB>([&](auto bi) {
    constexpr int b = decltype(bi)::value;
    const int n = s + OA * b;
    if (n >= rec.clo[2] && n < rec.chi[2]) zconv |= 1u << b;
    if (n >= rec.lo[2] && n < rec.hi[2]) zrec |= 1u << b;
  });
  int j = 0;
#pragma unroll 1
  for (; cur.x < d.nx; j ^= 1) {
    const long long b_idx = cur.b;
    const int x = cur.x, y0 = cur.yt * Z::ROWS;
    const uint8_t* la = lab0 + j * (Z::ROWS * N + 16) + label_shift<N>(m, d, x) + (2 * p) * N;
    const uint8_t* lb = la + N;
    const int ya = y0 + 2 * p, yb = ya + 1;
    const bool va = ya < d.ny, vb = yb < d.ny;  // this pencil's rows exist
    float* pb = p_all + b_idx * d.ncell;
    float2* S = S0 + b_idx * d.nspec;
    const long long rowa = ((long long)x * d.ny + ya) * N, rowb = rowa + N;
    // this thread's pressures load while the staged spectrum is transformed
    // (after it where A-value registers would not leave room for them)
    float pa[OB], pbv[OB];
    auto load_p = [&]() {
      static_for<0, OB>([&](auto bi) {
        constexpr int b = decltype(bi)::value;
        const int n = s + OA * b;
        pa[b] = (s < OA && va) ? __ldg(pb + rowa + n) : 0.f;
        pbv[b] = (s < OA && vb) ? __ldg(pb + rowb + n) : 0.f;
      });
    };
    float* const rows = rows_of(cur);
    const unsigned bytes = rows_bytes(cur);
    // the sponge's x and y factors, read ahead of the transform where 16 threads
    // hold the cells (192x192x256 41.0 -> 39.4 us); else they would spill (300^3 138
    // -> 148, 150^3 24.6 -> 26.0) or not pay (160x160x192 x 8, 12 threads, 149 -> 152)
    constexpr bool SP = A == 16 && !INV;
    float spx = 0.f, sya = 0.f, syb = 0.f;
    auto sponge_xy = [&]() {
      spx = t.sx[x];
      sya = va ? t.sy[ya] : 0.f;
      syb = vb ? t.sy[yb] : 0.f;
    };
    if (SP) sponge_xy();
    if (Z::EARLY && !INV && !L::BULK) load_p();
    if constexpr (TMA) cgf::fence_proxy_async();  // see the u-pass
    cgf::cp_async_wait0();
    __syncthreads();
    cur.next(n_members, ytiles);
    if (cur.x < d.nx) prefetch(cur, j ^ 1);
    float2* bufj = sm + L::OFF_BUF + (size_t)j * Z::BUF;
    float2 v[A], w[OB];
    if constexpr (TMA) zt_wait(bars, phase, j, ztma.err);
    z_inputs_box<N>(v, zt_stage<N, L>(sm, j), p, s, nullptr);
    __syncthreads();  // the staging is read: the buffer becomes the exchange
    const RowEx<A, B, Z::WARP> exi{bufj + p * Z::EX};
    const RowEx<OB, OA, Z::WARP> exf{bufj + p * Z::EX};
    fft2<A, B, true>(v, w, s, sm, exi);
    if constexpr (INV) {
      if (s < OA) static_for<0, OB>([&](auto bi) {
        constexpr int b = decltype(bi)::value;
        const int n = s + OA * b;
        if (va) pb[rowa + n] = w[b].x;
        if (vb) pb[rowb + n] = w[b].y;
      });
        continue;
    }
    if (!Z::EARLY && !L::BULK) load_p();
    if constexpr (L::BULK) {
      zt_wait(bars, phase, 2, ztma.err);
      static_for<0, OB>([&](auto bi) {
        constexpr int b = decltype(bi)::value;
        pa[b] = (s < OA) ? fld[2 * p * N + s + OA * b] : 0.f;
        pbv[b] = (s < OA) ? fld[(2 * p + 1) * N + s + OA * b] : 0.f;
      });
    }
    if (!SP) sponge_xy();
    const float spa = spx * sya, spb = spx * syb;
    // p <- (p - (rho c^2 dt [+ 2 beta dt p]) div u) * absorb * sponge   (engine.py:470-477)
    constexpr int RC = z_chunk(OB);
    auto update = [&](auto bi, float4 ca, float4 cb) {
      constexpr int b = decltype(bi)::value;
      const int n = s + OA * b;
      const float sz = sz_s[n];
      const float poa = pa[b], pob = pbv[b];
      float pna = m.nonlinear ? poa - (ca.y + ca.w * poa) * w[b].x : poa - ca.y * w[b].x;
      float pnb = m.nonlinear ? pob - (cb.y + cb.w * pob) * w[b].y : pob - cb.y * w[b].y;
      pna = pna * ca.z;
      pnb = pnb * cb.z;
      // rounded here: the transform below takes the stored value, so that the
      // forward-only pass rebuilds the same spectrum from it bit for bit
      w[b] = make_float2(__fmul_rn(pna, spa * sz), vb ? __fmul_rn(pnb, spb * sz) : 0.f);
    };
    if constexpr (lab) {
      if (s < OA) static_for<0, OB>([&](auto bi) {
        const int n = s + OA * decltype(bi)::value;
        update(bi, tab_s[la[n]], tab_s[lb[n]]);
      });
    } else if (s < OA) {
      static_for<0, OB / RC>([&](auto ci) {
        constexpr int c0 = decltype(ci)::value * RC;
        float4 ca[RC], cb[RC];
        static_for<0, RC>([&](auto ji) {
          constexpr int j = decltype(ji)::value;
          const int n = s + OA * (c0 + j);
          ca[j] = va ? z_dense_p(m, rowa + n) : make_float4(0.f, 0.f, 0.f, 0.f);
          cb[j] = vb ? z_dense_p(m, rowb + n) : make_float4(0.f, 0.f, 0.f, 0.f);
        });
        static_for<0, RC>([&](auto ji) {
          constexpr int j = decltype(ji)::value;
          update(std::integral_constant<int, c0 + j>{}, ca[j], cb[j]);
        });
      });
    }
    // source (engine.py:478-482): entries of rows ya, yb owned by this thread
    if (drive_on && s < OA && va) {
      const int ra = x * d.ny + ya;
      const int e0 = src.row_ptr[ra], e1 = src.row_ptr[ra + 1], e2 = vb ? src.row_ptr[ra + 2] : e1;
      for (int e = e0; e < e2; ++e) {
        const int zz = src.zidx[e];
        if (zz % OA != s) continue;
        const int k2 = zz / OA;
        const float acv = src.ac[b_idx * src.S + e];
        const float asv = src.as[b_idx * src.S + e];
        const float add = dr.x * (dr.y * acv - dr.z * asv);
        const bool on_b = e >= e1;
        static_for<0, OB>([&](auto bi) {
          constexpr int b = decltype(bi)::value;
          if (k2 == b) {
            if (on_b) w[b].y += add;
            else w[b].x += add;
          }
        });
      }
    }
    // write p, convergence peak, record window (z-range membership of this
    // thread's cells is a per-kernel bit mask, the y/x membership per tile)
    unsigned int lpeak = 0u;
    const bool x_conv = x >= rec.clo[0] && x < rec.chi[0];
    const bool x_rec = REC && record && x >= rec.lo[0] && x < rec.hi[0];
    const bool conv_a = x_conv && va && ya >= rec.clo[1] && ya < rec.chi[1];
    const bool conv_b = x_conv && vb && yb >= rec.clo[1] && yb < rec.chi[1];
    const bool rec_a = x_rec && va && ya >= rec.lo[1] && ya < rec.hi[1];
    const bool rec_b = x_rec && vb && yb >= rec.lo[1] && yb < rec.hi[1];
    if (s < OA) static_for<0, OB>([&](auto bi) {
      constexpr int b = decltype(bi)::value;
      const int n = s + OA * b;
      const float pna = w[b].x, pnb = w[b].y;
      if constexpr (L::BULK) {
        fld[2 * p * N + n] = pna;
        fld[(2 * p + 1) * N + n] = pnb;
      } else {
        if (va) pb[rowa + n] = pna;
        if (vb) pb[rowb + n] = pnb;
      }
      if ((zconv >> b) & 1u) {
        if (conv_a) lpeak = max(lpeak, __float_as_uint(fabsf(pna)));
        if (conv_b) lpeak = max(lpeak, __float_as_uint(fabsf(pnb)));
      }
    });
    if constexpr (REC) {
      // phase bin m (Kahan-compensated sum) and running max |p| of this
      // thread's recorded cells, RC cells per row at a time: every load of a
      // chunk is issued before its first store, so the chunk costs one round
      // trip to memory instead of one per cell
      if (s < OA && (rec_a || rec_b)) {
        float* __restrict__ bins = rec.bins + (b_idx * rec.spp + m_bin) * rec.nrec;
        float* __restrict__ comp = rec.comp + (b_idx * rec.spp + m_bin) * rec.nrec;
        float* __restrict__ pmax = rec.pmax + b_idx * rec.nrec;
        const long long ra = ((long long)(x - rec.lo[0]) * Ry + (ya - rec.lo[1])) * Rz - rec.lo[2];
        const long long rb = ra + Rz;  // row yb = ya + 1
        static_for<0, OB / RC>([&](auto ci) {
          constexpr int c0 = decltype(ci)::value * RC;
          float sv[2 * RC], cm[2 * RC], pm[2 * RC];
          static_for<0, RC>([&](auto ji) {
            constexpr int j = decltype(ji)::value, b = c0 + j;
            const int n = s + OA * b;
            const bool in = (zrec >> b) & 1u;
            sv[j] = (in && rec_a) ? bins[ra + n] : 0.f;
            cm[j] = (in && rec_a) ? comp[ra + n] : 0.f;
            pm[j] = (in && rec_a) ? pmax[ra + n] : 0.f;
            sv[RC + j] = (in && rec_b) ? bins[rb + n] : 0.f;
            cm[RC + j] = (in && rec_b) ? comp[rb + n] : 0.f;
            pm[RC + j] = (in && rec_b) ? pmax[rb + n] : 0.f;
          });
          static_for<0, RC>([&](auto ji) {
            constexpr int j = decltype(ji)::value, b = c0 + j;
            const int n = s + OA * b;
            if (!((zrec >> b) & 1u)) return;
            for (int r = 0; r < 2; ++r) {
              if (r ? !rec_b : !rec_a) continue;
              const long long ri = (r ? rb : ra) + n;
              const float pn = r ? w[b].y : w[b].x, apn = fabsf(pn);
              const int k = r * RC + j;
              const float yk = pn - cm[k];
              const float tk = sv[k] + yk;
              comp[ri] = (tk - sv[k]) - yk;
              bins[ri] = tk;
              pmax[ri] = (apn > pm[k] || apn != apn) ? apn : pm[k];
            }
          });
        });
      }
    }
    // convergence peak: a running max per warp over its tiles, written to
    // the period log (an integer max over the float bits) when the batch
    // member changes and at the end -- no barrier per tile
    lpeak = __reduce_max_sync(0xffffffffu, lpeak);
    if (b_idx != wmember) {
      if ((threadIdx.x & 31) == 0 && wpeak && per_log < rec.max_periods)
        atomicMax(&rec.peaks[(long long)wmember * rec.max_periods + per_log], wpeak);
      wpeak = 0u;
      wmember = (int)b_idx;
    }
    wpeak = max(wpeak, lpeak);
    if constexpr (L::BULK) {
      cgf::fence_proxy_async();
      __syncthreads();
      if (threadIdx.x == 0) cgf::bulk_store(rows, fld, bytes);
    }
    float2 X[A];
    fft2<OB, OA, false>(w, X, s, sm + L::TWF, exf);
    if constexpr (L::BULK)
      if (threadIdx.x == 0 && cur.x < d.nx) {  // cur: the next tile
        cgf::bulk_wait_read();
        load_rows(cur);
      }
    z_split_store<N, Z::P, false>(bufj, X, S, d, x, y0, p, s, nullptr);
  }
  if constexpr (L::BULK)
    if (threadIdx.x == 0) cgf::bulk_wait();
  if ((threadIdx.x & 31) == 0 && wpeak && wmember >= 0 && per_log < rec.max_periods)
    atomicMax(&rec.peaks[(long long)wmember * rec.max_periods + per_log], wpeak);
}

// ------------------------------------------------ per-length launchers --
// persistent z-passes (any N of CG_FAST_ZSIZES); ztma (encoded descriptors,
// host memory) selects the tensor-map staging where the length allows it
static const ZTma kNoZTma = {};
// one CTA per item up to `per_sm` resident CTAs on every SM
static int zp_grid(long long items, int per_sm) {
  const long long slots = (long long)cgf::sm_count() * per_sm;
  return (int)(items < slots ? items : slots);
}
template <int N>
static long long zp_tiles(const Dims& d, int batch) {
  return (long long)d.nx * ((d.ny + ZPShape<N>::ROWS - 1) / ZPShape<N>::ROWS) * batch;
}
template <int N, bool DENSE>
void zp_launch_u(const Dims& d, const Tables& t, const MediumDev& m, float* u, float2* S0, float2* S1, float2* S2,
                 int batch, cudaStream_t st, const ZTma* ztma) {
  const long long items = 3 * zp_tiles<N>(d, batch);
  const dim3 block(ZPShape<N>::THREADS);
  if constexpr (ZPShape<N>::TMA_OK) {
    if (ztma) {
      using L = ZPLayout<N, true, true>;
      cgf::launch(d.pdl, kfp_zpass_u<N, true, DENSE>, dim3(zp_grid(items, L::MINB)), block, L::smem, st, d, t, m, u, S0, S1,
                  S2, batch, *ztma);
      return;
    }
  }
  using L = ZPLayout<N, true, false>;
  cgf::launch(d.pdl, kfp_zpass_u<N, false, DENSE>, dim3(zp_grid(items, L::MINB)), block, L::smem, st, d, t, m, u, S0, S1, S2,
              batch, kNoZTma);
}
template <int N>
void zp_run_u(const Dims& d, const Tables& t, const MediumDev& m, float* u, float2* S0, float2* S1, float2* S2,
              int batch, cudaStream_t st, const ZTma* ztma) {
  if (m.labels)
    zp_launch_u<N, false>(d, t, m, u, S0, S1, S2, batch, st, ztma);
  else
    zp_launch_u<N, true>(d, t, m, u, S0, S1, S2, batch, st, ztma);
}

template <int N, bool REC, bool DENSE>
void zp_launch_p(const Dims& d, const Tables& t, const MediumDev& m, const SourceDev& src, const RecordDev& rec,
                 const long long* ctl, int n_local, int record, float* p, float2* S0, int batch, cudaStream_t st,
                 const ZTma* ztma) {
  const dim3 block(ZPShape<N>::THREADS);
  if constexpr (ZPShape<N>::TMA_OK) {
    if (ztma) {
      using L = ZPLayout<N, false, true>;
      cgf::launch(d.pdl, kfp_zpass_p<N, REC, false, true, false, DENSE>, dim3(zp_grid(zp_tiles<N>(d, batch), L::MINB)), block,
                  L::smem, st, d, t, m, src, rec, ctl, n_local, record, p, S0, batch, *ztma);
      return;
    }
  }
  using L = ZPLayout<N, false, false>;
  cgf::launch(d.pdl, kfp_zpass_p<N, REC, false, false, false, DENSE>, dim3(zp_grid(zp_tiles<N>(d, batch), L::MINB)), block,
              L::smem, st, d, t, m, src, rec, ctl, n_local, record, p, S0, batch, kNoZTma);
}
template <int N>
void zp_run_p(const Dims& d, const Tables& t, const MediumDev& m, const SourceDev& src, const RecordDev& rec,
              const long long* ctl, int n_local, int record, float* p, float2* S0, int batch, cudaStream_t st,
              const ZTma* ztma) {
  auto run = [&](auto rec_, auto dense) {
    zp_launch_p<N, decltype(rec_)::value, decltype(dense)::value>(d, t, m, src, rec, ctl, n_local, record, p, S0, batch,
                                                                  st, ztma);
  };
  if (m.labels && record)
    run(std::true_type{}, std::false_type{});
  else if (m.labels)
    run(std::false_type{}, std::false_type{});
  else if (record)
    run(std::true_type{}, std::true_type{});
  else
    run(std::false_type{}, std::true_type{});
}

// p -> S0 (forward) or S0 -> p (inverse) alone
template <int N>
void zp_run_half(bool inverse, const Dims& d, const Tables& t, const MediumDev& m, float* p, float2* S0, int batch,
                 cudaStream_t st) {
  using L = ZPLayout<N, false, false>;
  SourceDev src;
  memset(&src, 0, sizeof(src));
  RecordDev rec;
  memset(&rec, 0, sizeof(rec));
  rec.spp = 1;
  if (inverse)
    cgf::launch(d.pdl, kfp_zpass_p<N, false, false, false, true>, dim3(zp_grid(zp_tiles<N>(d, batch), L::MINB)),
                dim3(ZPShape<N>::THREADS), L::smem, st, d, t, m, src, rec, (const long long*)nullptr, 0, 0, p, S0, batch, kNoZTma);
  else
    cgf::launch(d.pdl, kfp_zpass_p<N, false, true>, dim3(zp_grid(zp_tiles<N>(d, batch), ZPFwd<N>::MINB)),
                dim3(ZPShape<N>::THREADS), ZPFwd<N>::smem, st, d, t, m, src, rec, (const long long*)nullptr, 0, 0, p, S0, batch,
                kNoZTma);
}

template <typename K>
static bool zp_allow(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) == cudaSuccess;
}

template <int N, bool TMA, bool DENSE>
static bool zp_allow_step() {
  constexpr size_t su = ZPLayout<N, true, TMA>::smem, sp = ZPLayout<N, false, TMA>::smem;
  return zp_allow(kfp_zpass_u<N, TMA, DENSE>, su) && zp_allow(kfp_zpass_p<N, true, false, TMA, false, DENSE>, sp) &&
         zp_allow(kfp_zpass_p<N, false, false, TMA, false, DENSE>, sp);
}
template <int N>
int zp_prepare() {
  constexpr size_t sp = ZPLayout<N, false, false>::smem;
  bool ok = zp_allow(kfp_zpass_p<N, false, true>, ZPFwd<N>::smem) && zp_allow(kfp_zpass_p<N, false, false, false, true>, sp) &&
            zp_allow_step<N, false, false>() && zp_allow_step<N, false, true>();
  if constexpr (ZPShape<N>::TMA_OK) ok = ok && zp_allow_step<N, true, false>() && zp_allow_step<N, true, true>();
  return ok ? 0 : -1;
}

// one-tile-per-CTA z-passes (N of CG_FAST_SIZES, any ny)
template <int N>
void zt_run_u(const Dims& d, const Tables& t, const MediumDev& m, float* u, float2* S0, float2* S1, float2* S2,
              int batch, cudaStream_t st) {
  const dim3 grid((unsigned)(d.nx * ((d.ny + CG_ZROWS - 1) / CG_ZROWS)), batch);
  cgf::launch(d.pdl, kf_zpass_u<N>, grid, dim3(CG_THREADS), ZShape<N>::smem, st, d, t, m, u, S0, S1, S2);
}

template <int N>
void zt_run_p(int mode, const Dims& d, const Tables& t, const MediumDev& m, const SourceDev& src, const RecordDev& rec,
              const long long* ctl, int n_local, int record, float* p, float2* S0, int batch, cudaStream_t st) {
  const dim3 grid((unsigned)(d.nx * ((d.ny + CG_ZROWS - 1) / CG_ZROWS)), batch);
  if (mode == 0)
    cgf::launch(d.pdl, kf_zpass_p<N, 0>, grid, dim3(CG_THREADS), ZShape<N>::smem, st, d, t, m, src, rec, ctl, n_local,
                record, p, S0);
  else
    cgf::launch(d.pdl, kf_zpass_p<N, 1>, grid, dim3(CG_THREADS), ZShape<N>::smem, st, d, t, m, src, rec, ctl, n_local,
                record, p, S0);
}

template <int N>
int zt_prepare() {
  const int sm = (int)ZShape<N>::smem;
  return (cudaFuncSetAttribute(kf_zpass_u<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) != cudaSuccess ||
          cudaFuncSetAttribute(kf_zpass_p<N, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) != cudaSuccess ||
          cudaFuncSetAttribute(kf_zpass_p<N, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm) != cudaSuccess)
             ? -1
             : 0;
}

#define CG_ZP_INSTANTIATE(n)                                                                                       \
  template void zp_run_u<n>(const Dims&, const Tables&, const MediumDev&, float*, float2*, float2*, float2*, int,  \
                            cudaStream_t, const ZTma*);                                                            \
  template void zp_run_p<n>(const Dims&, const Tables&, const MediumDev&, const SourceDev&, const RecordDev&,     \
                            const long long*, int, int, float*, float2*, int, cudaStream_t, const ZTma*);         \
  template void zp_run_half<n>(bool, const Dims&, const Tables&, const MediumDev&, float*, float2*, int,            \
                               cudaStream_t);                                                                      \
  template int zp_prepare<n>();
#define CG_ZT_INSTANTIATE(n)                                                                                       \
  template void zt_run_u<n>(const Dims&, const Tables&, const MediumDev&, float*, float2*, float2*, float2*, int,  \
                            cudaStream_t);                                                                         \
  template void zt_run_p<n>(int, const Dims&, const Tables&, const MediumDev&, const SourceDev&, const RecordDev&, \
                            const long long*, int, int, float*, float2*, int, cudaStream_t);                      \
  template int zt_prepare<n>();
