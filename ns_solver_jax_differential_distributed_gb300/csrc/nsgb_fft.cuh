// Block-level FFT building blocks for power-of-two lengths 16..4096.
//
// A transform of length N is carried by T = N/E threads, each holding E
// complex values in registers (E = 16 or 8, at most N; E the radix, or half a
// radix of 16).  Thread j holds elements j + s*T
// (s = 0..E-1) on entry and X[j + s*T] on exit, so the first pass reads and
// the last pass writes "natural" strided positions; rows stored contiguously
// in global memory are therefore loaded and stored fully coalesced.
//
// The transform is the radix-E Stockham autosort algorithm (a final pass of
// smaller radix when log2(N) is not a multiple of log2(E)).  Radix 8 needs
// half the registers per thread of radix 16 for the same arithmetic, so twice
// as many threads (and warps) carry a transform.  Between passes the values
// are exchanged through shared memory as float2, padded by one element every
// 16 (index i -> i + i/16), which keeps the 64-bit pass writes and reads
// bank-conflict free within each half warp.  Twiddles come from per-pass tables computed on
// the host in double precision and rounded to float: the pass with stride NS
// and radix RP stores W_{NS*RP}^{bm*r} at [r*NS + bm], so the twiddle loads of
// a warp (consecutive bm) are contiguous.  A plan holds the radix-16 tables
// followed by the radix-8 tables (host_twiddles).
#pragma once

#include <algorithm>
#include <cmath>

#include "nsgb_common.cuh"

namespace nsgb {
namespace fft {

__host__ __device__ constexpr int ept(int N) { return N < 16 ? N : 16; }
__host__ __device__ constexpr int padlen(int N) { return N + N / 16 + 4; }
__device__ __forceinline__ int pad(int i) { return i + (i >> 4); }

template <int R>
__device__ __forceinline__ constexpr int bitrev(int k) {
  int r = 0;
  for (int b = 1; b < R; b <<= 1) {
    r = (r << 1) | (k & 1);
    k >>= 1;
  }
  return r;
}

// cos / sin of 2*pi*m/16 for m = 0..7
__device__ __forceinline__ float c16(int m) {
  switch (m) {
    case 0: return 1.0f;
    case 1: return 0.923879532511286756f;
    case 2: return 0.707106781186547524f;
    case 3: return 0.382683432365089772f;
    case 4: return 0.0f;
    case 5: return -0.382683432365089772f;
    case 6: return -0.707106781186547524f;
    default: return -0.923879532511286756f;
  }
}
__device__ __forceinline__ float s16(int m) {
  switch (m) {
    case 0: return 0.0f;
    case 1: return 0.382683432365089772f;
    case 2: return 0.707106781186547524f;
    case 3: return 0.923879532511286756f;
    case 4: return 1.0f;
    case 5: return 0.923879532511286756f;
    case 6: return 0.707106781186547524f;
    default: return 0.382683432365089772f;
  }
}

// d * exp(-+ 2 pi i m / 16): forward uses the minus sign.
template <bool INV>
__device__ __forceinline__ float2 rot16(float2 d, int m) {
  if (m == 0) return d;
  if (m == 4) return INV ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);
  const float c = c16(m);
  const float s = INV ? s16(m) : -s16(m);
  return make_float2(d.x * c - d.y * s, d.x * s + d.y * c);
}

// Stages of span LEN, LEN/2, .. 2 of the in-register DFT of size R (2, 4, 8 or
// 16; LEN = R: the whole DFT), natural order in and out.
template <int R, bool INV, int LEN = R>
__device__ __forceinline__ void dft(float2 (&a)[R]) {
#pragma unroll
  for (int len = LEN; len >= 2; len >>= 1) {
    const int half = len >> 1;
#pragma unroll
    for (int s = 0; s < R; s += len) {
#pragma unroll
      for (int t = 0; t < half; ++t) {
        const float2 u = a[s + t];
        const float2 v = a[s + t + half];
        a[s + t] = cadd(u, v);
        a[s + t + half] = rot16<INV>(csub(u, v), t * (16 / len));
      }
    }
  }
  float2 b[R];
#pragma unroll
  for (int k = 0; k < R; ++k) b[k] = a[bitrev<R>(k)];
#pragma unroll
  for (int k = 0; k < R; ++k) a[k] = b[k];
}

// Sum and difference of u and v g, the last pair of the first stage of a
// transform whose inputs are multiplied by a spectral multiplier: the products
// of all other inputs are rounded, the last one's (fused) is not.  Spelled out,
// because the fusing a compiler finds for itself changes from kernel to kernel
// and with it the last bits of a solve, and an upwind gradient is not
// continuous in those: a cell of |u| below them takes the other one-sided
// difference in the adjoint step.
__device__ __forceinline__ void scaled_butterfly(float2 u, float2 v, float g, bool fused, float2& sum, float2& dif) {
  if (fused) {
    sum = make_float2(__fmaf_rn(v.x, g, u.x), __fmaf_rn(v.y, g, u.y));
    dif = make_float2(__fmaf_rn(-v.x, g, u.x), __fmaf_rn(-v.y, g, u.y));
  } else {
    const float x = fmul(v.x, g), y = fmul(v.y, g);
    sum = make_float2(fadd(u.x, x), fadd(u.y, y));
    dif = make_float2(fsub(u.x, x), fsub(u.y, y));
  }
}

// Offset (in complex entries) of the twiddle table of the pass with stride
// NS in the radix-R tables: the passes before it all have radix R and stride
// R, R^2, ...
template <int R>
__host__ __device__ constexpr int tw_offset(int NS) {
  int off = 0;
  for (int ns = R; ns < NS; ns *= R) off += R * ns;
  return off;
}
// Twiddle entries of the radix-R tables for length N.
template <int R>
__host__ __device__ constexpr int tw_entries(int N) {
  int off = 0;
  for (int ns = R; ns < N; ns *= R) off += ((N / ns >= R) ? R : N / ns) * ns;
  return off > 0 ? off : 1;
}
// Entries of a plan's table (radix 16, then radix 8) and the radix-8 offset.
__host__ __device__ constexpr int tw_total(int N) { return tw_entries<16>(N) + tw_entries<8>(N); }
__host__ __device__ constexpr int tw8_offset(int N) { return tw_entries<16>(N); }

// Fill a plan's twiddle table (tw_total(N) entries): per pass with stride ns
// and radix rp, W_{ns*rp}^{bm*r} at [off + r*ns + bm], in double then rounded.
inline void host_twiddles(int N, float2* out) {
  for (int i = 0; i < tw_total(N); ++i) out[i] = make_float2(1.f, 0.f);
  for (int R = 16, base = 0; R >= 8; base += tw_entries<16>(N), R /= 2) {
    for (int ns = R, off = base; ns < N; off += (N / ns >= R ? R : N / ns) * ns, ns *= R) {
      const int rp = N / ns >= R ? R : N / ns;
      for (int r = 1; r < rp; ++r)
        for (int bm = 0; bm < ns; ++bm) {
          const double ang = -2.0 * M_PI * (double)bm * r / ((double)ns * rp);
          out[off + r * ns + bm] = make_float2((float)std::cos(ang), (float)std::sin(ang));
        }
    }
  }
}

// Squared wavenumbers k2[m] (N entries) and the factor `scale` such that the
// Poisson multiplier is -scale / (k2[a] + k2[b]).  k = 2 pi fftfreq(N, dx) in
// float32 as NS_solver.py:518-519 evaluates it: (m / float32(dx*N)) * 2 *
// float32(pi), then squared in float32; then scaled by the power of two that
// brings k2[1] to [1, 2) (exact, as are the 1/2 of the two-for-one split and
// the 1/N^2 of the inverse transform in `scale`), so that every sum of two
// entries lies well inside the range of the kernels' reciprocal.
inline void host_wavenumbers(int N, double L, float* k2, float* scale) {
  const double dx = L / N;
  const float dn = (float)(dx * N);
  for (int m = 0; m < N; ++m) {
    const int mm = m < N / 2 ? m : m - N;
    volatile float k = (float)mm / dn;
    k = k * 2.0f;
    k = k * (float)M_PI;
    volatile float kk = k * k;
    k2[m] = kk;
  }
  int e = 0;
  if (k2[1] > 0.0f && std::isfinite(k2[1])) e = std::min(100, std::max(-100, -std::ilogb(k2[1])));
  for (int m = 0; m < N; ++m) k2[m] = (float)std::ldexp((double)k2[m], e);
  *scale = (float)std::ldexp(1.0 / (2.0 * (double)N * (double)N), e);
}

// a[s] = buffer[pad(j + s*T)], s = 0..E-1 (and the store of the same
// positions): with T a multiple of 16 the padded positions are pad(j) plus
// constants.
template <int T, int E>
__device__ __forceinline__ void load_strided(float2 (&a)[E], const float2* __restrict__ sb, int j) {
  if constexpr (T % 16 == 0) {
    const float2* src = sb + pad(j);
#pragma unroll
    for (int s = 0; s < E; ++s) a[s] = src[s * (T + T / 16)];
  } else {
#pragma unroll
    for (int s = 0; s < E; ++s) a[s] = sb[pad(j + s * T)];
  }
}
template <int T, int E>
__device__ __forceinline__ void store_strided(const float2 (&a)[E], float2* __restrict__ sb, int j) {
  if constexpr (T % 16 == 0) {
    float2* dst = sb + pad(j);
#pragma unroll
    for (int s = 0; s < E; ++s) dst[s * (T + T / 16)] = a[s];
  } else {
#pragma unroll
    for (int s = 0; s < E; ++s) sb[pad(j + s * T)] = a[s];
  }
}

// Barrier of the threads that carry one transform: the whole CTA (BAR = 0),
// the NT threads of a warp group using hardware barrier BAR (kernels in which
// other warps run other work at the same time), or the warp (BAR = -1:
// transforms of at most 32 threads, every lane of the warp calling).
template <int BAR, int NT>
__device__ __forceinline__ void group_sync() {
  if constexpr (BAR == 0) {
    __syncthreads();
  } else if constexpr (BAR < 0) {
    static_assert(NT <= 32, "a transform inside one warp");
    __syncwarp();
  } else {
    asm volatile("bar.sync %0, %1;" ::"n"(BAR), "n"(NT) : "memory");
  }
}

// a b, each part one rounded product and one fused; the imaginary part fuses
// a.x b.y or (cmul_y) a.y b.x.
__device__ __forceinline__ float2 cmul_x(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -fmul(a.y, b.y)), __fmaf_rn(a.x, b.y, fmul(a.y, b.x)));
}
__device__ __forceinline__ float2 cmul_y(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -fmul(a.y, b.y)), __fmaf_rn(a.y, b.x, fmul(a.x, b.y)));
}
// Products with a twiddle of the table, and of two of them.
template <bool INV>
__device__ __forceinline__ float2 cmul_tw(float2 a, float2 w) {
  return INV ? cmul_y(a, w) : cmul_x(a, w);
}

// W^1, W^2, W^4, W^8 of position bm of a radix-16 pass (conjugate if INV).
// W^r is one of them or the product of at most three (a few ulps), so a
// radix-16 pass issues 4 twiddle loads instead of 15.
template <int NS, bool INV>
__device__ __forceinline__ void load_twiddles16(const float2* __restrict__ tw, int bm, float2& w1, float2& w2,
                                                float2& w4, float2& w8) {
  const float2* __restrict__ tp = tw + tw_offset<16>(NS) + bm;
  w1 = gldg(tp + NS), w2 = gldg(tp + 2 * NS), w4 = gldg(tp + 4 * NS), w8 = gldg(tp + 8 * NS);
  if (INV) {
    w1.y = -w1.y;
    w2.y = -w2.y;
    w4.y = -w4.y;
    w8.y = -w8.y;
  }
}

// Twiddled inputs x[r] *= W^r of a butterfly of size RP at position bm of the
// pass with stride NS, from the radix-R tables.  The radix-16 products are
// spelled out, as in scaled_butterfly: half_butterfly forms the same ones.
template <int NS, int RP, int R, bool INV>
__device__ __forceinline__ void twiddle(float2 (&x)[RP], int bm, const float2* __restrict__ tw) {
  if constexpr (RP == 16) {
    float2 w1, w2, w4, w8;
    load_twiddles16<NS, INV>(tw, bm, w1, w2, w4, w8);
    const float2 w3 = cmul_tw<INV>(w2, w1), w12 = cmul_tw<INV>(w8, w4);
    x[1] = cmul_tw<INV>(x[1], w1);
    x[2] = cmul_tw<INV>(x[2], w2);
    x[3] = cmul_x(x[3], w3);
    x[4] = cmul_tw<INV>(x[4], w4);
    x[5] = cmul_x(x[5], cmul_tw<INV>(w4, w1));
    x[6] = cmul_x(x[6], cmul_tw<INV>(w4, w2));
    x[7] = cmul_x(x[7], cmul_x(w4, w3));
    x[8] = cmul_tw<INV>(x[8], w8);
    x[9] = cmul_x(x[9], cmul_tw<INV>(w8, w1));
    x[10] = cmul_x(x[10], cmul_tw<INV>(w8, w2));
    x[11] = cmul_x(x[11], cmul_x(w8, w3));
    x[12] = cmul_x(x[12], w12);
    x[13] = cmul_x(x[13], cmul_tw<INV>(w12, w1));
    x[14] = cmul_x(x[14], cmul_tw<INV>(w12, w2));
    x[15] = cmul_x(x[15], cmul_x(w12, w3));
  } else {
    const float2* __restrict__ tp = tw + tw_offset<R>(NS) + bm;
#pragma unroll
    for (int r = 1; r < RP; ++r) {
      float2 w = gldg(tp + r * NS);
      if (INV) w.y = -w.y;
      x[r] = cmul(x[r], w);
    }
  }
}

// Outputs r0, r0 + DR, .. of butterfly b of a pass with stride NS and radix RP
// into the exchange buffer.
template <int NS, int RP, int DR, int CNT>
__device__ __forceinline__ void exchange_store(const float2 (&x)[CNT], float2* __restrict__ sb, int b, int r0) {
  const int base = (b / NS) * (NS * RP) + (b & (NS - 1));
  if constexpr (NS == 1 || NS % 16 == 0) {
    // base + r stays inside one 16-entry block (NS = 1) or r * NS is a
    // multiple of 16: the padded positions are pad(base) plus constants
    float2* dst = sb + pad(base) + r0 * (NS + NS / 16);
#pragma unroll
    for (int k = 0; k < CNT; ++k) dst[k * DR * (NS + NS / 16)] = x[k];
  } else {
#pragma unroll
    for (int k = 0; k < CNT; ++k) sb[pad(base + (r0 + k * DR) * NS)] = x[k];
  }
}

// One radix-16 butterfly by two threads of 8 values each (R = 2 E): thread j
// of T = N/8 holds the inputs r = h + 2 s of butterfly b = j % (N/16), h = j /
// (N/16).  The first stage pairs r and r + 8, both the thread's own; then half
// h = 0 goes on with the eight sums and h = 1 with the eight differences, each
// a DFT of size 8, for which the two exchange four values by shuffles.  Every
// value is rounded as in a whole butterfly's registers, so the results are
// those of radix 16 bit for bit, with twice the threads per transform and an
// exchange through shared memory less than in radix 8.
// SCALED: the last input still has its factor g to come (scaled_butterfly).  On
// return a[k] is output 2 k + h.
template <int N, int NS, bool INV, bool SCALED>
__device__ __forceinline__ void half_butterfly(float2 (&a)[8], float g, int b, int h,
                                               const float2* __restrict__ tw) {
  constexpr int LX = N / 16 < 16 ? N / 16 : 16;  // the partner's lane, see split_index
  if constexpr (NS > 1) {
    float2 w1, w2, w4, w8;
    load_twiddles16<NS, INV>(tw, b & (NS - 1), w1, w2, w4, w8);
    const float2 w3 = cmul_tw<INV>(w2, w1), w12 = cmul_tw<INV>(w8, w4);
    // r = h + 2 s.  x q by cmul_x or, for INV and an even r, by cmul_y.
    auto pick = [h](float2 odd, float2 even) { return h ? odd : even; };
    auto mul = [h](float2 x, float2 q) {
      float2 v = cmul_x(x, q);
      if (INV) v.y = h ? v.y : cmul_y(x, q).y;
      return v;
    };
    const float2 v = pick(w3, w2);
    a[0] = pick(cmul_tw<INV>(a[0], w1), a[0]);
    a[1] = mul(a[1], v);
    a[2] = mul(a[2], pick(cmul_tw<INV>(w4, w1), w4));
    a[3] = cmul_x(a[3], mul(w4, v));
    a[4] = mul(a[4], pick(cmul_tw<INV>(w8, w1), w8));
    a[5] = cmul_x(a[5], mul(w8, v));
    a[6] = cmul_x(a[6], pick(cmul_tw<INV>(w12, w1), w12));
    a[7] = cmul_x(a[7], mul(w12, v));
  }
  float2 e[8];
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    float2 sum, dif;
    if (SCALED && s == 3) {
      scaled_butterfly(a[3], a[7], g, h, sum, dif);  // r = 15, or 14 if h = 0
    } else {
      sum = cadd(a[s], a[s + 4]);
      dif = csub(a[s], a[s + 4]);
    }
    const float2 keep = h ? dif : sum, give = h ? sum : dif;
    const float2 got = {__shfl_xor_sync(0xffffffffu, give.x, LX), __shfl_xor_sync(0xffffffffu, give.y, LX)};
    e[2 * s] = h ? got : keep;
    e[2 * s + 1] = h ? keep : got;
  }
#pragma unroll
  for (int t = 1; t < 8; ++t) {
    const float2 r = rot16<INV>(e[t], t);
    e[t] = h ? r : e[t];
  }
  dft<8, INV>(e);
#pragma unroll
  for (int k = 0; k < 8; ++k) a[k] = e[k];
}

// Thread of a transform that lane x of its T = N/8 lanes carries: the two
// threads of a butterfly are N/16 apart, at N = 512 one warp; there the lanes
// are dealt out so that they share one (lanes 0-15 and 16-31 still hold
// neighbouring elements).
template <int N>
__device__ __forceinline__ int split_index(int x) {
  static_assert(N <= 512, "two warps per transform at most");
  if constexpr (N < 512)
    return x;
  else
    return (x & 15) | ((x & 32) >> 1) | ((x & 16) << 1);
}

// One Stockham pass (stride NS) and, recursively, the remaining passes: R the
// radix, E values per thread, E = R or (radix 16) R / 2.  SCALED: the first
// pass multiplies the last input by g.
template <int N, int NS, bool INV, int E, int BAR, int R, bool SCALED>
__device__ __forceinline__ void pass(float2 (&a)[E], float g, float2* __restrict__ sb, int j,
                                     const float2* __restrict__ tw) {
  static_assert(E == R || (E == 8 && R == 16), "radix");
  constexpr int T = N / E;
  constexpr int REM = N / NS;
  constexpr int RP = REM >= R ? R : REM;
  constexpr bool LAST = (NS * RP == N);
  if constexpr (RP > E) {
    const int b = j & (N / 16 - 1), h = j / (N / 16);
    half_butterfly<N, NS, INV, SCALED>(a, g, b, h, tw);
    if constexpr (!LAST) exchange_store<NS, 16, 2>(a, sb, b, h);
  } else {
    constexpr int Q = E / RP;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const int b = j + q * T;
      float2 x[RP];
#pragma unroll
      for (int r = 0; r < RP; ++r) x[r] = a[q + r * Q];
      if constexpr (NS > 1) twiddle<NS, RP, R, INV>(x, b & (NS - 1), tw);
      if constexpr (SCALED) {
        static_assert(Q == 1, "one butterfly per thread");
#pragma unroll
        for (int t = 0; t < RP / 2; ++t) {
          float2 sum, dif;
          if (t == RP / 2 - 1) {
            scaled_butterfly(x[t], x[t + RP / 2], g, true, sum, dif);
          } else {
            sum = cadd(x[t], x[t + RP / 2]);
            dif = csub(x[t], x[t + RP / 2]);
          }
          x[t] = sum;
          x[t + RP / 2] = rot16<INV>(dif, t * (16 / RP));
        }
        dft<RP, INV, RP / 2>(x);
      } else {
        dft<RP, INV>(x);
      }
      if constexpr (LAST) {
#pragma unroll
        for (int r = 0; r < RP; ++r) a[q + r * Q] = x[r];
      } else {
        exchange_store<NS, RP, 1>(x, sb, b, 0);
      }
    }
  }
  if constexpr (!LAST) {
    group_sync<BAR, T>();
    load_strided<T, E>(a, sb, j);
    group_sync<BAR, T>();
    pass<N, NS * RP, INV, E, BAR, R, false>(a, g, sb, j, tw);
  }
}

// Full FFT of length N (unnormalised; INV uses exp(+2 pi i ...)) in radix R
// with E values per thread, `tw` the radix-R tables.  Every thread of the CTA
// (BAR = 0), or of the N/E-thread group synchronised by BAR, must call it (at
// E < R every lane of the warp): it synchronises those threads between passes,
// the last time after their last read of the exchange buffer, which is free
// for reuse on return.
template <int N, bool INV, int E, int BAR = 0, int R = E>
__device__ __forceinline__ void block_fft(float2 (&a)[E], float2* sb, int j, const float2* __restrict__ tw) {
  pass<N, 1, INV, E, BAR, R, false>(a, 0.0f, sb, j, tw);
}
// The transform of a[s] g[s].
template <int N, bool INV, int E, int BAR = 0, int R = E>
__device__ __forceinline__ void block_fft_scaled(float2 (&a)[E], const float (&g)[E], float2* sb, int j,
                                                 const float2* __restrict__ tw) {
#pragma unroll
  for (int s = 0; s < E - 1; ++s) a[s] = make_float2(fmul(a[s].x, g[s]), fmul(a[s].y, g[s]));
  pass<N, 1, INV, E, BAR, R, true>(a, g[E - 1], sb, j, tw);
}

}  // namespace fft
}  // namespace nsgb
