// The tiled form of the fused Chorin step (one TH x TW tile per CTA of 32 x 8
// threads), shared by k_stencil / k_stencil_batch (nsgb_stencil.cu) and the
// persistent ensemble kernel (nsgb_ens_persistent.cu).
#pragma once

#include "nsgb_internal.h"

namespace nsgb {

// Shared-memory layout of one TW x TH tile (TW a multiple of 4, TH even).
// Tiles are fetched from HBM as aligned float4 groups covering columns
// j0-4 .. j0+TW+3 (a 16-byte-aligned superset of the halos); each field
// component has its own plane, so a warp's accesses along a row are
// consecutive words.
template <int TW, int TH>
struct StencilSmem {
  static constexpr int G = TW / 4 + 2;        // float4 groups per tile row
  static constexpr int W4 = 4 * G;            // = TW + 8 columns, from j0 - 4
  static constexpr int PH = TH + 6, UH = TH + 4, SH = TH + 2, SW = TW + 2;
  static constexpr int P_OFF = 0;                     // PH x W4
  static constexpr int UX_OFF = P_OFF + PH * W4;      // UH x W4
  static constexpr int UY_OFF = UX_OFF + UH * W4;     // UH x W4
  static constexpr int SX_OFF = UY_OFF + UH * W4;     // SH x SW
  static constexpr int SY_OFF = SX_OFF + SH * SW;     // SH x SW
  static constexpr int F_OFF = SY_OFF + SH * SW;      // SH forcing rows
  static constexpr int R_OFF = F_OFF + SH + 2;        // 8 partial sums
  static constexpr int FLOATS = R_OFF + 8;
};

// Tile (bx, by) of a gx x gy tiling (the objective partial's slot); COH:
// L2-only loads of fields other CTAs of the same launch wrote.
template <int SCHEME, int MODE, int TW, int TH, bool COH = false>
__device__ __forceinline__ void stencil_body(const StencilArgs& a, int step_off, int bx, int by, int gx, int gy) {
  using L = StencilSmem<TW, TH>;
  constexpr int G = L::G, W4 = L::W4, PH = L::PH, UH = L::UH, SH = L::SH, SW = L::SW;
  static_assert(TH % 2 == 0, "the u* phase works on pairs of rows");
  extern __shared__ __align__(16) float sm[];
  float* sP = sm + L::P_OFF;
  float* sUx = sm + L::UX_OFF;
  float* sUy = sm + L::UY_OFF;
  float* sSx = sm + L::SX_OFF;
  float* sSy = sm + L::SY_OFF;
  float* sF = sm + L::F_OFF;
  float* sRed = sm + L::R_OFF;
  const StepConsts& c = a.c;
  const int N = c.N, M = N - 1;
  const size_t NN = (size_t)N * N;
  const int j0 = bx * TW, i0 = by * TH;
  const int tid = threadIdx.y * 32 + threadIdx.x;

  int step = 0;
  float t = a.t_fixed;
  if (MODE == MODE_ROLLOUT) {
    step = (a.step_ctr ? gld(a.step_ctr) : 0) + a.step_fixed + step_off;
    if (a.t_from_step) t = fmul((float)step, c.dt);
  }
  const float nu = (a.theta != nullptr && a.theta_len == 3) ? gldg(a.theta + 2) : c.nu;
  const float cL = fmul(c.dtdx2, nu);

  // Tile loads: aligned float4 groups (a group never straddles the periodic
  // wrap because N and the group start are multiples of 4).
  const bool has_p = a.p != nullptr;
  if (has_p) {
    const float* __restrict__ pp = a.p;
    forflat<PH, G>(tid, [&](int r, int q) {
      const float4 v = gldfield<COH>(reinterpret_cast<const float4*>(pp + (size_t)((i0 - 3 + r) & M) * N +
                                                                     ((j0 - 4 + 4 * q) & M)));
      *reinterpret_cast<float4*>(sP + r * W4 + 4 * q) = v;
    });
  }
  {
    const float* __restrict__ us = a.us;
    forflat<UH, G>(tid, [&](int r, int q) {
      const size_t g = (size_t)((i0 - 2 + r) & M) * N + ((j0 - 4 + 4 * q) & M);
      *reinterpret_cast<float4*>(sUx + r * W4 + 4 * q) = gldfield<COH>(reinterpret_cast<const float4*>(us + g));
      *reinterpret_cast<float4*>(sUy + r * W4 + 4 * q) =
          gldfield<COH>(reinterpret_cast<const float4*>(us + NN + g));
    });
  }
  if (MODE == MODE_ROLLOUT && tid < SH) {
    const ForcingRow fr = forcing_time(gldg(a.theta), gldg(a.theta + 1), t, c);
    sF[tid] = forcing_fx((i0 - 1 + tid) & M, fr, c);
  }
  __syncthreads();

  // 1. pending projection u^n = u* - dt grad p on rows i0-2 .. i0+TH+1 and
  //    columns j0-2 .. j0+TW+1 (plane columns 2 .. TW+5)
  if (has_p) {
    forflat<UH, TW + 4>(tid, [&](int r, int cc) {
      const int col = cc + 2;
      const float* P0 = sP + (r + 1) * W4 + col;  // p at (i0-2+r, j0-2+cc)
      const int o = r * W4 + col;
      sUx[o] = fused_proj(sUx[o], P0[W4], P0[-W4], c.cP);
      sUy[o] = fused_proj(sUy[o], P0[1], P0[-1], c.cP);
    });
    __syncthreads();
  }

  // 2. objective partial on the state before the step; optional state output
  float jacc = 0.0f;
  forflat<TH, TW>(tid, [&](int r, int cc) {
    const int o = (r + 2) * W4 + cc + 4;
    if (MODE == MODE_ROLLOUT) jacc += sUx[o] * sF[r + 1];
    if (a.u_out) {
      const size_t g = (size_t)(i0 + r) * N + (j0 + cc);
      gst(a.u_out + g, sUx[o]);
      gst(a.u_out + NN + g, sUy[o]);
    }
  });

  // 3. u*^{n+1} on rows i0-1 .. i0+TH and columns j0-1 .. j0+TW, two
  //    vertically adjacent cells per thread (rows 2h and 2h+1 of the S tile)
  //    sharing their column loads
  forflat<SH / 2, SW>(tid, [&](int h, int cc) {
    const int r = 2 * h;
    const int o = (r + 1) * W4 + cc + 3;  // U cell of S cell (r, cc)
    float x[4], y[4];                     // U rows r .. r+3 at the cell's column
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = sUx[o + (k - 1) * W4];
      y[k] = sUy[o + (k - 1) * W4];
    }
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int ok = o + k * W4;
      const float ox = x[k + 1], oy = y[k + 1];
      const float lx = x[k], rx = x[k + 2], ux_ = sUx[ok + 1], dx_ = sUx[ok - 1];
      const float ly = y[k], ry = y[k + 2], uy_ = sUy[ok + 1], dy_ = sUy[ok - 1];
      float fx, fy;
      if (MODE == MODE_ROLLOUT) {
        fx = sF[r + k];
        fy = 0.0f;
      } else {
        const size_t g = (size_t)((i0 - 1 + r + k) & M) * N + ((j0 - 1 + cc) & M);
        fx = gldg(a.f + g);
        fy = gldg(a.f + NN + g);
      }
      const int so = (r + k) * SW + cc;
      sSx[so] = fused_ustar<SCHEME>(ox, lx, rx, ux_, dx_, ox, oy, cL, fmul(c.dt, fx), c);
      sSy[so] = fused_ustar<SCHEME>(oy, ly, ry, uy_, dy_, ox, oy, cL, fmul(c.dt, fy), c);
    }
  });
  __syncthreads();

  // 4. write u*^{n+1} and div(u*^{n+1}) / dt for the tile
  {
    float* __restrict__ uso = a.us_out;
    float* __restrict__ rhs = a.rhs;
    forflat<TH, TW>(tid, [&](int r, int cc) {
      const int o = (r + 1) * SW + cc + 1;
      const size_t g = (size_t)(i0 + r) * N + (j0 + cc);
      gst(uso + g, sSx[o]);
      gst(uso + NN + g, sSy[o]);
      gst(rhs + g, fused_rhs(sSx[o + SW], sSx[o - SW], sSy[o + 1], sSy[o - 1], c.cD));
    });
  }

  if (MODE == MODE_ROLLOUT) {
    const int tx = threadIdx.x, ty = threadIdx.y;
    jacc = warp_sum(jacc);
    if (tx == 0) sRed[ty] = jacc;
    __syncthreads();
    if (ty == 0) {
      float v = (tx < 8) ? sRed[tx] : 0.0f;
      v = warp_sum(v);
      if (tx == 0 && (unsigned)step < (unsigned)a.jpart_rows) {
        const int nblk = gx * gy;
        gst(a.jpart + (size_t)step * nblk + by * gx + bx, (double)v);
      }
    }
  }
}

// ---- four cells per thread: tiles at least 64 wide ----
//
// The same step for TW x TH tiles by TW/4 x TH threads, each working on aligned
// groups of four columns: a neighbour row costs one 16-byte shared load for
// four cells and the row's own neighbours two scalars, where the body above
// loads every neighbour of every cell.  All planes hold the columns j0-4 ..
// j0+TW+3; the outermost columns' values are not all meaningful (their own
// neighbours are not loaded) and nothing reads those.  Bound by shared memory
// (75% of its throughput in a batch).  Per step: N = 512, one solve 14.2 -> 13.7
// us, eleven in a batch 43.9 -> 40.1; N = 256 11.1 -> 10.7.  Neighbours by warp
// shuffles instead of scalar loads: 41.4 us; two rows per thread: 39.9.
template <int TW, int TH>
struct Stencil4Smem {
  static constexpr int G = TW / 4 + 2;        // groups per row
  static constexpr int W4 = 4 * G;
  static constexpr int PH = TH + 6, UH = TH + 4, SH = TH + 2;
  static constexpr int NT = TW / 4 * TH;      // threads
  static constexpr int P_OFF = 4;                     // PH rows (4 floats before: the first row's left neighbour)
  static constexpr int UX_OFF = P_OFF + PH * W4;      // UH rows each
  static constexpr int UY_OFF = UX_OFF + UH * W4;
  static constexpr int SX_OFF = UY_OFF + UH * W4;     // SH rows each
  static constexpr int SY_OFF = SX_OFF + SH * W4;
  static constexpr int F_OFF = SY_OFF + SH * W4 + 4;  // SH forcing rows
  static constexpr int R_OFF = F_OFF + SH + 2;        // partial sums of up to 8 warps
  static constexpr int FLOATS = R_OFF + 8;
  static_assert(NT % 32 == 0 && NT <= 256, "threads");
};

// Tiles at least 64 wide use the body with four cells per thread (a block of
// TW/4 x TH threads in one dimension), narrower ones a block of 32 x 8.
template <int TW>
constexpr bool wide_tile() {
  return TW >= 64;
}
template <int TW, int TH>
constexpr int tile_threads() {
  return wide_tile<TW>() ? TW / 4 * TH : 256;
}

// Asynchronous 16-byte copy into shared memory through L2.
__device__ __forceinline__ void copy16(float* dst, const float* src, int line = __builtin_LINE()) {
  if (!bounds_ok(src, 16, line)) return;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void get4(const float* s, float (&v)[4]) {
  const float4 w = *reinterpret_cast<const float4*>(s);
  v[0] = w.x, v[1] = w.y, v[2] = w.z, v[3] = w.w;
}
// The group at s and its left and right neighbours.
__device__ __forceinline__ void get6(const float* s, float (&v)[6]) {
  const float4 w = *reinterpret_cast<const float4*>(s);
  v[0] = s[-1], v[1] = w.x, v[2] = w.y, v[3] = w.z, v[4] = w.w, v[5] = s[4];
}
__device__ __forceinline__ void set4(float* s, const float (&v)[4]) {
  *reinterpret_cast<float4*>(s) = make_float4(v[0], v[1], v[2], v[3]);
}

// Projects rows of two planes in place: rows of `ux`, `uy` are one row below
// those of `P` (row r of them is row r + 1 of P).
template <int ROWS, int G, int NT>
__device__ __forceinline__ void project4(float* ux, float* uy, const float* P, float cP, int tid) {
  constexpr int W4 = 4 * G;
#pragma unroll
  for (int e = tid; e < ROWS * G; e += NT) {
    float x[4], y[4], pn[4], pm[4], pc[6];
    get4(ux + 4 * e, x);
    get4(uy + 4 * e, y);
    get4(P + 4 * e + 2 * W4, pn);
    get4(P + 4 * e, pm);
    get6(P + 4 * e + W4, pc);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = fused_proj(x[k], pn[k], pm[k], cP);
      y[k] = fused_proj(y[k], pc[k + 2], pc[k], cP);
    }
    set4(ux + 4 * e, x);
    set4(uy + 4 * e, y);
  }
}

// Right-hand sides of the four cells whose next field's plane rows sx, sy point
// at (W4 apart).
template <int W4>
__device__ __forceinline__ float4 rhs4(const float* sx, const float* sy, float cD) {
  float xp[4], xm[4], y[6], r[4];
  get4(sx + W4, xp);
  get4(sx - W4, xm);
  get6(sy, y);
#pragma unroll
  for (int k = 0; k < 4; ++k) r[k] = fused_rhs(xp[k], xm[k], y[k + 2], y[k], cD);
  return make_float4(r[0], r[1], r[2], r[3]);
}

template <int SCHEME, int MODE, int TW, int TH>
__device__ __forceinline__ void stencil4_body(const StencilArgs& a, int step_off, int bx, int by, int gx, int gy) {
  using L = Stencil4Smem<TW, TH>;
  constexpr int G = L::G, W4 = L::W4, PH = L::PH, UH = L::UH, SH = L::SH, NT = L::NT;
  extern __shared__ __align__(16) float sm[];
  float* sP = sm + L::P_OFF;
  float* sUx = sm + L::UX_OFF;
  float* sUy = sm + L::UY_OFF;
  float* sSx = sm + L::SX_OFF;
  float* sSy = sm + L::SY_OFF;
  float* sF = sm + L::F_OFF;
  float* sRed = sm + L::R_OFF;
  const StepConsts& c = a.c;
  const int N = c.N, M = N - 1;
  const size_t NN = (size_t)N * N;
  const int j0 = bx * TW, i0 = by * TH;
  const int tid = threadIdx.x;

  const bool has_p = a.p != nullptr;
#pragma unroll
  for (int e = tid; e < UH * G; e += NT) {
    const int r = e / G, q = e % G;
    const size_t g = (size_t)((i0 - 2 + r) & M) * N + ((j0 - 4 + 4 * q) & M);
    copy16(sUx + 4 * e, a.us + g);
    copy16(sUy + 4 * e, a.us + NN + g);
  }
  if (has_p) {
#pragma unroll
    for (int e = tid; e < PH * G; e += NT) {
      const int r = e / G, q = e % G;
      copy16(sP + 4 * e, a.p + (size_t)((i0 - 3 + r) & M) * N + ((j0 - 4 + 4 * q) & M));
    }
  }
  int step = 0;
  float t = a.t_fixed;
  if (MODE == MODE_ROLLOUT) {
    step = (a.step_ctr ? gld(a.step_ctr) : 0) + a.step_fixed + step_off;
    if (a.t_from_step) t = fmul((float)step, c.dt);
    if (tid < SH) {
      const ForcingRow fr = forcing_time(gldg(a.theta), gldg(a.theta + 1), t, c);
      sF[tid] = forcing_fx((i0 - 1 + tid) & M, fr, c);
    }
  }
  const float nu = (a.theta != nullptr && a.theta_len == 3) ? gldg(a.theta + 2) : c.nu;
  const float cL = fmul(c.dtdx2, nu);
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  // 1. pending projection on rows i0-2 .. i0+TH+1
  if (has_p) {
    project4<UH, G, NT>(sUx, sUy, sP, c.cP, tid);
    __syncthreads();
  }

  // 2. u* of the next state on rows i0-1 .. i0+TH
#pragma unroll
  for (int e = tid; e < SH * G; e += NT) {
    const int r = e / G, q = e % G;
    const float* ux = sUx + 4 * e;  // row r of the U planes: one row up
    const float* uy = sUy + 4 * e;
    float xs[4], xn[4], ys[4], yn[4], X[6], Y[6], x[4], y[4], fx[4], fy[4];
    get4(ux, xs);
    get6(ux + W4, X);
    get4(ux + 2 * W4, xn);
    get4(uy, ys);
    get6(uy + W4, Y);
    get4(uy + 2 * W4, yn);
    if (MODE == MODE_ROLLOUT) {
#pragma unroll
      for (int k = 0; k < 4; ++k) fx[k] = sF[r], fy[k] = 0.0f;
    } else {
      const size_t g = (size_t)((i0 - 1 + r) & M) * N + ((j0 - 4 + 4 * q) & M);
      const float4 v = gldg4(a.f + g), w = gldg4(a.f + NN + g);
      fx[0] = v.x, fx[1] = v.y, fx[2] = v.z, fx[3] = v.w;
      fy[0] = w.x, fy[1] = w.y, fy[2] = w.z, fy[3] = w.w;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float ox = X[k + 1], oy = Y[k + 1];
      x[k] = fused_ustar<SCHEME>(ox, xs[k], xn[k], X[k + 2], X[k], ox, oy, cL, fmul(c.dt, fx[k]), c);
      y[k] = fused_ustar<SCHEME>(oy, ys[k], yn[k], Y[k + 2], Y[k], ox, oy, cL, fmul(c.dt, fy[k]), c);
    }
    set4(sSx + 4 * e, x);
    set4(sSy + 4 * e, y);
  }
  __syncthreads();

  // 3. the thread's own group: u* and its right-hand side, state, objective
  const int r = tid / (TW / 4), q = tid % (TW / 4) + 1;
  const size_t g = (size_t)(i0 + r) * N + (j0 - 4 + 4 * q);
  const int os = (r + 1) * W4 + 4 * q, ou = (r + 2) * W4 + 4 * q;
  float x[4], y[4], u[4], v[4];
  get4(sSx + os, x);
  get4(sSy + os, y);
  gst4(a.us_out + g, make_float4(x[0], x[1], x[2], x[3]));
  gst4(a.us_out + NN + g, make_float4(y[0], y[1], y[2], y[3]));
  gst4(a.rhs + g, rhs4<W4>(sSx + os, sSy + os, c.cD));
  get4(sUx + ou, u);
  if (a.u_out) {
    get4(sUy + ou, v);
    gst4(a.u_out + g, make_float4(u[0], u[1], u[2], u[3]));
    gst4(a.u_out + NN + g, make_float4(v[0], v[1], v[2], v[3]));
  }
  if (MODE == MODE_ROLLOUT) {
    const float f = sF[r + 1];
    float jacc = fmul(u[0], f);
#pragma unroll
    for (int k = 1; k < 4; ++k) jacc = __fmaf_rn(u[k], f, jacc);
    jacc = warp_sum(jacc);
    if (tid % 32 == 0) sRed[tid / 32] = jacc;
    __syncthreads();
    if (tid < 32) {
      // a warp's 128 cells in float, 8 roundings deep as a 32 x 8 tile's 256; the
      // warps' sums in double-float (error over the summed magnitudes at N = 512
      // 1.5e-9 -> 5.7e-10, 9.4e-10 with tiles of 32 x 8)
      DFloat s = {tid < NT / 32 ? sRed[tid] : 0.0f, 0.0f};
      s = fold1(fold1(fold1(s, 4), 2), 1);
      if (tid == 0 && (unsigned)step < (unsigned)a.jpart_rows)
        gst(a.jpart + (size_t)step * gx * gy + by * gx + bx, (double)s.hi + (double)s.lo);
    }
  }
}

}  // namespace nsgb
