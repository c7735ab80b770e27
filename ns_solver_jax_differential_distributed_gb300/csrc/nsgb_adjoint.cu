// Discrete adjoint of one Chorin step (the reverse-mode derivative that
// jax.grad takes of SingleCoreNSSolver.objective, NS_solver.py:725, 742-756).
//
// Forward step s (exact arithmetic):  v = u + dt (nu L u + A(u) + f_s),
// u_{s+1} = Pr v with Pr = I - G P^-1 D, and J += jscale <u_x, f_x>,
// jscale = dt dx^2.  With periodic central differences G^T = -D and the
// spectral inverse Laplacian symmetric, so Pr^T = Pr and the adjoint recursion
// (lambda_S = 0) is
//   mu_s      = Pr lambda_{s+1}
//   lambda_s  = mu_s + dt (nu L mu_s + A'(u_s)^T mu_s) + jscale (f_x, 0)
//   dJ/dA,B  += sum_cells (jscale u_x + dt mu_x) dfx/dA,B
//   dJ/dnu   += dt <mu_s, L u_s>
// A'(u)^T for central advection A_c = -(u_x Gx u_c + u_y Gy u_c):
//   (A'^T mu)_x = -(mu_x Gx u_x + mu_y Gx u_y) + Gx(mu_x u_x) + Gy(mu_x u_y)
//   (A'^T mu)_y = -(mu_x Gy u_x + mu_y Gy u_y) + Gx(mu_y u_x) + Gy(mu_y u_y)
// and for upwind differences (masks m = [u >= 0] held fixed, as the
// derivative of jnp.where is taken):
//   (A'^T mu)_c = -(mu_x DX u_c... ) terms as below, with the transposed
//   one-sided operator (DX^m)^T w (i) = [(2m_i - 1) w_i - m_{i+1} w_{i+1}
//   + (1 - m_{i-1}) w_{i-1}] / dx.
// The projection Pr lambda_{s+1} reuses the forward machinery: the previous
// adjoint kernel wrote rhs = div(lambda_{s+1}) / dt, the FFT kernels solved for
// p, and this kernel applies mu = lambda - dt grad p on its tile.  The cell
// arithmetic uses the folded coefficients of the fused forward step (dt/h,
// dt nu/dx^2, 1/(h dt)) and FMAs; the theta sensitivities are summed in
// double-float, after float over a thread's few cells (one-cell tiles larger
// than a block) or a row's four (bands), and in double across blocks and steps.
#include "nsgb_adjoint_cell.cuh"
#include "nsgb_rows.cuh"
#include "nsgb_stencil_body.cuh"

namespace nsgb {

// Shared-memory planes of one TW x TH tile: p with a 3-cell halo, u and
// lambda with a 2-cell halo, all fetched as aligned float4 groups from column
// j0 - 4 (pitch W4 = TW + 8), then lambda_s on the tile + 1 halo (pitch SW).
template <int TW, int TH>
struct AdjointSmem {
  static constexpr int G = TW / 4 + 2;
  static constexpr int W4 = 4 * G;
  static constexpr int PH = TH + 6, UH = TH + 4, SH = TH + 2, SW = TW + 2;
  static constexpr int P_OFF = 0;
  static constexpr int UX_OFF = P_OFF + PH * W4;
  static constexpr int UY_OFF = UX_OFF + UH * W4;
  static constexpr int MX_OFF = UY_OFF + UH * W4;
  static constexpr int MY_OFF = MX_OFF + UH * W4;
  static constexpr int LX_OFF = MY_OFF + UH * W4;
  static constexpr int LY_OFF = LX_OFF + SH * SW;
  static constexpr int F_OFF = LY_OFF + SH * SW;  // fx for the SH rows
  static constexpr int DA_OFF = F_OFF + SH;        // dfx/dA, dfx/dB for the TH rows
  static constexpr int DB_OFF = DA_OFF + TH;
  static constexpr int RED_OFF = (DB_OFF + TH + 1) & ~1;  // 3 x 8 double-floats
  static constexpr size_t BYTES = (size_t)RED_OFF * sizeof(float) + 24 * sizeof(DFloat);
};

// Adds a block's theta sensitivities of one adjoint step to its running sums
// (double, one triple per block, steps in backward order); the first adjoint
// step (no lambda yet) starts them.  Keeping the sums per block leaves one
// small reduction per gradient (launch_gsum).
__device__ __forceinline__ void add_theta_partials(const AdjointArgs& a, int blk, DFloat v0, DFloat v1, DFloat v2) {
  double* gp = a.gpart + (size_t)blk * 3;
  const bool more = a.lam != nullptr;
  const double w0 = (double)v0.hi + (double)v0.lo, w1 = (double)v1.hi + (double)v1.lo;
  // the nu partial carries the Laplacian's 1/dx^2 and the step's dt
  const double w2 = ((double)v2.hi + (double)v2.lo) * ((double)a.c.dt * (double)a.c.rdx2);
  gst(gp, more ? gld(gp) + w0 : w0);
  gst(gp + 1, more ? gld(gp + 1) + w1 : w1);
  gst(gp + 2, more ? gld(gp + 2) + w2 : w2);
}

template <int SCHEME, int TW, int TH>
__device__ __forceinline__ void adjoint_body(const AdjointArgs& a) {
  using Lay = AdjointSmem<TW, TH>;
  constexpr int G = Lay::G, W4 = Lay::W4, PH = Lay::PH, UH = Lay::UH, SH = Lay::SH, SW = Lay::SW;
  extern __shared__ __align__(16) float sm[];
  float* sP = sm + Lay::P_OFF;
  float* sUx = sm + Lay::UX_OFF;
  float* sUy = sm + Lay::UY_OFF;
  float* sMx = sm + Lay::MX_OFF;
  float* sMy = sm + Lay::MY_OFF;
  float* sLx = sm + Lay::LX_OFF;
  float* sLy = sm + Lay::LY_OFF;
  float* sF = sm + Lay::F_OFF;
  float* sDA = sm + Lay::DA_OFF;
  float* sDB = sm + Lay::DB_OFF;
  DFloat* sRed = reinterpret_cast<DFloat*>(sm + Lay::RED_OFF);
  const StepConsts& c = a.c;
  const int N = c.N, M = N - 1;
  const size_t NN = (size_t)N * N;
  const int j0 = blockIdx.x * TW, i0 = blockIdx.y * TH;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int tid = ty * 32 + tx;

  const float dt = c.dt;
  const float jscale = c.jscale;  // float32(dt * dx^2) = dJ/du_x / f_x
  const float nu = (a.theta_len == 3) ? gldg(a.theta + 2) : c.nu;
  const float cL = fmul(c.dtdx2, nu);                              // dt nu / dx^2
  const float cA = SCHEME == NSGB_SCHEME_CENTRAL ? c.cAc : c.cAu;  // dt / h
  const float t = fmul((float)a.step, dt);
  const float A = gldg(a.theta), B = gldg(a.theta + 1);

  const bool has_lam = a.lam != nullptr;
  const bool has_p = a.p != nullptr;
  // aligned float4 tile loads (a group never straddles the periodic wrap)
  if (has_p) {
    const float* __restrict__ pp = a.p;
    forflat<PH, G>(tid, [&](int r, int q) {
      const float4 v = gldg4(pp + (size_t)((i0 - 3 + r) & M) * N + ((j0 - 4 + 4 * q) & M));
      *reinterpret_cast<float4*>(sP + r * W4 + 4 * q) = v;
    });
  }
  {
    const float* __restrict__ u = a.u;
    const float* __restrict__ lam = a.lam;
    forflat<UH, G>(tid, [&](int r, int q) {
      const size_t g = (size_t)((i0 - 2 + r) & M) * N + ((j0 - 4 + 4 * q) & M);
      const int o = r * W4 + 4 * q;
      *reinterpret_cast<float4*>(sUx + o) = gldg4(u + g);
      *reinterpret_cast<float4*>(sUy + o) = gldg4(u + NN + g);
      const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(sMx + o) = has_lam ? gldg4(lam + g) : z;
      *reinterpret_cast<float4*>(sMy + o) = has_lam ? gldg4(lam + NN + g) : z;
    });
  }
  {
    const ForcingRow fr = forcing_time(A, B, t, c);
    if (tid < SH) {
      sF[tid] = forcing_fx((i0 - 1 + tid) & M, fr, c);
    } else if (tid >= 64 && tid < 64 + TH) {
      const int r = tid - 64;
      forcing_theta_grad((i0 + r) & M, fr, A, B, t, c, sDA[r], sDB[r]);
    }
  }
  __syncthreads();

  // mu = lambda - dt grad p on rows i0-2 .. i0+TH+1, columns j0-2 .. j0+TW+1
  if (has_p) {
    forflat<UH, TW + 4>(tid, [&](int r, int cc) {
      const int col = cc + 2;
      const float* P0 = sP + (r + 1) * W4 + col;
      const int o = r * W4 + col;
      sMx[o] = fused_proj(sMx[o], P0[W4], P0[-W4], c.cP);
      sMy[o] = fused_proj(sMy[o], P0[1], P0[-1], c.cP);
    });
    __syncthreads();
  }

  // theta sensitivities of the interior cells: float over a thread's few
  // cells, double-float across the block's threads, double across blocks and
  // steps (the nu term is a small difference of large contributions)
  float fA = 0.f, fB = 0.f, fN = 0.f;
  forflat<TH, TW>(tid, [&](int r, int cc) {
    const int o = (r + 2) * W4 + (cc + 4);
    const float w = fmaf(jscale, sUx[o], dt * sMx[o]);
    fA = fmaf(w, sDA[r], fA);
    fB = fmaf(w, sDB[r], fB);
    // Laplacian sums from neighbour differences: for a smooth field each
    // difference of close values is exact, so the small sum keeps its digits
    // (summing the neighbours first would cancel about two of them)
    const float ox = sUx[o], oy = sUy[o];
    const float lux = ((sUx[o - W4] - ox) + (sUx[o + W4] - ox)) + ((sUx[o + 1] - ox) + (sUx[o - 1] - ox));
    const float luy = ((sUy[o - W4] - oy) + (sUy[o + W4] - oy)) + ((sUy[o + 1] - oy) + (sUy[o - 1] - oy));
    fN = fmaf(sMx[o], lux, fmaf(sMy[o], luy, fN));
  });

  // lambda_s on rows i0-1 .. i0+TH, columns j0-1 .. j0+TW
  forflat<SH, SW>(tid, [&](int r, int cc) {
    const int o = (r + 1) * W4 + (cc + 3);
    const int n = o + W4, s = o - W4, e = o + 1, w = o - 1;  // i+1, i-1, j+1, j-1
    const AdjNbr Mx = {sMx[o], sMx[n], sMx[s], sMx[e], sMx[w]};
    const AdjNbr My = {sMy[o], sMy[n], sMy[s], sMy[e], sMy[w]};
    const AdjNbr Ux = {sUx[o], sUx[n], sUx[s], sUx[e], sUx[w]};
    const AdjNbr Uy = {sUy[o], sUy[n], sUy[s], sUy[e], sUy[w]};
    adjoint_cell<SCHEME>(Mx, My, Ux, Uy, cL, cA, jscale * sF[r], sLx[r * SW + cc], sLy[r * SW + cc]);
  });
  __syncthreads();

  {
    float* __restrict__ lo = a.lam_out;
    float* __restrict__ rhs = a.rhs;
    forflat<TH, TW>(tid, [&](int r, int cc) {
      const int o = (r + 1) * SW + (cc + 1);
      const size_t g = (size_t)(i0 + r) * N + (j0 + cc);
      gst(lo + g, sLx[o]);
      gst(lo + NN + g, sLy[o]);
      gst(rhs + g, fused_rhs(sLx[o + SW], sLx[o - SW], sLy[o + 1], sLy[o - 1], c.cD));
    });
  }

  const DFloat gA = warp_sum_df({fA, 0.f});
  const DFloat gB = warp_sum_df({fB, 0.f});
  const DFloat gN = warp_sum_df({fN, 0.f});
  if (tx == 0) {
    sRed[ty] = gA;
    sRed[8 + ty] = gB;
    sRed[16 + ty] = gN;
  }
  __syncthreads();
  if (ty == 0) {
    const DFloat z = {0.f, 0.f};
    const DFloat v0 = warp_sum_df(tx < 8 ? sRed[tx] : z);
    const DFloat v1 = warp_sum_df(tx < 8 ? sRed[8 + tx] : z);
    const DFloat v2 = warp_sum_df(tx < 8 ? sRed[16 + tx] : z);
    if (tx == 0) {
      add_theta_partials(a, blockIdx.y * gridDim.x + blockIdx.x, v0, v1, v2);
    }
  }
}

// Tiles at least 64 wide: four cells per thread, as the wide forward tiles
// (nsgb_stencil_body.cuh), asynchronous loads, 16-byte shared-memory accesses
// and stores: shared-memory instructions bound the one-cell body.  A forward and
// an adjoint step at the default tile, N = 256 20.0 -> 19.5 us, 512 27.6 -> 26.5;
// at 1024 in 128 x 8 tiles 50.1 -> 47.5 (its default are the row bands below).
template <int TW, int TH>
struct Adjoint4Smem {
  static constexpr int G = TW / 4 + 2;        // groups per row
  static constexpr int W4 = 4 * G;
  static constexpr int PH = TH + 6, UH = TH + 4, SH = TH + 2;
  static constexpr int NT = tile_threads<TW, TH>();
  static constexpr int P_OFF = 4;                     // PH rows (4 floats before: the first row's left neighbour)
  static constexpr int UX_OFF = P_OFF + PH * W4;      // UH rows each
  static constexpr int UY_OFF = UX_OFF + UH * W4;
  static constexpr int MX_OFF = UY_OFF + UH * W4;
  static constexpr int MY_OFF = MX_OFF + UH * W4;
  static constexpr int LX_OFF = MY_OFF + UH * W4;     // SH rows each
  static constexpr int LY_OFF = LX_OFF + SH * W4;
  static constexpr int F_OFF = LY_OFF + SH * W4 + 4;  // fx of the SH rows
  static constexpr int DA_OFF = F_OFF + SH;           // dfx/dA, dfx/dB of the TH rows
  static constexpr int DB_OFF = DA_OFF + TH;
  static constexpr int RED_OFF = (DB_OFF + TH + 1) & ~1;  // 3 x 8 double-floats
  static constexpr size_t BYTES = (size_t)RED_OFF * sizeof(float) + 24 * sizeof(DFloat);
  static_assert(NT % 32 == 0 && NT <= 256 && NT >= 64 + TH && SH <= 64, "threads");
};

template <int SCHEME, int TW, int TH>
__device__ __forceinline__ void adjoint4_body(const AdjointArgs& a) {
  using Lay = Adjoint4Smem<TW, TH>;
  constexpr int G = Lay::G, W4 = Lay::W4, PH = Lay::PH, UH = Lay::UH, SH = Lay::SH, NT = Lay::NT;
  extern __shared__ __align__(16) float sm[];
  float* sP = sm + Lay::P_OFF;
  float* sUx = sm + Lay::UX_OFF;
  float* sUy = sm + Lay::UY_OFF;
  float* sMx = sm + Lay::MX_OFF;
  float* sMy = sm + Lay::MY_OFF;
  float* sLx = sm + Lay::LX_OFF;
  float* sLy = sm + Lay::LY_OFF;
  float* sF = sm + Lay::F_OFF;
  float* sDA = sm + Lay::DA_OFF;
  float* sDB = sm + Lay::DB_OFF;
  DFloat* sRed = reinterpret_cast<DFloat*>(sm + Lay::RED_OFF);
  const StepConsts& c = a.c;
  const int N = c.N, M = N - 1;
  const size_t NN = (size_t)N * N;
  const int j0 = blockIdx.x * TW, i0 = blockIdx.y * TH;
  const int tid = threadIdx.x;
  const bool has_lam = a.lam != nullptr;
  const bool has_p = a.p != nullptr;

#pragma unroll
  for (int e = tid; e < UH * G; e += NT) {
    const int r = e / G, q = e % G;
    const size_t g = (size_t)((i0 - 2 + r) & M) * N + ((j0 - 4 + 4 * q) & M);
    copy16(sUx + 4 * e, a.u + g);
    copy16(sUy + 4 * e, a.u + NN + g);
    if (has_lam) {
      copy16(sMx + 4 * e, a.lam + g);
      copy16(sMy + 4 * e, a.lam + NN + g);
    } else {
      *reinterpret_cast<float4*>(sMx + 4 * e) = make_float4(0.f, 0.f, 0.f, 0.f);
      *reinterpret_cast<float4*>(sMy + 4 * e) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  if (has_p) {
#pragma unroll
    for (int e = tid; e < PH * G; e += NT) {
      const int r = e / G, q = e % G;
      copy16(sP + 4 * e, a.p + (size_t)((i0 - 3 + r) & M) * N + ((j0 - 4 + 4 * q) & M));
    }
  }
  const float dt = c.dt;
  const float jscale = c.jscale;  // float32(dt * dx^2) = dJ/du_x / f_x
  {
    const float t = fmul((float)a.step, dt);
    const float A = gldg(a.theta), B = gldg(a.theta + 1);
    const ForcingRow fr = forcing_time(A, B, t, c);
    if (tid < SH)
      sF[tid] = forcing_fx((i0 - 1 + tid) & M, fr, c);
    else if (tid >= 64 && tid < 64 + TH)
      forcing_theta_grad((i0 + tid - 64) & M, fr, A, B, t, c, sDA[tid - 64], sDB[tid - 64]);
  }
  const float nu = (a.theta_len == 3) ? gldg(a.theta + 2) : c.nu;
  const float cL = fmul(c.dtdx2, nu);                              // dt nu / dx^2
  const float cA = SCHEME == NSGB_SCHEME_CENTRAL ? c.cAc : c.cAu;  // dt / h
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();

  // mu = lambda - dt grad p on rows i0-2 .. i0+TH+1
  if (has_p) {
    project4<UH, G, NT>(sMx, sMy, sP, c.cP, tid);
    __syncthreads();
  }

  // lambda_s on rows i0-1 .. i0+TH
#pragma unroll 1
  for (int e = tid; e < SH * G; e += NT) {
    struct Cells {
      float s[4], o[6], n[4];
      __device__ __forceinline__ AdjNbr at(int k) const { return {o[k + 1], n[k], s[k], o[k + 2], o[k]}; }
    } mx, my, ux, uy;
    auto cells = [&](const float* f, Cells& d) {  // row e / G of f: one row up
      get4(f + 4 * e, d.s);
      get6(f + 4 * e + W4, d.o);
      get4(f + 4 * e + 2 * W4, d.n);
    };
    cells(sMx, mx);
    cells(sMy, my);
    cells(sUx, ux);
    cells(sUy, uy);
    const float fterm = jscale * sF[e / G];
    float lx[4], ly[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      adjoint_cell<SCHEME>(mx.at(k), my.at(k), ux.at(k), uy.at(k), cL, cA, fterm, lx[k], ly[k]);
    set4(sLx + 4 * e, lx);
    set4(sLy + 4 * e, ly);
  }

  // theta sensitivities of the thread's own cells (adjoint_body), summed in
  // double-float from the first cell on: dJ/dnu is a small difference of large
  // terms (the sums' rounding in float over two cells showed in it; the step
  // took the same time)
  const int r = tid / (TW / 4), q = tid % (TW / 4) + 1;
  DFloat vA, vB, vN;
  {
    const int o = (r + 2) * W4 + 4 * q;
    float mx[4], my[4], ux[6], uy[6], us[4], un[4], vs[4], vn[4];
    get4(sMx + o, mx);
    get4(sMy + o, my);
    get6(sUx + o, ux);
    get4(sUx + o - W4, us);
    get4(sUx + o + W4, un);
    get6(sUy + o, uy);
    get4(sUy + o - W4, vs);
    get4(sUy + o + W4, vn);
    float fA[4], fB[4], fN[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float ox = ux[k + 1], oy = uy[k + 1];
      const float w = fmaf(jscale, ox, dt * mx[k]);
      fA[k] = w * sDA[r];
      fB[k] = w * sDB[r];
      const float lux = ((us[k] - ox) + (un[k] - ox)) + ((ux[k + 2] - ox) + (ux[k] - ox));
      const float luy = ((vs[k] - oy) + (vn[k] - oy)) + ((uy[k + 2] - oy) + (uy[k] - oy));
      fN[k] = fmaf(mx[k], lux, my[k] * luy);
    }
    auto sum4 = [](const float (&f)[4]) {
      return df_add(two_sum(f[0], f[1]), two_sum(f[2], f[3]));
    };
    vA = sum4(fA);
    vB = sum4(fB);
    vN = sum4(fN);
  }
  const int lane = tid & 31;
  // lanes 0-7: A, 16-23: B, 8-15 and 24-31: nu
  DFloat v = fold<8>(fold<16>(vA, vB, lane), fold1(vN, 16), lane);
  v = fold1(fold1(fold1(v, 4), 2), 1);
  if (lane % 8 == 0 && lane < 24) sRed[(lane == 0 ? 0 : lane == 16 ? 8 : 16) + tid / 32] = v;
  __syncthreads();

  const size_t g = (size_t)(i0 + r) * N + (j0 - 4 + 4 * q);
  const int os = (r + 1) * W4 + 4 * q;
  float x[4], y[4];
  get4(sLx + os, x);
  get4(sLy + os, y);
  gst4(a.lam_out + g, make_float4(x[0], x[1], x[2], x[3]));
  gst4(a.lam_out + NN + g, make_float4(y[0], y[1], y[2], y[3]));
  gst4(a.rhs + g, rhs4<W4>(sLx + os, sLy + os, c.cD));
  if (tid < 32) {
    DFloat s = tid < 24 && tid % 8 < NT / 32 ? sRed[tid] : DFloat{0.f, 0.f};
    s = fold1(fold1(fold1(s, 4), 2), 1);  // lanes 0, 8, 16: A, B, nu
    const DFloat s1 = {__shfl_sync(0xffffffffu, s.hi, 8), __shfl_sync(0xffffffffu, s.lo, 8)};
    const DFloat s2 = {__shfl_sync(0xffffffffu, s.hi, 16), __shfl_sync(0xffffffffu, s.lo, 16)};
    if (tid == 0) add_theta_partials(a, blockIdx.y * gridDim.x + blockIdx.x, s, s1, s2);
  }
}

template <int SCHEME, int TW, int TH>
__global__ void __launch_bounds__((tile_threads<TW, TH>())) k_adjoint(const AdjointArgs a) {
  if constexpr (wide_tile<TW>())
    adjoint4_body<SCHEME, TW, TH>(a);
  else
    adjoint_body<SCHEME, TW, TH>(a);
}
// Batched form: blockIdx.z selects the solve's arguments.
template <int SCHEME, int TW, int TH>
__global__ void __launch_bounds__((tile_threads<TW, TH>())) k_adjoint_b(const AdjointArgs* __restrict__ tab) {
  if constexpr (wide_tile<TW>())
    adjoint4_body<SCHEME, TW, TH>(tab[blockIdx.z]);
  else
    adjoint_body<SCHEME, TW, TH>(tab[blockIdx.z]);
}

// a: the shape, scheme and N of the launch; tab (device, count entries) or
// nullptr for the single launch with a itself.
template <int SCHEME, int TW, int TH>
static cudaError_t launch_adjoint_t(const AdjointArgs& a, const AdjointArgs* tab, int count, cudaStream_t st) {
  const cudaError_t e = tab ? raise_smem_limit(k_adjoint_b<SCHEME, TW, TH>) : raise_smem_limit(k_adjoint<SCHEME, TW, TH>);
  if (e != cudaSuccess) return e;
  const dim3 grid(a.c.N / TW, a.c.N / TH, tab ? count : 1);
  const dim3 block = wide_tile<TW>() ? dim3(tile_threads<TW, TH>()) : dim3(32, 8);
  const size_t smem = wide_tile<TW>() ? Adjoint4Smem<TW, TH>::BYTES : AdjointSmem<TW, TH>::BYTES;
  if (tab)
    k_adjoint_b<SCHEME, TW, TH><<<grid, block, smem, st>>>(tab);
  else
    k_adjoint<SCHEME, TW, TH><<<grid, block, smem, st>>>(a);
  return cudaGetLastError();
}

template <int SCHEME>
static cudaError_t launch_adjoint_s(const AdjointArgs& a, const AdjointArgs* tab, int count, cudaStream_t st) {
#define NSGB_TILE_CASE(W, H) \
  if (a.tw == W && a.th == H) return launch_adjoint_t<SCHEME, W, H>(a, tab, count, st);
  NSGB_STENCIL_TILES(NSGB_TILE_CASE)
#undef NSGB_TILE_CASE
  return cudaErrorInvalidValue;
}

// ------------------------------------------------------ row-streaming --
// The adjoint step marched down row bands, as the forward row kernel does
// (nsgb_rows.cuh): thread g owns four columns and at iteration t
//   - forms mu(t) = lambda_{s+1}(t) - dt grad p from p rows t-1, t, t+1,
//   - forms lambda_s(t-1) from mu rows t-2, t-1, t (registers), the edge
//     values of mu(t-1) of the neighbouring groups and u rows t-2 .. t (ring),
//     and adds the theta partials of row t-1,
//   - writes lambda_s(t-2) and rhs(t-2) = div(lambda_s)/dt.
// p, lambda_{s+1} and u_s stream through shared-memory rings by asynchronous
// copies kAhead rows ahead; the cells use the tiled kernel's arithmetic
// (adjoint_cell), so lambda_s and rhs have the same bits.
namespace adjrows {
constexpr int F_MX = 0, F_MY = 1, F_LY = 2;  // exchanged fields
constexpr int kAhead = 3;                    // rows copied ahead of use
constexpr int kPRing = 8;                    // p rows t-1 .. t+1+kAhead
constexpr int kLRing = 4;                    // lambda rows t .. t+kAhead
constexpr int kURing = 8;                    // u rows t-2 .. t+kAhead
static_assert(kPRing >= kAhead + 3 && kLRing >= kAhead + 1 && kURing >= kAhead + 3, "ring depth");
constexpr int kMaxWarps = 32;
// rings, edges [2 slots][3 fields][2 sides][G], f_x of RH + 2 rows, dfx/dA and
// dfx/dB of RH rows, per-warp double-float partials
inline size_t smem_bytes(int N, int W, int RH) {
  return sizeof(float) * ((size_t)(kPRing + 2 * kLRing + 2 * kURing) * rows::ring_stride(W) +
                          (size_t)12 * rows::groups(N, W) + (RH + 2) + 2 * RH) +
         sizeof(DFloat) * 3 * kMaxWarps;
}
}  // namespace adjrows

template <int SCHEME>
__device__ __forceinline__ void adjoint_rows_body(const AdjointArgs& a) {
  using namespace rows;
  using adjrows::kAhead;
  using adjrows::kLRing;
  using adjrows::kPRing;
  using adjrows::kURing;
  using adjrows::F_LY;
  using adjrows::F_MX;
  using adjrows::F_MY;
  const StepConsts& c = a.c;
  const int N = c.N, M = N - 1;
  const size_t NN = (size_t)N * N;
  const int W = band_width(N, a.tw);
  const bool wrap = (W == N);
  const int G = groups(N, W);
  const int RH = a.th;
  const int r0 = blockIdx.y * RH;
  const int r1 = min(r0 + RH, N);
  const int j0 = blockIdx.x * W;
  const int tid = threadIdx.x;
  const bool active = tid < G;
  const int g = active ? tid : G - 1;  // idle lanes shadow the last group
  const int col = wrap ? 4 * g : ((j0 - 4 + 4 * g) & M);
  const bool store = active && (wrap || (g >= 1 && g <= G - 2));
  const int gl = g == 0 ? (wrap ? G - 1 : 0) : g - 1;
  const int gr = g == G - 1 ? (wrap ? 0 : G - 1) : g + 1;
  const int RS = ring_stride(W);
  const int bi = 4 + 4 * g + (wrap ? 4 : 0);  // the group's first column in a ring row

  extern __shared__ __align__(16) float sm[];
  float* sP = sm;                   // [kPRing][RS]
  float* sLX = sP + kPRing * RS;    // [kLRing][RS]
  float* sLY = sLX + kLRing * RS;   // [kLRing][RS]
  float* sUX = sLY + kLRing * RS;   // [kURing][RS]
  float* sUY = sUX + kURing * RS;   // [kURing][RS]
  float* sE = sUY + kURing * RS;    // [slot][field][side][G]
  float* sF = sE + 12 * G;          // f_x of rows r0-1 .. r1
  float* sDA = sF + RH + 2;         // dfx/dA of rows r0 .. r1-1
  float* sDB = sDA + RH;            // dfx/dB
  DFloat* sRed = reinterpret_cast<DFloat*>(sDB + RH);  // [3][kMaxWarps]
  auto edge = [&](int slot, int f, int side) { return sE + ((slot * 3 + f) * 2 + side) * G; };

  const float dt = c.dt;
  const float jscale = c.jscale;
  const float nu = (a.theta_len == 3) ? gldg(a.theta + 2) : c.nu;
  const float cL = fmul(c.dtdx2, nu);
  const float cA = SCHEME == NSGB_SCHEME_CENTRAL ? c.cAc : c.cAu;
  const float tf = fmul((float)a.step, dt);
  const float A = gldg(a.theta), B = gldg(a.theta + 1);
  {
    const ForcingRow fr = forcing_time(A, B, tf, c);
    for (int k = tid; k < r1 - r0 + 2; k += blockDim.x) sF[k] = forcing_fx((r0 - 1 + k) & M, fr, c);
    for (int k = tid; k < r1 - r0; k += blockDim.x) forcing_theta_grad((r0 + k) & M, fr, A, B, tf, c, sDA[k], sDB[k]);
  }

  const bool has_p = a.p != nullptr;
  const bool has_lam = a.lam != nullptr;
  const uint64_t pol = evict_first_policy();
  // one copy group: p row `pr` (if do_p), lambda and u rows `lr` (if do_lu)
  auto issue = [&](int pr, bool do_p, int lr, bool do_lu) {
    if (do_p && has_p) copy_row(sP + (pr & (kPRing - 1)) * RS, a.p, pr, N, M, wrap, active, tid, G, bi, col, pol);
    if (do_lu) {
      if (has_lam && active) {  // only the group's own columns of lambda are read
        const size_t o = (size_t)(lr & M) * N + col;
        cp16(sLX + (lr & (kLRing - 1)) * RS + bi, a.lam + o, pol);
        cp16(sLY + (lr & (kLRing - 1)) * RS + bi, a.lam + NN + o, pol);
      }
      copy_row(sUX + (lr & (kURing - 1)) * RS, a.u, lr, N, M, wrap, active, tid, G, bi, col, pol);
      copy_row(sUY + (lr & (kURing - 1)) * RS, a.u + NN, lr, N, M, wrap, active, tid, G, bi, col, pol);
    }
    cp_commit();
  };
  // prologue: p rows r0-3, r0-2, then the groups of iterations r0-2-kAhead ..
  // r0-3 (p rows r0-1 .., lambda and u rows r0-2 ..); wait for those of
  // iteration r0-2
  issue(r0 - 3, true, 0, false);
  issue(r0 - 2, true, 0, false);
#pragma unroll
  for (int k = kAhead; k >= 1; --k) issue(r0 - 1 - k + kAhead, true, r0 - 2 - k + kAhead, true);
  cp_wait<kAhead - 1>();
  __syncthreads();

  // registers entering iteration t: mu rows t-1, t-2; lambda_s x rows t-3,
  // t-2 and y row t-2
  float m1x[4] = {0, 0, 0, 0}, m1y[4] = {0, 0, 0, 0}, m2x[4] = {0, 0, 0, 0}, m2y[4] = {0, 0, 0, 0};
  float lx3[4] = {0, 0, 0, 0}, lx2[4] = {0, 0, 0, 0}, ly2[4] = {0, 0, 0, 0};
  // theta partials: float over a row's four cells, double-float over rows
  DFloat gA = {0.f, 0.f}, gB = {0.f, 0.f}, gN = {0.f, 0.f};
  float* __restrict__ lo_x = a.lam_out;
  float* __restrict__ lo_y = a.lam_out + NN;
  float* __restrict__ rhs_g = a.rhs;
#pragma unroll 1
  for (int t = r0 - 2; t <= r1 + 1; ++t) {
    const int rs = (t - 1) & 1, ws = t & 1;
    issue(t + 1 + kAhead, true, t + kAhead, true);

    // mu(t) = lambda(t) - dt grad p
    float mx[4] = {0, 0, 0, 0}, my[4] = {0, 0, 0, 0};
    if (has_lam) {
      ld4s(sLX + (t & (kLRing - 1)) * RS + bi, mx);
      ld4s(sLY + (t & (kLRing - 1)) * RS + bi, my);
    }
    if (has_p) {
      float pm[4], pn[4], q[4];
      ld4s(sP + ((t - 1) & (kPRing - 1)) * RS + bi, pm);
      ld4s(sP + ((t + 1) & (kPRing - 1)) * RS + bi, pn);
      const float* pc = sP + (t & (kPRing - 1)) * RS + bi;
      ld4s(pc, q);
      const float P[6] = {pc[-1], q[0], q[1], q[2], q[3], pc[4]};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        mx[k] = fused_proj(mx[k], pn[k], pm[k], c.cP);
        my[k] = fused_proj(my[k], P[k + 2], P[k], c.cP);
      }
    }

    // lambda_s(t-1) and the theta partials of row t-1
    float lx1[4] = {0, 0, 0, 0}, ly1[4] = {0, 0, 0, 0};
    if (t >= r0) {
      const float* ucx = sUX + ((t - 1) & (kURing - 1)) * RS + bi;
      const float* ucy = sUY + ((t - 1) & (kURing - 1)) * RS + bi;
      float cx[4], cy[4], nx[4], ny[4], sx[4], sy[4];
      ld4s(ucx, cx);
      ld4s(ucy, cy);
      ld4s(sUX + (t & (kURing - 1)) * RS + bi, nx);
      ld4s(sUY + (t & (kURing - 1)) * RS + bi, ny);
      ld4s(sUX + ((t - 2) & (kURing - 1)) * RS + bi, sx);
      ld4s(sUY + ((t - 2) & (kURing - 1)) * RS + bi, sy);
      const float UX[6] = {ucx[-1], cx[0], cx[1], cx[2], cx[3], ucx[4]};
      const float UY[6] = {ucy[-1], cy[0], cy[1], cy[2], cy[3], ucy[4]};
      const float MX[6] = {edge(rs, F_MX, 1)[gl], m1x[0], m1x[1], m1x[2], m1x[3], edge(rs, F_MX, 0)[gr]};
      const float MY[6] = {edge(rs, F_MY, 1)[gl], m1y[0], m1y[1], m1y[2], m1y[3], edge(rs, F_MY, 0)[gr]};
      const float fterm = jscale * sF[t - r0];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const AdjNbr Mx = {MX[k + 1], mx[k], m2x[k], MX[k + 2], MX[k]};
        const AdjNbr My = {MY[k + 1], my[k], m2y[k], MY[k + 2], MY[k]};
        const AdjNbr Ux = {UX[k + 1], nx[k], sx[k], UX[k + 2], UX[k]};
        const AdjNbr Uy = {UY[k + 1], ny[k], sy[k], UY[k + 2], UY[k]};
        adjoint_cell<SCHEME>(Mx, My, Ux, Uy, cL, cA, fterm, lx1[k], ly1[k]);
      }
      if (store && t - 1 >= r0 && t - 1 < r1) {
        const float dA = sDA[t - 1 - r0], dB = sDB[t - 1 - r0];
        float fA = 0.f, fB = 0.f, fN = 0.f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const float ox = UX[k + 1], oy = UY[k + 1];
          const float w = fmaf(jscale, ox, dt * MX[k + 1]);
          fA = fmaf(w, dA, fA);
          fB = fmaf(w, dB, fB);
          // Laplacian sums from neighbour differences (the tiled kernel's order)
          const float lux = ((sx[k] - ox) + (nx[k] - ox)) + ((UX[k + 2] - ox) + (UX[k] - ox));
          const float luy = ((sy[k] - oy) + (ny[k] - oy)) + ((UY[k + 2] - oy) + (UY[k] - oy));
          fN = fmaf(MX[k + 1], lux, fmaf(MY[k + 1], luy, fN));
        }
        gA = df_add(gA, {fA, 0.f});
        gB = df_add(gB, {fB, 0.f});
        gN = df_add(gN, {fN, 0.f});
      }
    }

    // lambda_s(t-2) and rhs(t-2)
    if (t >= r0 + 2 && store) {
      const float Y2[6] = {edge(rs, F_LY, 1)[gl], ly2[0], ly2[1], ly2[2], ly2[3], edge(rs, F_LY, 0)[gr]};
      float rh[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) rh[k] = fused_rhs(lx1[k], lx3[k], Y2[k + 2], Y2[k], c.cD);
      const size_t o = (size_t)((t - 2) & M) * N + col;
      st4_stream(lo_x, o, lx2);
      st4_stream(lo_y, o, ly2);
      st4(rhs_g, o, rh);
    }

    // edge values for the next iteration: mu(t), lambda_s y(t-1)
    if (active) {
      edge(ws, F_MX, 0)[g] = mx[0];
      edge(ws, F_MX, 1)[g] = mx[3];
      edge(ws, F_MY, 0)[g] = my[0];
      edge(ws, F_MY, 1)[g] = my[3];
      edge(ws, F_LY, 0)[g] = ly1[0];
      edge(ws, F_LY, 1)[g] = ly1[3];
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      m2x[k] = m1x[k];
      m2y[k] = m1y[k];
      m1x[k] = mx[k];
      m1y[k] = my[k];
      lx3[k] = lx2[k];
      lx2[k] = lx1[k];
      ly2[k] = ly1[k];
    }
    cp_wait<kAhead - 1>();  // the rows of iteration t+1 have landed
    __syncthreads();
  }
  cp_wait<0>();

  // theta partials of the CTA: double-float across threads
  gA = warp_sum_df(gA);
  gB = warp_sum_df(gB);
  gN = warp_sum_df(gN);
  const int lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  if (lane == 0) {
    sRed[warp] = gA;
    sRed[adjrows::kMaxWarps + warp] = gB;
    sRed[2 * adjrows::kMaxWarps + warp] = gN;
  }
  __syncthreads();
  if (warp == 0) {
    const DFloat z = {0.f, 0.f};
    const DFloat v0 = warp_sum_df(lane < nwarps ? sRed[lane] : z);
    const DFloat v1 = warp_sum_df(lane < nwarps ? sRed[adjrows::kMaxWarps + lane] : z);
    const DFloat v2 = warp_sum_df(lane < nwarps ? sRed[2 * adjrows::kMaxWarps + lane] : z);
    if (lane == 0) {
      add_theta_partials(a, blockIdx.y * gridDim.x + blockIdx.x, v0, v1, v2);
    }
  }
}

// Bands up to 512 columns (at most 160 threads) run three CTAs per SM, which
// the upwind kernel's 131 unbounded registers would cut to two; a band of 1024
// columns fills the SM's shared memory with its rings and keeps its registers.
constexpr int kNarrow = 512;
template <int SCHEME, bool NARROW>
__global__ void __launch_bounds__(NARROW ? kNarrow / 4 + 32 : NSGB_ADJ_ROWS_MAX_W / 4 + 32, NARROW ? 3 : 1)
    k_adjoint_rows(const AdjointArgs a) {
  adjoint_rows_body<SCHEME>(a);
}
template <int SCHEME, bool NARROW>
__global__ void __launch_bounds__(NARROW ? kNarrow / 4 + 32 : NSGB_ADJ_ROWS_MAX_W / 4 + 32, NARROW ? 3 : 1)
    k_adjoint_rows_b(const AdjointArgs* __restrict__ tab) {
  adjoint_rows_body<SCHEME>(tab[blockIdx.z]);
}

bool adjoint_rows_supported(int N, int tw, int th) {
  if (!stencil_rows_mode(tw) || (tw & (tw - 1)) != 0 || tw > NSGB_ADJ_ROWS_MAX_W) return false;
  return th >= 1 && th <= N && adjrows::smem_bytes(N, rows::band_width(N, tw), th) <= 227 * 1024;
}

template <int SCHEME, bool NARROW>
static cudaError_t launch_adjoint_rows_t(const AdjointArgs& a, const AdjointArgs* tab, int count, int W,
                                         cudaStream_t st) {
  const int N = a.c.N;
  const size_t smem = adjrows::smem_bytes(N, W, a.th);
  if (smem > 48 * 1024) {
    const cudaError_t e =
        tab ? raise_smem_limit(k_adjoint_rows_b<SCHEME, NARROW>) : raise_smem_limit(k_adjoint_rows<SCHEME, NARROW>);
    if (e != cudaSuccess) return e;
  }
  const dim3 grid(N / W, (N + a.th - 1) / a.th, tab ? count : 1);
  if (tab)
    k_adjoint_rows_b<SCHEME, NARROW><<<grid, rows::threads(N, W), smem, st>>>(tab);
  else
    k_adjoint_rows<SCHEME, NARROW><<<grid, rows::threads(N, W), smem, st>>>(a);
  return cudaGetLastError();
}

template <int SCHEME>
static cudaError_t launch_adjoint_rows(const AdjointArgs& a, const AdjointArgs* tab, int count, cudaStream_t st) {
  const int W = rows::band_width(a.c.N, a.tw);
  return W <= kNarrow ? launch_adjoint_rows_t<SCHEME, true>(a, tab, count, W, st)
                      : launch_adjoint_rows_t<SCHEME, false>(a, tab, count, W, st);
}

static cudaError_t launch_adjoint_any(const AdjointArgs& a, const AdjointArgs* tab, int count, cudaStream_t st) {
  if (stencil_rows_mode(a.tw))
    return a.scheme == NSGB_SCHEME_CENTRAL ? launch_adjoint_rows<NSGB_SCHEME_CENTRAL>(a, tab, count, st)
                                           : launch_adjoint_rows<NSGB_SCHEME_UPWIND>(a, tab, count, st);
  return a.scheme == NSGB_SCHEME_CENTRAL ? launch_adjoint_s<NSGB_SCHEME_CENTRAL>(a, tab, count, st)
                                         : launch_adjoint_s<NSGB_SCHEME_UPWIND>(a, tab, count, st);
}

cudaError_t launch_adjoint_stencil(const AdjointArgs& a, cudaStream_t st) {
  return launch_adjoint_any(a, nullptr, 1, st);
}

cudaError_t launch_adjoint_batch(const AdjointArgs& shape, const AdjointArgs* tab, int count, cudaStream_t st) {
  if (!tab || count < 1) return cudaErrorInvalidValue;
  return launch_adjoint_any(shape, tab, count, st);
}

// dJ/dtheta from the blocks' sums, in a fixed order.
__global__ void k_gsum(const double* __restrict__ gpart, int nblk, int theta_len, float* __restrict__ dJ) {
  __shared__ double red[3][256];
  const int t = threadIdx.x;
  double v[3] = {0, 0, 0};
  for (int b = t; b < nblk; b += 256)
    for (int k = 0; k < 3; ++k) v[k] += gld(gpart + 3 * (size_t)b + k);
  for (int k = 0; k < 3; ++k) red[k][t] = v[k];
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (t < h)
      for (int k = 0; k < 3; ++k) red[k][t] += red[k][t + h];
    __syncthreads();
  }
  if (t < theta_len) gst(dJ + t, (float)red[t][0]);
}

cudaError_t launch_gsum(const double* gpart, int nblk, int theta_len, float* dJ, cudaStream_t st) {
  k_gsum<<<1, 256, 0, st>>>(gpart, nblk, theta_len, dJ);
  return cudaGetLastError();
}

NSGB_BOUNDS_UNIT(adjoint, 3)

}  // namespace nsgb
