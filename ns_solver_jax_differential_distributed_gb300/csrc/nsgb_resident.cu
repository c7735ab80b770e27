// Resident solves of small grids: a whole rollout, or a whole gradient (forward
// steps, recomputed segments and adjoint steps), or any stretch of a batched
// gradient's operations, in one launch of one thread block cluster per solve.
//
// Up to N = 128 a step's four launches cost more than their work.  Here C CTAs,
// one cluster, own R = N / C rows each and keep the state (u* or lambda, the
// pressure, and the spectrum's pieces) in shared memory for all steps.
// Measured per step against four launches in a graph: N = 32 3.6 / 8.7 us, 64
// 3.5 / 8.5, 128 4.4 / 9.0; with the gradient, every state kept, 8.5 / 17.4, 8.4 /
// 17.7, 10.8 / 17.7.  At N = 256 sixteen CTAs have too many cells each (9.9 / 9.6
// and 24 / 19.6 us), so the four launches stay; N = 16 is less than one 32-wide
// tile of the sums below.  What bounds a step is latency: three cluster barriers
// of about 0.35 us and four transforms of a few warps of about 0.5 us; so two
// threads share a radix-16 butterfly (fft::half_butterfly; whole ones on half
// the threads took 9.4 us per step at N = 128, radix 8 5.2 against 4.6 and at N =
// 64 3.4 against 3.6), cells go four to a thread, and the objective and theta
// sums run in the warps that the row transforms leave
// idle.  A step is three phases between cluster barriers:
//   1. stencil of the own rows (halo rows are kept beside them), right-hand
//      side, forward row transforms, split into the two rows' half spectra and
//      sent to the CTAs that own the columns (distributed shared memory);
//   2. column transforms, multiplier, inverse column transforms, sent back to
//      the CTAs that own the rows;
//   3. inverse row transforms into the pressure rows, the first and last three
//      of them also sent to the neighbouring CTAs' halos.
// The CTAs of a cluster are scheduled together by the hardware, so the barriers
// need no residency check and no polling.
//
// The arithmetic is that of the batched kernels at the default 32 x 8 tiles,
// value for value: the same cell functions, the same radix-16 transforms,
// objective and theta partials summed per 32 x 8 tile in the same
// order, so a resident solve, an ensemble member and a batched gradient give
// the same bits.
#include <type_traits>

#include "nsgb_adjoint_cell.cuh"
#include "nsgb_fft_bodies.cuh"
#include "nsgb_internal.h"

namespace nsgb {
namespace res {

constexpr int kTileW = 32, kTileH = 8;  // tiles of the objective and theta partials

// R rows per CTA of N x N, radix-16 transforms with E values per thread.
template <int N, int R, int E>
struct Lay {
  static constexpr int M = N - 1, H = N / 2;
  static constexpr int C = N / R;             // CTAs per cluster
  static constexpr int NT = N * R >= 1024 ? 512 : 256;
  static constexpr int NW = NT / 32;
  static constexpr int T = N / E;             // threads of a transform
  static constexpr int PR = R / 2;            // row pairs
  static constexpr int KC = (H + 1 + C - 1) / C;             // columns of a CTA
  static constexpr int KP = (KC * T + 31) / 32 * 32 / T;     // ... in whole warps
  static constexpr int S = N / kTileW;        // column segments
  static constexpr int UP = (R + 4) * N;      // plane of u*, lambda or u with two halo rows each side
  static constexpr int PS = pair_stride<N>(); // float2 of an exchange buffer
  static constexpr int XBN = PR > KP ? PR : KP;
  static constexpr int A_OFF = 0;
  static constexpr int B_OFF = A_OFF + 2 * UP;
  static constexpr int P_OFF = B_OFF + 2 * UP;               // (R + 6) x N: three halo rows each side
  static constexpr int X_OFF = P_OFF + (R + 6) * N;          // exchange buffers
  static constexpr int CI_OFF = X_OFF + 2 * XBN * PS;        // columns received: KP x N float2
  static constexpr int RI_OFF = CI_OFF + 2 * KP * N;         // rows received: PR x (H + 1) float4
  static constexpr int J_OFF = RI_OFF + 4 * PR * (H + 1);    // objective sums of 32 cells: R x S
  static constexpr int F_OFF = J_OFF + R * S;                // f_x of rows r0-1 .. r0+R
  static constexpr int FWD = (F_OFF + R + 2 + 3) / 4 * 4;    // floats of a forward solve
  static constexpr int U_OFF = FWD;                          // gradient: u_s with two halo rows each side
  static constexpr int DA_OFF = U_OFF + 2 * UP;              // dfx/dA, dfx/dB of the own rows
  static constexpr int G_OFF = DA_OFF + 2 * R;               // theta sums of 32 cells: R x S x 3 double-floats
  static constexpr int GA_OFF = G_OFF + 6 * R * S;           // running sums per tile: 3 doubles
  static constexpr int GRAD = GA_OFF + 6 * (R / kTileH) * S;
  static_assert(R % kTileH == 0 && C >= 2 && C <= 16, "rows per CTA");
  static_assert(6 * (R / kTileH) * S <= NT, "one thread per tile sum in half a block");
  static_assert((PR * T) % 32 == 0 && T <= 32 && KP * T <= NT - 64, "transforms in whole warps, two warps to spare");
  static_assert(X_OFF % 4 == 0 && CI_OFF % 4 == 0 && RI_OFF % 4 == 0 && U_OFF % 4 == 0 && PS % 2 == 0, "alignment");
  static_assert(G_OFF % 2 == 0 && GA_OFF % 2 == 0, "alignment");
};

__device__ __forceinline__ unsigned cta_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Orders this CTA's stores (to any CTA's shared memory, and to global memory)
// before the other CTAs' reads after the barrier.
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// The CTAs of a cluster are placed together but need not have begun together:
// no store to another CTA's shared memory before it runs (arrive when a CTA
// begins, wait before its first such store), none after it has ended.
__device__ __forceinline__ void cluster_begin() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_begun() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t remote(uint32_t local, unsigned rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  return a;
}
__device__ __forceinline__ void st_remote(uint32_t a, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_remote2(uint32_t a, float x, float y) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void st_remote4(uint32_t a, float x, float y, float z, float w) {
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(x), "f"(y), "f"(z), "f"(w)
               : "memory");
}

template <int N, int R, int E, int SCHEME, bool GRAD>
struct Solve {
  using L = Lay<N, R, E>;
  static constexpr int M = L::M, H = L::H, C = L::C, NT = L::NT, NW = L::NW, T = L::T, PR = L::PR, S = L::S, UP = L::UP;
  const ResidentArgs& a;
  const StepConsts& c;
  float* sm;
  uint32_t sm32;
  unsigned rank, prev, next;
  int r0, tid, lane, warp;
  float *A, *B;  // planes x, y of the current and the next field
  float nu, cL;

  __device__ __forceinline__ Solve(const ResidentArgs& args, float* smem) : a(args), c(args.c), sm(smem) {
    sm32 = (uint32_t)__cvta_generic_to_shared(smem);
    rank = cta_rank();
    prev = (rank + C - 1) % C;
    next = (rank + 1) % C;
    r0 = (int)rank * R;
    tid = threadIdx.x;
    lane = tid & 31;
    warp = tid >> 5;
    A = sm + L::A_OFF;
    B = sm + L::B_OFF;
    nu = a.theta_len == 3 ? gldg(a.theta + 2) : c.nu;
    cL = fmul(c.dtdx2, nu);
  }
  __device__ __forceinline__ void swap() {
    float* t = A;
    A = B;
    B = t;
  }
  __device__ __forceinline__ uint32_t addr(const float* p) const { return sm32 + 4u * (uint32_t)(p - sm); }

  // ROWS rows of NPLANES planes of a global field, from row `first` (mod N),
  // into shared memory.  L2 loads: the field may be this launch's own.
  template <int ROWS, int NPLANES>
  __device__ __forceinline__ void load(float* dst, const float* src, int first) const {
    constexpr int Q = N / 4;
    for (int e = tid; e < ROWS * NPLANES * Q; e += NT) {
      const int pl = e / (ROWS * Q), r = (e / Q) % ROWS, q = e % Q;
      const float4 v = gldcg(reinterpret_cast<const float4*>(src + (size_t)pl * N * N +
                                                             (size_t)((first + r) & M) * N + 4 * q));
      *reinterpret_cast<float4*>(dst + (pl * ROWS + r) * N + 4 * q) = v;
    }
  }
  // Starts the copy of the state u_s of an adjoint step (and its halo rows).
  __device__ __forceinline__ void prefetch_u(const float* src, int line = __builtin_LINE()) const {
    constexpr int Q = N / 4, ROWS = R + 4;
    for (int e = tid; e < 2 * ROWS * Q; e += NT) {
      const int pl = e / (ROWS * Q), r = (e / Q) % ROWS, q = e % Q;
      const float* g = src + (size_t)pl * N * N + (size_t)((r0 - 2 + r) & M) * N + 4 * q;
      if (!bounds_ok(g, 16, line)) continue;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sm32 + 4u * (uint32_t)(L::U_OFF + pl * UP + r * N + 4 * q)),
                   "l"(g)
                   : "memory");
    }
  }
  // The own rows of both planes of a field to global memory.
  __device__ __forceinline__ void store_own(const float* f, float* dst) const {
    constexpr int Q = N / 4;
    for (int e = tid; e < 2 * R * Q; e += NT) {
      const int pl = e / (R * Q), r = (e / Q) % R, q = e % Q;
      gst4(dst + (size_t)pl * N * N + (size_t)(r0 + r) * N + 4 * q,
           *reinterpret_cast<const float4*>(f + pl * UP + (r + 2) * N + 4 * q));
    }
  }

  // f_x of rows r0-1 .. r0+R (and the sensitivities of the own rows) for a
  // step, by the last two warps, which no transform uses.
  __device__ __forceinline__ void forcing(int step, bool adjoint) {
    if (warp < NW - 2) return;
    const float t = a.t_from_step ? fmul((float)step, c.dt) : a.t_fixed;
    const float tA = gldg(a.theta), tB = gldg(a.theta + 1);
    const ForcingRow fr = forcing_time(tA, tB, t, c);
    if (warp == NW - 1) {
      if (lane < R + 2) sm[L::F_OFF + lane] = forcing_fx((r0 - 1 + lane) & M, fr, c);
    } else if (GRAD && adjoint && lane < R) {
      forcing_theta_grad((r0 + lane) & M, fr, tA, tB, t, c, sm[L::DA_OFF + lane], sm[L::DA_OFF + R + lane]);
    }
  }

  // Four consecutive values of a shared-memory row, and with the neighbours at
  // both ends (periodic).
  __device__ __forceinline__ static void get4(const float* row, int c4, float (&v)[4]) {
    const float4 w = *reinterpret_cast<const float4*>(row + c4);
    v[0] = w.x, v[1] = w.y, v[2] = w.z, v[3] = w.w;
  }
  __device__ __forceinline__ static void get6(const float* row, int c4, float (&v)[6]) {
    const float4 w = *reinterpret_cast<const float4*>(row + c4);
    v[0] = row[(c4 - 1) & M], v[1] = w.x, v[2] = w.y, v[3] = w.z, v[4] = w.w, v[5] = row[(c4 + 4) & M];
  }
  __device__ __forceinline__ static void set4(float* row, int c4, const float (&v)[4]) {
    *reinterpret_cast<float4*>(row + c4) = make_float4(v[0], v[1], v[2], v[3]);
  }

  // u* -> u (or lambda -> mu): the pending projection on the own rows and two
  // halo rows each side, in place.
  __device__ __forceinline__ void project() {
    const float* P = sm + L::P_OFF;
#pragma unroll
    for (int e = tid; e < UP / 4; e += NT) {
      const int r = e / (N / 4), c4 = e % (N / 4) * 4;
      float x[4], y[4], pn[4], pm[4], pc[6];
      get4(A + r * N, c4, x);
      get4(A + UP + r * N, c4, y);
      get4(P + (r + 2) * N, c4, pn);
      get4(P + r * N, c4, pm);
      get6(P + (r + 1) * N, c4, pc);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        x[k] = fused_proj(x[k], pn[k], pm[k], c.cP);
        y[k] = fused_proj(y[k], pc[k + 2], pc[k], c.cP);
      }
      set4(A + r * N, c4, x);
      set4(A + UP + r * N, c4, y);
    }
  }

  // Four values (x, y) of row rr - 1 + r0 of the next field: kept, and sent to
  // the neighbour that needs them as its outer halo row.
  __device__ __forceinline__ void put4(int rr, int c4, const float (&x)[4], const float (&y)[4]) {
    set4(B + (rr + 1) * N, c4, x);
    set4(B + UP + (rr + 1) * N, c4, y);
    // own row 1 is the previous CTA's row R + 1, own row R - 2 the next one's -2
    if (rr == 2 || rr == R - 1) {
      const uint32_t d = remote(addr(B + (rr == 2 ? R + 3 : 0) * N + c4), rr == 2 ? prev : next);
      st_remote4(d, x[0], x[1], x[2], x[3]);
      st_remote4(d + 4u * UP, y[0], y[1], y[2], y[3]);
    }
  }

  // Right-hand side div(next field)/dt of the own rows, as row pairs in the
  // exchange buffers.
  __device__ __forceinline__ void rhs_rows() {
    float2* X = reinterpret_cast<float2*>(sm + L::X_OFF);
#pragma unroll
    for (int e = tid; e < PR * N / 4; e += NT) {
      const int q = e / (N / 4), c4 = e % (N / 4) * 4;
      float x0[4], x1[4], x2[4], x3[4], y0[6], y1[6];
      const float* bx = B + (2 * q + 1) * N;
      get4(bx, c4, x0);
      get4(bx + N, c4, x1);
      get4(bx + 2 * N, c4, x2);
      get4(bx + 3 * N, c4, x3);
      get6(B + UP + (2 * q + 2) * N, c4, y0);
      get6(B + UP + (2 * q + 3) * N, c4, y1);
      float2* d = X + q * L::PS + pad(c4);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        d[k] = make_float2(fused_rhs(x2[k], x0[k], y0[k + 2], y0[k], c.cD),
                           fused_rhs(x3[k], x1[k], y1[k + 2], y1[k], c.cD));
    }
  }

  // What a step's idle warps sum while the row transforms run: nothing, the
  // objective or the theta sensitivities of the state in A.
  enum Sums { kNone, kObjective, kTheta };
  // Sums over 32 cells of a row each, by warps w0 and up.
  template <int KIND>
  __device__ __forceinline__ void sums(int w0) {
    if (KIND == kNone || warp < w0) return;
    const float* sF = sm + L::F_OFF;
#pragma unroll 2
    for (int i = warp - w0; i < R * S; i += NW - w0) {
      const int r = i / S, cc = i % S * kTileW + lane, o = (r + 2) * N + cc;
      if constexpr (KIND == kObjective) {
        const float v = warp_sum(fmul(A[o], sF[r + 1]));
        if (lane == 0) sm[L::J_OFF + i] = v;
      } else {
        const float* U = sm + L::U_OFF;
        const float* dA = sm + L::DA_OFF;
        const int e1 = (r + 2) * N + ((cc + 1) & M), w1 = (r + 2) * N + ((cc - 1) & M);
        const float mx = A[o], my = A[UP + o], ux = U[o], uy = U[UP + o];
        const float w = fmaf(c.jscale, ux, c.dt * mx);
        const float fA = fmaf(w, dA[r], 0.f), fB = fmaf(w, dA[R + r], 0.f);
        const float lux = ((U[o - N] - ux) + (U[o + N] - ux)) + ((U[e1] - ux) + (U[w1] - ux));
        const float luy = ((U[UP + o - N] - uy) + (U[UP + o + N] - uy)) + ((U[UP + e1] - uy) + (U[UP + w1] - uy));
        const float fN = fmaf(mx, lux, fmaf(my, luy, 0.f));
        // lanes 0-7: A, 16-23: B, 8-15 and 24-31: nu
        DFloat v = fold<8>(fold<16>({fA, 0.f}, {fB, 0.f}, lane), fold1({fN, 0.f}, 16), lane);
        v = fold1(fold1(fold1(v, 4), 2), 1);
        if (lane % 8 == 0 && lane < 24)
          reinterpret_cast<DFloat*>(sm + L::G_OFF)[i * 3 + (lane == 0 ? 0 : lane == 16 ? 1 : 2)] = v;
      }
    }
  }
  // ... and the tiles' sums of eight such rows (after a barrier): the partials
  // of step jstep, or the running theta sums (first: their first step).
  // By the upper half of the block, which the split after it needs least.
  template <int KIND>
  __device__ __forceinline__ void combine(int jstep, bool first) {
    const int t = tid - NT / 2;
    if (t < 0) return;
    if (KIND == kObjective && t < (R / kTileH) * S) {
      const int ty = t / S, tx = t % S;
      const float* v = sm + L::J_OFF + ty * kTileH * S + tx;
      const float s = ((v[0] + v[4 * S]) + (v[2 * S] + v[6 * S])) + ((v[S] + v[5 * S]) + (v[3 * S] + v[7 * S]));
      gst(a.jpart + (size_t)jstep * (N / kTileH * S) + (r0 / kTileH + ty) * S + tx, (double)s);
    }
    if (KIND == kTheta && t < (R / kTileH) * S * 3) {
      const int comp = t % 3, tile = t / 3, ty = tile / S, tx = tile % S;
      const DFloat* v = reinterpret_cast<const DFloat*>(sm + L::G_OFF) + (ty * kTileH * S + tx) * 3 + comp;
      constexpr int D = 3 * S;  // one row down
      const DFloat s = df_add(df_add(df_add(v[0], v[4 * D]), df_add(v[2 * D], v[6 * D])),
                              df_add(df_add(v[D], v[5 * D]), df_add(v[3 * D], v[7 * D])));
      double w = (double)s.hi + (double)s.lo;
      if (comp == 2) w *= (double)c.dt * (double)c.rdx2;
      double* acc = reinterpret_cast<double*>(sm + L::GA_OFF) + t;
      *acc = first ? w : *acc + w;
    }
  }

  // The Poisson solve of the right-hand side in the exchange buffers into the
  // pressure rows.  On the side: the sums of KIND (see combine), the forcing of
  // step fstep (>= 0) and the copy of u_next (gradients).
  template <int KIND>
  __device__ __forceinline__ void poisson(int jstep, bool first, int fstep, const float* u_next) {
    float2* X = reinterpret_cast<float2*>(sm + L::X_OFF);
    const int j = tid % T, y = tid / T;
    if (tid < PR * T) {
      float2 v[E];
      float2* sb = X + y * L::PS;
      fft::load_strided<T, E>(v, sb, j);
      __syncwarp();
      fft::block_fft<N, false, E, -1, 16>(v, sb, j, a.tw);
      fft::store_strided<T, E>(v, sb, j);
    } else {
      sums<KIND>(PR * T / 32);
    }
    __syncthreads();
    combine<KIND>(jstep, first);
    if (GRAD && u_next) prefetch_u(u_next);
    // split (rows_fwd_body) and send to the columns' owners
#pragma unroll
    for (int e = tid; e < PR * (H + 1); e += NT) {
      const int q = e % PR, k = e / PR;
      const float2 zk = X[q * L::PS + pad(k)], wk = X[q * L::PS + pad((N - k) & M)];
      const uint32_t d = remote(sm32 + 4u * (uint32_t)(L::CI_OFF + 2 * ((k / C) * N + r0 + 2 * q)), (unsigned)(k % C));
      st_remote4(d, zk.x + wk.x, zk.y - wk.y, zk.y + wk.y, wk.x - zk.x);
    }
    cluster_barrier();
    if (tid < L::KP * T) {
      const int k = y * C + (int)rank;
      const bool valid = y < L::KC && k <= H;
      const float2* ci = reinterpret_cast<const float2*>(sm + L::CI_OFF) + y * N;
      float2 v[E];
#pragma unroll
      for (int s = 0; s < E; ++s) v[s] = ci[j + s * T];
      float2* sb = X + y * L::PS;
      fft::block_fft<N, false, E, -1, 16>(v, sb, j, a.tw);
      const float k2y = gldg(a.k2 + (valid ? k : H));
      float g[E];
#pragma unroll
      for (int s = 0; s < E; ++s) g[s] = poisson_mult<true>(gldg(a.k2 + j + s * T), k2y, a.scale);
      fft::block_fft_scaled<N, true, E, -1, 16>(v, g, sb, j, a.tw);
      if (valid) {
#pragma unroll
        for (int s = 0; s < E; ++s) {
          const int i = j + s * T, lr = i % R;
          const uint32_t d = remote(
              sm32 + 4u * (uint32_t)(L::RI_OFF + 4 * ((lr / 2) * (H + 1) + k) + 2 * (lr & 1)), (unsigned)(i / R));
          st_remote2(d, v[s].x, v[s].y);
        }
      }
    }
    if (fstep >= 0) forcing(fstep, KIND == kTheta);
    cluster_barrier();
    float* P = sm + L::P_OFF;
    if (tid < PR * T) {
      // Z of the row pair (rows_inv_body), inverse transform, pressure rows
      const float4* ri = reinterpret_cast<const float4*>(sm + L::RI_OFF) + y * (H + 1);
      float2 v[E];
#pragma unroll
      for (int s = 0; s < E; ++s) {
        const int m = j + s * T, k = m <= H ? m : N - m;
        const float4 w = ri[k];
        v[s] = (k == 0 || k == H) ? make_float2(w.x, w.z)
               : m < H            ? make_float2(w.x - w.w, w.y + w.z)
                                  : make_float2(w.x + w.w, w.z - w.y);
      }
      fft::block_fft<N, true, E, -1, 16>(v, X + y * L::PS, j, a.tw);
#pragma unroll
      for (int s = 0; s < E; ++s) {
        P[(2 * y + 3) * N + j + s * T] = v[s].x;
        P[(2 * y + 4) * N + j + s * T] = v[s].y;
      }
    }
    __syncthreads();
    // the first three own rows to the previous CTA's halo, the last three to the next one's
#pragma unroll
    for (int e = tid; e < 6 * N / 4; e += NT) {
      const int h = e / (N / 4), c4 = e % (N / 4) * 4;
      float v[4];
      get4(P + (h < 3 ? 3 + h : R - 3 + h) * N, c4, v);  // h >= 3: own row R - 3 + (h - 3)
      const uint32_t d = remote(addr(P + (h < 3 ? R + 3 + h : h - 3) * N + c4), h < 3 ? prev : next);
      st_remote4(d, v[0], v[1], v[2], v[3]);
    }
    cluster_barrier();
  }

  // One forward step of the field in A (pending projection if has_p): u* of
  // the next state into B, its right-hand side into the exchange buffers.
  // u_out: the projected state.
  __device__ __forceinline__ void forward(bool has_p, float* u_out) {
    if (has_p) {
      project();
      __syncthreads();
    }
    const float* sF = sm + L::F_OFF;
    if (u_out) store_own(A, u_out);
#pragma unroll
    for (int e = tid; e < (R + 2) * N / 4; e += NT) {
      const int rr = e / (N / 4), c4 = e % (N / 4) * 4;
      float xs[4], xn[4], ys[4], yn[4], X[6], Y[6], x[4], y[4];
      get4(A + rr * N, c4, xs);
      get6(A + (rr + 1) * N, c4, X);
      get4(A + (rr + 2) * N, c4, xn);
      get4(A + UP + rr * N, c4, ys);
      get6(A + UP + (rr + 1) * N, c4, Y);
      get4(A + UP + (rr + 2) * N, c4, yn);
      const float cFx = fmul(c.dt, sF[rr]), cFy = fmul(c.dt, 0.0f);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float ox = X[k + 1], oy = Y[k + 1];
        x[k] = fused_ustar<SCHEME>(ox, xs[k], xn[k], X[k + 2], X[k], ox, oy, cL, cFx, c);
        y[k] = fused_ustar<SCHEME>(oy, ys[k], yn[k], Y[k + 2], Y[k], ox, oy, cL, cFy, c);
      }
      put4(rr, c4, x, y);
    }
    __syncthreads();
    rhs_rows();
    __syncthreads();
  }

  // One adjoint step: lambda_s into B from lambda_{s+1} in A and u_s, its
  // right-hand side into the exchange buffers.
  __device__ __forceinline__ void adjoint(bool has_p) {
    if (has_p) {
      project();
      __syncthreads();
    }
    const float* sF = sm + L::F_OFF;
    const float* U = sm + L::U_OFF;
    const float cA = SCHEME == NSGB_SCHEME_CENTRAL ? c.cAc : c.cAu;
#pragma unroll 1
    for (int e = tid; e < (R + 2) * N / 4; e += NT) {
      const int rr = e / (N / 4), c4 = e % (N / 4) * 4;
      struct Cells {
        float s[4], o[6], n[4];
        __device__ __forceinline__ AdjNbr at(int k) const { return {o[k + 1], n[k], s[k], o[k + 2], o[k]}; }
      } mx, my, ux, uy;
      auto cells = [&](const float* f, Cells& d) {
        get4(f + rr * N, c4, d.s);
        get6(f + (rr + 1) * N, c4, d.o);
        get4(f + (rr + 2) * N, c4, d.n);
      };
      cells(A, mx);
      cells(A + UP, my);
      cells(U, ux);
      cells(U + UP, uy);
      const float fterm = c.jscale * sF[rr];
      float lx[4], ly[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        adjoint_cell<SCHEME>(mx.at(k), my.at(k), ux.at(k), uy.at(k), cL, cA, fterm, lx[k], ly[k]);
      put4(rr, c4, lx, ly);
    }
    __syncthreads();
    rhs_rows();
    __syncthreads();
  }

  // ---- the schedule (nsgb_capi.cu: grad_op) ----
  enum Kind { kFwd, kRec, kAdj };
  struct Op {
    int kind, s, s0, s1;  // step; its segment [s0, s1) (recomputed and adjoint steps)
  };
  __device__ __forceinline__ Op segment(int seg) const {  // the first operation of a segment
    const int s0 = seg * a.every, s1 = min(a.steps, s0 + a.every);
    return {s1 - s0 > 1 ? kRec : kAdj, s0, s0, s1};  // a one-step segment's state is its checkpoint
  }
  __device__ __forceinline__ Op op_at(int k) const {
    if (k < a.steps) return {kFwd, k, 0, 0};
    k -= a.steps;
    for (int seg = (a.steps - 1) / a.every;; --seg) {
      Op o = segment(seg);
      const int len = o.s1 - o.s0, n = len > 1 ? 2 * len : 1;
      if (k >= n) {
        k -= n;
        continue;
      }
      if (len > 1 && k < len)
        o.s = o.s0 + k;
      else
        o.kind = kAdj, o.s = o.s1 - 1 - (len > 1 ? k - len : k);
      return o;
    }
  }
  __device__ __forceinline__ Op next_op(Op o) const {
    if (o.kind == kFwd) {
      if (++o.s < a.steps) return o;
      return segment((a.steps - 1) / a.every);
    }
    if (o.kind == kRec) {
      if (++o.s == o.s1) o.kind = kAdj, --o.s;
      return o;
    }
    if (--o.s >= o.s0) return o;
    return segment(o.s0 / a.every - 1);
  }
  // The buffers of a step's results, by parity (grad_fwd_args, grad_adj_args).
  __device__ __forceinline__ float* us_of(const Op& o) const {
    return (o.s - (o.kind == kRec ? o.s0 : 0)) % 2 == 0 ? a.usA : a.usB;
  }
  __device__ __forceinline__ float* lam_of(int s) const { return (a.steps - 1 - s) % 2 == 0 ? a.lamA : a.lamB; }
  __device__ __forceinline__ const float* u_of(const Op& o) const {  // u_s of an adjoint step
    return o.s1 - o.s0 == 1 ? a.ckpt + (size_t)(o.s0 / a.every) * 2 * N * N
                            : a.ustore + (size_t)(o.s - o.s0) * 2 * N * N;
  }

  // The field in A and the pressure to or from global memory.
  __device__ __forceinline__ void save(float* f, float* p) const {
    store_own(A, f);
    const float* P = sm + L::P_OFF;
    for (int e = tid; e < R * N; e += NT) gst(p + (size_t)r0 * N + e, P[3 * N + e]);
  }
  __device__ __forceinline__ void restore(const float* f, const float* p) {
    load<R + 4, 2>(A, f, r0 - 2);
    load<R + 6, 1>(sm + L::P_OFF, p, r0 - 3);
  }

  // Makes the state of operation o present; `before`: the kind of the operation
  // this launch ran before it, -1 if none.  The caller's next barrier publishes
  // it within the CTA.
  __device__ __forceinline__ void enter(const Op& o, int before, int prev_s) {
    if (o.kind == kFwd) {
      if (o.s == 0)
        load<R + 4, 2>(A, a.u0, r0 - 2);
      else
        restore(us_of({kFwd, o.s - 1, 0, 0}), a.p);
    } else if (o.kind == kRec) {
      if (before == kAdj) {  // lambda and its pressure wait in global memory
        save(lam_of(prev_s), a.padj);
        cluster_barrier();
      }
      if (o.s == o.s0)
        load<R + 4, 2>(A, a.ckpt + (size_t)(o.s0 / a.every) * 2 * N * N, r0 - 2);
      else
        restore(us_of({kRec, o.s - 1, o.s0, o.s1}), a.p);
    } else if (o.s == a.steps - 1) {
      for (int e = tid; e < 2 * UP; e += NT) A[e] = 0.f;
    } else if (before != kAdj) {
      restore(lam_of(o.s + 1), a.padj);
    }
    if (GRAD && o.kind == kAdj) prefetch_u(u_of(o));
    forcing(o.s, o.kind == kAdj);
  }

  __device__ __forceinline__ void project_final() const {
    const float* P = sm + L::P_OFF;
    for (int e = tid; e < R * N; e += NT) {
      const int r = e / N, cc = e % N, o = (r + 2) * N + cc;
      const float* p0 = P + (r + 3) * N;
      gst(a.u_final + (size_t)r0 * N + e, fused_proj(A[o], p0[N + cc], p0[cc - N], c.cP));
      gst(a.u_final + (size_t)N * N + (size_t)r0 * N + e,
          fused_proj(A[UP + o], p0[(cc + 1) & M], p0[(cc - 1) & M], c.cP));
    }
  }

  // Operations [op0, op1), in runs of one kind (one loop each: a loop over
  // operations of every kind cost 0.4 us per step).
  __device__ __forceinline__ void run() {
    if (a.op0 >= a.op1) return;
    cluster_begin();
    constexpr int NG = (R / kTileH) * S * 3;  // the CTA's running theta sums
    double* acc = reinterpret_cast<double*>(sm + L::GA_OFF);
    Op o = op_at(a.op0);
    if constexpr (GRAD) {
      // adjoint steps done by earlier launches
      if (o.kind != kFwd && a.steps - (o.kind == kRec ? o.s1 : o.s + 1) > 0)
        for (int e = tid; e < NG; e += NT) acc[e] = gld(a.gpart + (size_t)(r0 / kTileH) * S * 3 + e);
    }
    enter(o, -1, 0);
    cluster_begun();
    __syncthreads();
    int left = a.op1 - a.op0;
    if (o.kind == kFwd) {
      const int s1 = min(a.steps, o.s + left);
      left -= s1 - o.s;
      for (int s = o.s; s < s1; ++s) {
        forward(s > 0, (GRAD && s % a.every == 0) ? a.ckpt + (size_t)(s / a.every) * 2 * N * N : nullptr);
        poisson<kObjective>(s, false, s + 1 < s1 ? s + 1 : -1, nullptr);
        swap();
      }
      o.s = s1 - 1;
      if (s1 < a.steps) {
        if constexpr (GRAD) save(us_of(o), a.p);
        return;
      }
      if (a.u_final) project_final();
    }
    if constexpr (GRAD) {
      if (o.kind == kFwd) {
        if (!left) return;
        const Op nx = next_op(o);
        __syncthreads();  // the state is not overwritten under a reader
        enter(nx, kFwd, o.s);
        __syncthreads();
        o = nx;
      }
      for (;;) {
        if (o.kind == kRec) {
          const int s1 = min(o.s1, o.s + left);
          left -= s1 - o.s;
          for (int s = o.s; s < s1; ++s) {
            forward(s > o.s0, a.ustore + (size_t)(s - o.s0) * 2 * N * N);
            if (s + 1 < o.s1)
              poisson<kNone>(0, false, s + 1 < s1 ? s + 1 : -1, nullptr);
            else
              cluster_barrier();  // the neighbours' states are written
            swap();
          }
          o.s = s1 - 1;
        } else {
          // states kept one by one: one run through all segments
          const int low = max(o.s + 1 - left, a.every == 1 ? 0 : o.s0);
          left -= o.s + 1 - low;
          const float* u = u_of(o);
          for (int s = o.s; s >= low; --s) {
            const bool first = s == a.steps - 1;
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            adjoint(!first);
            u -= 2 * N * N;
            if (s > 0) {
              // the next adjoint step's state arrives during the Poisson solve
              poisson<kTheta>(0, first, s > low ? s - 1 : -1, s > low ? u : nullptr);
            } else {
              sums<kTheta>(0);
              __syncthreads();
              combine<kTheta>(0, first);
              if (a.dJdu0) store_own(B, a.dJdu0);
              cluster_barrier();  // the neighbours' halo rows have arrived: CTAs may end
            }
            swap();
          }
          o.s = low;
          if (a.every == 1) o.s0 = low;
        }
        if (!left) break;
        const Op nx = next_op(o);
        __syncthreads();  // the state is not overwritten under a reader
        enter(nx, o.kind, o.s);
        __syncthreads();
        o = nx;
      }
      // what the next launch takes up
      if (o.kind == kRec && o.s + 1 < o.s1) save(us_of(o), a.p);
      if (o.kind == kAdj && o.s > 0) save(lam_of(o.s), a.padj);
      __syncthreads();
      if (o.kind == kAdj || o.s1 < a.steps)
        for (int e = tid; e < NG; e += NT) gst(a.gpart + (size_t)(r0 / kTileH) * S * 3 + e, acc[e]);
    }
  }
};

template <int N, int R, int E, int SCHEME, bool GRAD>
__global__ void __launch_bounds__(Lay<N, R, E>::NT, 1) k_resident(const ResidentArgs a) {
  extern __shared__ __align__(16) float sm_res[];
  Solve<N, R, E, SCHEME, GRAD> s(a, sm_res);
  s.run();
}

// Gradients of several solves: cluster blockIdx.x / C takes the solve's entry.
template <int N, int R, int E, int SCHEME>
__global__ void __launch_bounds__(Lay<N, R, E>::NT, 1) k_resident_batch(const ResidentArgs* __restrict__ tab) {
  extern __shared__ __align__(16) float sm_res[];
  static_assert(std::is_trivially_copyable<ResidentArgs>::value && sizeof(ResidentArgs) % 16 == 0, "table entries");
  __shared__ uint4 raw[sizeof(ResidentArgs) / 16];
  const uint4* src = reinterpret_cast<const uint4*>(tab + blockIdx.x / Lay<N, R, E>::C);
  for (int e = threadIdx.x; e < (int)(sizeof(ResidentArgs) / 16); e += Lay<N, R, E>::NT) raw[e] = gld(src + e);
  __syncthreads();
  Solve<N, R, E, SCHEME, true> s(*reinterpret_cast<const ResidentArgs*>(raw), sm_res);
  s.run();
}

}  // namespace res

// Rows per CTA and values per transform thread of the resident kernel's instances.
#ifndef NSGB_RESIDENT
#define NSGB_RESIDENT(X) X(32, 16, 8) X(64, 8, 8) X(128, 8, 8)
#endif

// Configuration of `count` clusters of an instance; attr outlives it.
template <class L>
static cudaLaunchConfig_t cluster_config(bool grad, int count, cudaLaunchAttribute* attr, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(L::C * count);
  cfg.blockDim = dim3(L::NT);
  cfg.dynamicSmemBytes = sizeof(float) * (grad ? L::GRAD : L::FWD);
  cfg.stream = st;
  attr->id = cudaLaunchAttributeClusterDimension;
  attr->val.clusterDim.x = L::C;
  attr->val.clusterDim.y = 1;
  attr->val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cfg;
}

// Prepares a kernel for its clusters and asks how many of them the device runs
// at once (0: none).
template <class L, class K>
static int probe_clusters(K* kernel, bool grad) {
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cluster_config<L>(grad, 1, &attr, nullptr);
  int n = 0;
  if (raise_smem_limit(kernel) != cudaSuccess ||
      (L::C > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
      cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

template <int N, int R, int E, int SCHEME, bool GRAD>
static cudaError_t launch_resident_t(const ResidentArgs& a, cudaStream_t st) {
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cluster_config<res::Lay<N, R, E>>(GRAD, 1, &attr, st);
  return cudaLaunchKernelEx(&cfg, res::k_resident<N, R, E, SCHEME, GRAD>, a);
}
template <int N, int R, int E, int SCHEME>
static cudaError_t launch_resident_batch_t(const ResidentArgs* tab, int count, cudaStream_t st) {
  cudaLaunchAttribute attr;
  const cudaLaunchConfig_t cfg = cluster_config<res::Lay<N, R, E>>(true, count, &attr, st);
  return cudaLaunchKernelEx(&cfg, res::k_resident_batch<N, R, E, SCHEME>, tab);
}

bool resident_size(int N) {
#define NSGB_RESIDENT_CASE(NN, R, E) if (N == NN) return true;
  NSGB_RESIDENT(NSGB_RESIDENT_CASE)
#undef NSGB_RESIDENT_CASE
  return false;
}

template <int N, int R, int E, int SCHEME>
static int probe_instances() {
  using L = res::Lay<N, R, E>;
  const int f = probe_clusters<L>(res::k_resident<N, R, E, SCHEME, false>, false);
  const int g = probe_clusters<L>(res::k_resident<N, R, E, SCHEME, true>, true);
  const int b = probe_clusters<L>(res::k_resident_batch<N, R, E, SCHEME>, true);
  return f > 0 && g > 0 ? b : 0;
}

int resident_clusters(int N) {
#define NSGB_RESIDENT_CASE(NN, R, E)                                                  \
  if (N == NN) {                                                                      \
    const int n = probe_instances<NN, R, E, NSGB_SCHEME_CENTRAL>();                   \
    const int m = probe_instances<NN, R, E, NSGB_SCHEME_UPWIND>();                    \
    return n < m ? n : m;                                                             \
  }
  NSGB_RESIDENT(NSGB_RESIDENT_CASE)
#undef NSGB_RESIDENT_CASE
  return 0;
}

cudaError_t launch_resident(int N, const ResidentArgs& a, cudaStream_t st) {
  const bool up = a.scheme == NSGB_SCHEME_UPWIND, grad = a.ckpt != nullptr;
#define NSGB_RESIDENT_CASE(NN, R, E)                                                            \
  if (N == NN) {                                                                                \
    if (grad)                                                                                   \
      return up ? launch_resident_t<NN, R, E, NSGB_SCHEME_UPWIND, true>(a, st)                  \
                : launch_resident_t<NN, R, E, NSGB_SCHEME_CENTRAL, true>(a, st);                \
    return up ? launch_resident_t<NN, R, E, NSGB_SCHEME_UPWIND, false>(a, st)                   \
              : launch_resident_t<NN, R, E, NSGB_SCHEME_CENTRAL, false>(a, st);                 \
  }
  NSGB_RESIDENT(NSGB_RESIDENT_CASE)
#undef NSGB_RESIDENT_CASE
  return cudaErrorInvalidValue;
}

cudaError_t launch_resident_batch(int N, int scheme, const ResidentArgs* tab, int count, cudaStream_t st) {
#define NSGB_RESIDENT_CASE(NN, R, E)                                                                     \
  if (N == NN)                                                                                           \
    return scheme == NSGB_SCHEME_UPWIND ? launch_resident_batch_t<NN, R, E, NSGB_SCHEME_UPWIND>(tab, count, st) \
                                        : launch_resident_batch_t<NN, R, E, NSGB_SCHEME_CENTRAL>(tab, count, st);
  NSGB_RESIDENT(NSGB_RESIDENT_CASE)
#undef NSGB_RESIDENT_CASE
  return cudaErrorInvalidValue;
}

NSGB_BOUNDS_UNIT(resident, 7)

}  // namespace nsgb
