// FFT-Poisson kernels: the hand-written replacement of SpectralPoissonSolver
// (NS_solver.py:507-527).
//
// The real N x N right-hand side is transformed in two passes:
//   rows (along y, contiguous): two real rows a, b are packed as a + i b, one
//     complex length-N FFT gives both half spectra X_a[k], X_b[k], k=0..N/2.
//     The half spectrum is stored transposed, spec[k][i] (k = 0..N/2, i
//     contiguous): N/2 + 1 rows of N complex values.
//   columns (along x): each spec[k] row is transformed, multiplied by
//     -1/|k|^2 (0 at k = 0; NS_solver.py:521, 525-526), transformed back and
//     written in place.  Every ky column has its own row -- in particular the
//     DC and Nyquist columns are never packed together -- so a field that is
//     constant along y keeps exactly zero spectrum at ky != 0, as the
//     reference's C2C transforms do (its zero-state runs stay exactly
//     y-independent, which the upwind study at the diffusive stability limit
//     relies on).
//   rows again: the inverse two-for-one C2R transform writes p.
// All scale factors (the 1/2 of the two-for-one split and the 1/N^2 of ifft2)
// are powers of two folded into the spectral multiplier, so they round
// exactly.
#include "nsgb_fft_bodies.cuh"

namespace nsgb {

// ---------------------------------------------------------------- kernels --
// The column pass is bound by the FP32 pipe's operand bandwidth (a fused
// multiply-add of three different registers issues at 0.64 of the rate of one
// with two) and by shared memory; two CTAs of 256 threads per SM already
// saturate both, so registers matter more than warps: the radix-16 kernel is
// bounded to 80 registers (768 threads per SM), where the multipliers of a
// thread overlap and little spills.  Times of the pass in the step, with 64
// registers and a CUDA reciprocal before: N = 4096 46.4 -> 40.9 us, 1024 11.4 ->
// 8.4 us.  N = 8192 has CTAs of 512 threads and needs two of them per SM (213 us,
// against 240 us for one with 128 registers); so do threads of 8 values, whose
// registers allow it.
template <int N, int E>
constexpr bool cols_two() {
  return E == 8 || N >= 8192;
}
template <int N, int E, int R>
__device__ __forceinline__ int cols_thread() {
  if constexpr (E < R)
    return fft::split_index<N>(threadIdx.x);
  else
    return threadIdx.x;
}
template <int N, int E, int R>
__global__ void __launch_bounds__(1024) k_rows_fwd(const float* __restrict__ rhs, float2* __restrict__ spec,
                                                   const float2* __restrict__ tw) {
  rows_fwd_body<N, E, R>(rhs, spec, tw, threadIdx.x, threadIdx.y, blockDim.y, blockIdx.x);
}
template <int N, int E, int R>
__global__ void __launch_bounds__(cols_two<N, E>() ? 512 : 768, cols_two<N, E>() ? 2 : 1) k_cols(float2* __restrict__ spec,
                                                              const float2* __restrict__ tw,
                                                              const float* __restrict__ k2, float scale) {
  cols_body<N, E, R>(spec, tw, k2, scale, cols_thread<N, E, R>(), threadIdx.y, blockDim.y, blockIdx.x);
}
template <int N, int E, int R>
__global__ void __launch_bounds__(1024) k_rows_inv(const float2* __restrict__ spec, float* __restrict__ p,
                                                   const float2* __restrict__ tw) {
  rows_inv_body<N, E, R>(spec, p, tw, threadIdx.x, threadIdx.y, blockDim.y, blockIdx.x);
}
// Ensemble variants: blockIdx.y selects the member.
template <int N, int E, int R>
__global__ void __launch_bounds__(1024) k_rows_fwd_b(const SolveDev* __restrict__ sv,
                                                     const float2* __restrict__ tw) {
  const FftPtrs f = sv[blockIdx.y].fft;
  rows_fwd_body<N, E, R>(f.rhs, f.spec, tw, threadIdx.x, threadIdx.y, blockDim.y, blockIdx.x);
}
template <int N, int E, int R>
__global__ void __launch_bounds__(cols_two<N, E>() ? 512 : 768, cols_two<N, E>() ? 2 : 1) k_cols_b(const SolveDev* __restrict__ sv,
                                                                const float2* __restrict__ tw,
                                                                const float* __restrict__ k2, float scale) {
  cols_body<N, E, R>(sv[blockIdx.y].fft.spec, tw, k2, scale, cols_thread<N, E, R>(), threadIdx.y, blockDim.y, blockIdx.x);
}
template <int N, int E, int R>
__global__ void __launch_bounds__(1024) k_rows_inv_b(const SolveDev* __restrict__ sv,
                                                     const float2* __restrict__ tw) {
  const FftPtrs f = sv[blockIdx.y].fft;
  rows_inv_body<N, E, R>(f.spec, f.p, tw, threadIdx.x, threadIdx.y, blockDim.y, blockIdx.x);
}

// ------------------------------------------------------------- launchers --
// Radix-16 passes by threads of 8 values (fft::half_butterfly) where a step
// waits for the transforms' latency: the same bits from twice the threads.  Step
// with whole / split butterflies, us: N = 16 8.7 / 7.5, 256 11.6 / 10.3 (rows
// alone or columns alone 10.9), 512, columns only, 14.5 / 13.9; from N = 1024 on
// it waits for shared memory.  So do batches of a million cells and more:
// N = 256 x 8 15.6 / 14.2, x 16 20.4 / 20.2, x 20 23.0 / 23.1, x 30 29.3 / 30.0;
// 512 x 3 19.7 / 19.3, x 4 21.4 / 21.5, x 6 26.9 / 27.5, x 11 39.7 / 41.0; but not
// of smaller grids: 128 x 80 33.0 / 31.0, 64 x 300 35.2 / 32.2.  CTAs too large
// for twice the threads keep whole butterflies.
constexpr int kSplitRowsN = 256, kSplitColsN = 512;
template <int N>
static bool split_pays(int count) {
  return N < 256 || (size_t)count * N * N <= (size_t)1 << 20;
}
template <int N>
static bool rows_split(const FftLaunch& L, int count) {
  return N <= kSplitRowsN && L.radix_rows == 16 && L.rows_per_cta / 2 * (N / 8) <= 1024 && split_pays<N>(count);
}
template <int N>
static bool cols_split(const FftLaunch& L, int count) {
  return N <= kSplitColsN && L.radix_cols == 16 && L.cols_per_cta * (N / 8) <= 512 && split_pays<N>(count);
}

template <int N, int R>
static const float2* radix_tables(const FftLaunch& L) {
  return L.tw + (R == 8 ? fft::tw8_offset(N) : 0);
}

template <int N, int E, int R>
static cudaError_t stage_rows_fwd(const FftLaunch& L, const SolveDev* sv, int count, cudaStream_t st) {
  constexpr int T = N / E;
  const int P = L.rows_per_cta / 2;
  const size_t smem = (size_t)P * pair_stride<N>() * sizeof(float2);
  if (smem > 48 * 1024) {
    const cudaError_t e = raise_smem_limit(sv ? (const void*)k_rows_fwd_b<N, E, R> : (const void*)k_rows_fwd<N, E, R>);
    if (e != cudaSuccess) return e;
  }
  if (sv)
    k_rows_fwd_b<N, E, R><<<dim3(N / (2 * P), count), dim3(T, P), smem, st>>>(sv, radix_tables<N, R>(L));
  else
    k_rows_fwd<N, E, R><<<N / (2 * P), dim3(T, P), smem, st>>>(L.rhs, L.spec, radix_tables<N, R>(L));
  return cudaGetLastError();
}

template <int N, int E, int R>
static cudaError_t stage_cols(const FftLaunch& L, const SolveDev* sv, int count, cudaStream_t st) {
  constexpr int T = N / E;
  const int KB = L.cols_per_cta;
  const size_t smem = (size_t)KB * pair_stride<N>() * sizeof(float2);
  if (smem > 48 * 1024) {
    const cudaError_t e = raise_smem_limit(sv ? (const void*)k_cols_b<N, E, R> : (const void*)k_cols<N, E, R>);
    if (e != cudaSuccess) return e;
  }
  if (sv)
    k_cols_b<N, E, R><<<dim3((N / 2) / KB + 1, count), dim3(T, KB), smem, st>>>(sv, radix_tables<N, R>(L), L.k2,
                                                                            L.scale);
  else
    k_cols<N, E, R><<<(N / 2) / KB + 1, dim3(T, KB), smem, st>>>(L.spec, radix_tables<N, R>(L), L.k2, L.scale);
  return cudaGetLastError();
}

template <int N, int E, int R>
static cudaError_t stage_rows_inv(const FftLaunch& L, const SolveDev* sv, int count, cudaStream_t st) {
  constexpr int T = N / E;
  const int P = L.rows_per_cta / 2;
  const size_t smem = (size_t)P * pair_stride<N>() * sizeof(float2);
  if (smem > 48 * 1024) {
    const cudaError_t e = raise_smem_limit(sv ? (const void*)k_rows_inv_b<N, E, R> : (const void*)k_rows_inv<N, E, R>);
    if (e != cudaSuccess) return e;
  }
  if (sv)
    k_rows_inv_b<N, E, R><<<dim3(N / (2 * P), count), dim3(T, P), smem, st>>>(sv, radix_tables<N, R>(L));
  else
    k_rows_inv<N, E, R><<<N / (2 * P), dim3(T, P), smem, st>>>(L.spec, L.p, radix_tables<N, R>(L));
  return cudaGetLastError();
}

template <int N>
static cudaError_t launch_poisson_fft(const FftLaunch& L, const SolveDev* sv, int count, cudaStream_t st) {
  constexpr int E = fft::ept(N);
  const int r = rows_split<N>(L, count) ? 1 : L.radix_rows == 8 ? 2 : 0;
  const int c = cols_split<N>(L, count) ? 1 : L.radix_cols == 8 ? 2 : 0;
  cudaError_t e = cudaSuccess;
  if (sv || L.rhs) {
    if constexpr (N <= kSplitRowsN)
      if (r == 1) e = stage_rows_fwd<N, 8, 16>(L, sv, count, st);
    if (r == 2) e = stage_rows_fwd<N, 8, 8>(L, sv, count, st);
    if (r == 0) e = stage_rows_fwd<N, E, 16>(L, sv, count, st);
  }
  if (e == cudaSuccess && (sv || L.do_cols)) {
    if constexpr (N <= kSplitColsN)
      if (c == 1) e = stage_cols<N, 8, 16>(L, sv, count, st);
    if (c == 2) e = stage_cols<N, 8, 8>(L, sv, count, st);
    if (c == 0) e = stage_cols<N, E, 16>(L, sv, count, st);
  }
  if (e == cudaSuccess && (sv || L.p)) {
    if constexpr (N <= kSplitRowsN)
      if (r == 1) e = stage_rows_inv<N, 8, 16>(L, sv, count, st);
    if (r == 2) e = stage_rows_inv<N, 8, 8>(L, sv, count, st);
    if (r == 0) e = stage_rows_inv<N, E, 16>(L, sv, count, st);
  }
  return e;
}

size_t fft_rows_smem_bytes(int N, int rows_per_cta) {
  return (size_t)(rows_per_cta / 2) * (padlen(N) + 2) * sizeof(float2);
}
size_t fft_cols_smem_bytes(int N, int cols_per_cta) {
  return (size_t)cols_per_cta * (padlen(N) + 2) * sizeof(float2);
}

static cudaError_t dispatch(int N, const FftLaunch& L, const SolveDev* sv, int count, cudaStream_t st) {
  switch (N) {
    case 16: return launch_poisson_fft<16>(L, sv, count, st);
    case 32: return launch_poisson_fft<32>(L, sv, count, st);
    case 64: return launch_poisson_fft<64>(L, sv, count, st);
    case 128: return launch_poisson_fft<128>(L, sv, count, st);
    case 256: return launch_poisson_fft<256>(L, sv, count, st);
    case 512: return launch_poisson_fft<512>(L, sv, count, st);
    case 1024: return launch_poisson_fft<1024>(L, sv, count, st);
    case 2048: return launch_poisson_fft<2048>(L, sv, count, st);
    case 4096: return launch_poisson_fft<4096>(L, sv, count, st);
    case 8192: return launch_poisson_fft<8192>(L, sv, count, st);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t poisson_fft(int N, const FftLaunch& L, cudaStream_t st) { return dispatch(N, L, nullptr, 0, st); }

cudaError_t poisson_fft_batch(int N, const FftLaunch& L, const SolveDev* solves, int count, cudaStream_t st) {
  return dispatch(N, L, solves, count, st);
}

NSGB_BOUNDS_UNIT(fft, 2)

}  // namespace nsgb
