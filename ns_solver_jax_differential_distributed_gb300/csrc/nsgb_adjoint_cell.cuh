// Per-cell arithmetic of the adjoint step (derived in nsgb_adjoint.cu), shared
// by its tiled and row-streaming kernels and the resident kernel.
#pragma once

#include "nsgb_internal.h"

namespace nsgb {

// lambda_s of one cell from mu and u at the cell (o) and its four
// neighbours n = (i+1, j), s = (i-1, j), e = (i, j+1), w = (i, j-1);
// fterm = jscale * f_x(i).  All adjoint kernels use it, so they give the same
// bits.
struct AdjNbr {
  float o, n, s, e, w;
};
template <int SCHEME>
__device__ __forceinline__ void adjoint_cell(const AdjNbr& Mx, const AdjNbr& My, const AdjNbr& Ux, const AdjNbr& Uy,
                                             float cL, float cA, float fterm, float& lx, float& ly) {
  const float mx = Mx.o, my = My.o;
  const float lmx = fmaf(-4.0f, mx, (Mx.s + Mx.n) + (Mx.e + Mx.w));
  const float lmy = fmaf(-4.0f, my, (My.s + My.n) + (My.e + My.w));
  // at = h (A'(u)^T mu): the difference quotients' 1/h is folded into cA
  float atx, aty;
  if (SCHEME == NSGB_SCHEME_CENTRAL) {
    const float gxux = Ux.n - Ux.s, gxuy = Uy.n - Uy.s;
    const float gyux = Ux.e - Ux.w, gyuy = Uy.e - Uy.w;
    atx = -fmaf(mx, gxux, my * gxuy) + (fmaf(Mx.n, Ux.n, -Mx.s * Ux.s) + fmaf(Mx.e, Uy.e, -Mx.w * Uy.w));
    aty = -fmaf(mx, gyux, my * gyuy) + (fmaf(My.n, Ux.n, -My.s * Ux.s) + fmaf(My.e, Uy.e, -My.w * Uy.w));
  } else {
    const float uxo = Ux.o, uyo = Uy.o;
    const bool mxo = uxo >= 0.f, myo = uyo >= 0.f;
    // one-sided differences of u at o (the forward's dfx, dfy)
    const float dxux = mxo ? uxo - Ux.s : Ux.n - uxo;
    const float dxuy = mxo ? uyo - Uy.s : Uy.n - uyo;
    const float dyux = myo ? uxo - Ux.w : Ux.e - uxo;
    const float dyuy = myo ? uyo - Uy.w : Uy.e - uyo;
    atx = -fmaf(mx, dxux, my * dxuy);
    aty = -fmaf(mx, dyux, my * dyuy);
    // transposed one-sided operators applied to mu_c u_x (x) and mu_c u_y (y)
    const bool mxn = Ux.n >= 0.f, mxs = Ux.s >= 0.f;
    const bool mye = Uy.e >= 0.f, myw = Uy.w >= 0.f;
    auto dxt = [&](const AdjNbr& mu) {
      return (mxo ? mu.o * uxo : -mu.o * uxo) - (mxn ? mu.n * Ux.n : 0.f) + (mxs ? 0.f : mu.s * Ux.s);
    };
    auto dyt = [&](const AdjNbr& mu) {
      return (myo ? mu.o * uyo : -mu.o * uyo) - (mye ? mu.e * Uy.e : 0.f) + (myw ? 0.f : mu.w * Uy.w);
    };
    atx -= dxt(Mx) + dyt(Mx);
    aty -= dxt(My) + dyt(My);
  }
  lx = mx + fmaf(cL, lmx, fmaf(cA, atx, fterm));
  ly = my + fmaf(cL, lmy, cA * aty);
}

// dfx/dA and dfx/dB of row i at time t (the forcing's sensitivities to theta).
__device__ __forceinline__ void forcing_theta_grad(int i, const ForcingRow& fr, float A, float B, float t,
                                                   const StepConsts& c, float& dA, float& dB) {
  float fx, dmu, dsig;
  forcing_fx_grad(i, fr, c, fx, dmu, dsig);
  const float twopi = 6.28318548202514648f;
  const float argA = fmul(fmul(twopi, A), t);
  const float argB = fmul(fmul(twopi, B), t);
  const float cb = cosf(argB);
  // d mu/dA = cos(2 pi A t) 2 pi t ;  d sig/dB = -2 cos sin (2 pi B t) 2 pi t
  dA = dmu * (cosf(argA) * twopi * t);
  dB = dsig * (-2.0f * cb * sinf(argB) * twopi * t);
}

}  // namespace nsgb
