"""The tiled stencil with four cells per thread (tiles at least 64 wide) gives
the fields of the one-cell body (16 x 8 tiles) bit for bit: one tile across the
periodic grid, several, with and without a pending projection, forcing rows or
an explicit force field, both schemes; the objective to rounding."""
import math

import pytest
import torch

from ns_solver_jax_differential_distributed_gb300.workloads import spectral_u0

pytestmark = pytest.mark.gpu

L, NU, DT = 2 * math.pi, 1e-3, 1e-3


@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("N,tile", [(64, (64, 8)), (64, (64, 16)), (128, (128, 8)), (256, (64, 16)), (256, (128, 8)),
                                    (512, (64, 8))])
def test_wide_tiles_equal_narrow_ones(cuda_lib, N, tile, scheme):
    from ns_solver_jax_differential_distributed_gb300 import _native as nat
    dev = torch.device("cuda")
    u0 = torch.from_numpy(spectral_u0(N, 8, N)).cuda()
    f = torch.randn(2, N, N, device="cuda", generator=torch.Generator(device="cuda").manual_seed(N))
    th = torch.tensor([0.9, 0.4, 2e-3], device="cuda")
    plan = nat.get_plan(N, L, dev)
    old, old_adj = plan.tiles(), plan.adjoint_tiles()

    def run(w, h):
        plan.set_tiles(w, h, old[2], old[3])
        J, u = nat.op_rollout(u0, th, 5, L, NU, DT, scheme, 0.5, 0.1, 1.0, False)
        return float(J), u, nat.op_projector_step(u0, f, L, NU, DT, scheme)
    try:
        Jw, uw, pw = run(*tile)
        Jn, un, pn = run(16, 8)
    finally:
        plan.set_tiles(*old)
        plan.set_adjoint_tiles(*old_adj)
    assert torch.equal(uw, un) and torch.equal(pw, pn)
    assert abs(Jw - Jn) <= 1e-5 * abs(Jn) + 1e-9, (Jw, Jn)


@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("N,tile", [(64, (64, 8)), (64, (64, 16)), (128, (128, 8)), (256, (64, 16)), (256, (128, 8)),
                                    (512, (64, 8))])
def test_wide_adjoint_tiles_equal_narrow_ones(cuda_lib, N, tile, scheme):
    """dJ/du0 bit for bit; dJ/dA and dJ/dB to the rounding of float sums of at
    most eight cells (16 x 8 tiles have one cell per thread), 8 x 2^-24 of the
    summed magnitudes, taken as at most 20 times the larger of the two (dJ/dnu is
    a small difference of large terms, which no such bound holds)."""
    from ns_solver_jax_differential_distributed_gb300 import _native as nat
    dev = torch.device("cuda")
    u0 = torch.from_numpy(spectral_u0(N, 8, N)).cuda()
    th = torch.tensor([0.9, 0.4, 2e-3], device="cuda")
    plan = nat.get_plan(N, L, dev)
    old, old_adj = plan.tiles(), plan.adjoint_tiles()

    def run(w, h):
        plan.set_tiles(16, 8, old[2], old[3])
        plan.set_adjoint_tiles(w, h)
        return nat.rollout_grad_raw(u0, th, 6, 4, L, NU, DT, scheme, want_du0=True, own_workspace=True)
    try:
        _, gw, _, dw = run(*tile)
        _, gn, _, dn = run(16, 8)
    finally:
        plan.set_tiles(*old)
        plan.set_adjoint_tiles(*old_adj)
    assert torch.equal(dw, dn)
    assert (gw - gn)[:2].abs().max().item() <= 20 * 8 * 2.0 ** -24 * gn.abs().max().item(), (gw, gn)
