"""All three theta sensitivities of the wide adjoint tiles (four cells per
thread) against one-cell tiles: each cell's terms are the same floats, summed
in double-float or double from the first cell on, whose error of some 2^-44 of
the summed magnitudes stays below a float's rounding even for dJ/dnu, a small
difference of large terms; so the results agree to two units in the last
place."""
import math

import pytest
import torch

from ns_solver_jax_differential_distributed_gb300.workloads import spectral_u0

pytestmark = pytest.mark.gpu

L, NU, DT = 2 * math.pi, 1e-3, 1e-3


@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("N,tile", [(64, (64, 8)), (64, (64, 16)), (128, (128, 8)), (256, (64, 8)), (512, (128, 8))])
def test_wide_tiles_sum_theta_as_one_cell_tiles(cuda_lib, N, tile, scheme):
    from ns_solver_jax_differential_distributed_gb300 import _native as nat
    u0 = torch.from_numpy(spectral_u0(N, 8, N)).cuda()
    th = torch.tensor([0.9, 0.4, 2e-3], device="cuda")
    plan = nat.get_plan(N, L, torch.device("cuda"))
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
    assert ((gw - gn).abs() <= 2.0 ** -22 * gn.abs()).all(), (gw, gn)
