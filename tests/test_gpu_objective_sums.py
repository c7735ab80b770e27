"""The objective against float64 sums over the solver's own states and forcing
rows, so only its summation is measured: row bands, the fused row kernel, wide
and narrow tiles and the resident kernel.

Bound, from independent roundings.  Bands: four products and sums in float per
cell group (at most 4 x 2^-25 of it each, 2^-23 of the group's magnitude),
double-float from there; the rms over N^2/4 groups per step is 2^-23 S sqrt(4 /
N^2 / steps), S the summed magnitudes.  Tiles add float sums over up to 256
cells, whose last of eight levels has N^2/256 partials: eight roundings of
2^-25, 2^-22 S sqrt(256 / N^2 / steps).  Four times the rms, plus the rounding
of J itself."""
import math

import numpy as np
import pytest
import torch

from ns_solver_jax_differential_distributed_gb300.workloads import spectral_u0

pytestmark = pytest.mark.gpu

L, NU, STEPS = 2 * math.pi, 1e-3, 3


@pytest.mark.parametrize("N,tile,fused", [
    (64, (32, 8), 0), (64, (16, 8), 0), (256, (64, 8), 0), (512, (128, 8), 0), (256, (32, 8), 0),
    (1024, (1024, 7), 0), (1024, (256, 128), 0), (1024, (1024, 14), 14), (2048, (1024, 14), 0),
    (4096, (1024, 54), 0), (4096, (2048, 54), 54),
])
def test_objective_sums(cuda_lib, N, tile, fused):
    from ns_solver_jax_differential_distributed_gb300 import _native as nat
    plan = nat.get_plan(N, L, torch.device("cuda"))
    dt = float(np.float32(0.1 * L / N))
    u0 = torch.from_numpy(spectral_u0(N, min(8, N // 4), N)).cuda()
    th = torch.tensor([0.9, 0.4, NU], device="cuda")
    old, old_adj, old_fused = plan.tiles(), plan.adjoint_tiles(), plan.fused_rows()
    try:
        plan.set_tiles(tile[0], tile[1], old[2], old[3])
        plan.set_fused(fused)
        J, _ = nat.op_rollout(u0, th, STEPS, L, NU, dt, 0, 0.5, 0.1, 1.0, False)
        J = float(J)
    finally:
        plan.set_fused(old_fused)
        plan.set_tiles(*old)
        plan.set_adjoint_tiles(*old_adj)
    u, want, S = u0, 0.0, 0.0
    for s in range(STEPS):
        t = float(np.float32(s) * np.float32(dt))
        terms = u[0].double() * nat.op_forcing(th, t, N, L, 0.5, 0.1, 1.0)[0].double()
        want += float(terms.sum()) * dt * (L / N) ** 2
        S += float(terms.abs().sum()) * dt * (L / N) ** 2
        u = nat.op_step(u, th, t, L, NU, dt, 0, 0.5, 0.1, 1.0)
    groups = math.sqrt(4 if tile[0] >= 256 else 256) / N / math.sqrt(STEPS)
    unit = 2.0 ** -23 if tile[0] >= 256 else 2.0 ** -22
    assert abs(J - want) <= 4 * unit * S * groups + 2.0 ** -24 * abs(want), (J - want, S, want)
