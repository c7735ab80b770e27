"""Which way small grids run, and that the ways agree: the resident launch is
the one taken at the default shapes, its J and dJ/dtheta are those of the tick
path (batched stencil, adjoint and transform kernels at the same tiles) bit for
bit at every size, and both agree with other tiles."""
import math

import pytest
import torch

from ns_solver_jax_differential_distributed_gb300.workloads import spectral_u0

pytestmark = pytest.mark.gpu

L, NU, DT = 2 * math.pi, 1e-3, 1e-3
SIZES = [32, 64, 128]
TURNS = 4  # turns of clusters up to which a batch of gradients runs resident


@pytest.fixture(scope="module")
def nat(cuda_lib):
    from ns_solver_jax_differential_distributed_gb300 import _native
    return _native


def _plan(nat, N):
    return nat.get_plan(N, L, torch.device("cuda"))


def _inputs(N):
    u0 = torch.from_numpy(spectral_u0(N, min(8, N // 4), 3 + N)).cuda()
    return u0, torch.tensor([0.9, 0.4, 2e-3], device="cuda")


def _grad(nat, u0, th, steps, every, sch):
    return nat.rollout_grad_raw(u0, th, steps, every, L, NU, DT, sch, want_du0=True, own_workspace=True)


@pytest.mark.parametrize("N", SIZES)
def test_default_plans_run_resident(nat, N):
    plan = _plan(nat, N)
    assert plan.resident_clusters(False) > 0 and plan.resident_clusters(True) > 0
    old, old_r, old_adj = plan.tiles(), plan.fft_radix(), plan.adjoint_tiles()
    try:
        plan.set_adjoint_tiles(16, 8)
        assert plan.resident_clusters(False) > 0 and plan.resident_clusters(True) == 0
        plan.set_tiles(16, 8, old[2], old[3])
        assert plan.resident_clusters(False) == 0
        plan.set_tiles(*old)
        plan.set_fft_radix(16, 8)
        assert plan.resident_clusters(False) == 0
    finally:
        plan.set_fft_radix(*old_r)
        plan.set_tiles(*old)
        plan.set_adjoint_tiles(*old_adj)


@pytest.mark.parametrize("N", [16, 256])
def test_other_sizes_do_not(nat, N):
    assert _plan(nat, N).resident_clusters() == 0


@pytest.mark.parametrize("scheme", ["central", "upwind"])
@pytest.mark.parametrize("N", SIZES)
def test_tick_path_gives_the_resident_bits(nat, N, scheme):
    from ns_solver_jax_differential_distributed_gb300.ensemble import GradientBatch
    u0, th = _inputs(N)
    cases = [(5, 2), (4, 1), (3, 50)]
    want = [_grad(nat, u0, th, steps, every, nat.SCHEME_IDS[scheme]) for steps, every in cases]
    gb = GradientBatch()
    count = TURNS * _plan(nat, N).resident_clusters(True) + 1
    ids = [gb.add(u0, th, *cases[i % 3], L, NU, DT, scheme, want_du0=True) for i in range(count)]
    gb.advance(64)  # every schedule to its end, in one call: the group stays too large
    assert not gb.pending()
    for i, k in enumerate(ids):
        J, g, _, du = want[i % 3]
        Jb, gbt = gb.result(k)
        assert torch.equal(J, Jb) and torch.equal(g, gbt) and torch.equal(du, gb.du0(k)), i


@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("N", SIZES)
def test_sums_agree_with_other_tiles(nat, N, scheme):
    """dJ/dtheta to two units in the last place (double-float and double sums of
    the same floats), J to eight roundings a tile's float sum takes in either,
    of the summed magnitudes: at most dt dx^2 sum |u_x| a step, the speed growing
    by less than half in 20 steps."""
    u0, th = _inputs(N)
    plan, steps = _plan(nat, N), 20
    J, g, _, _ = _grad(nat, u0, th, steps, 6, scheme)
    old, old_adj = plan.tiles(), plan.adjoint_tiles()
    try:
        plan.set_tiles(16, 8, old[2], old[3])
        Jt, gt, _, _ = _grad(nat, u0, th, steps, 6, scheme)
        torch.cuda.synchronize()
    finally:
        plan.set_tiles(*old)
        plan.set_adjoint_tiles(*old_adj)
    S = 1.5 * steps * DT * (L / N) ** 2 * float(u0[0].abs().sum())
    assert abs(float(J) - float(Jt)) <= 2 * 8 * 2.0 ** -25 * S + 2.0 ** -23 * abs(float(Jt))
    assert ((g - gt).abs() <= 2.0 ** -22 * gt.abs()).all(), (g, gt)
