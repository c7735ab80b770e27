"""Captured graphs stand for any buffers: rollouts and gradients made through
one workspace with other u0, theta and output buffers each time (the first
call eager, the second captured, the rest replayed) equal the eager rollout and
the batched gradient of the same inputs bit for bit."""
import math

import pytest
import torch

from ns_solver_jax_differential_distributed_gb300.workloads import spectral_u0

pytestmark = pytest.mark.gpu

L, NU, DT = 2 * math.pi, 1e-3, 5e-4


@pytest.fixture(scope="module")
def nat(cuda_lib):
    from ns_solver_jax_differential_distributed_gb300 import _native
    return _native


def _inputs(N, k, n_theta):
    u0 = torch.from_numpy(spectral_u0(N, 8, k)).cuda()
    return u0, torch.tensor([0.9 + 0.01 * k, 0.4, 2e-3][:n_theta], device="cuda")


@pytest.mark.parametrize("N", [16, 256])
def test_rollout_replays_with_other_buffers(nat, N):
    keep = []
    for k in range(4):
        u0, th = _inputs(N, k, 3)
        J, u = nat.op_rollout(u0, th, 50, L, NU, DT, 1, 0.5, 0.1, 1.0, True)
        Je, ue = nat.op_rollout(u0, th, 50, L, NU, DT, 1, 0.5, 0.1, 1.0, False)
        assert torch.equal(J, Je) and torch.equal(u, ue), k
        keep.append((u0, th, J, u))  # so that no buffer is used twice


@pytest.mark.parametrize("N", [16, 256])
@pytest.mark.parametrize("steps,every", [(1, 1), (2, 1), (9, 1), (9, 4), (9, 50)])
def test_gradient_replays_with_other_buffers(nat, N, steps, every):
    from ns_solver_jax_differential_distributed_gb300.ensemble import GradientBatch
    keep = []
    for k in range(4):
        u0, th = _inputs(N, k, 2 if every == 4 else 3)
        J, g, uf, du = nat.rollout_grad_raw(u0, th, steps, every, L, NU, DT, 0, want_du0=k != 2)
        gb = GradientBatch()
        sid = gb.add(u0, th, steps, every, L, NU, DT, 0, want_du0=True, want_u_final=True)
        gb.run()
        Jb, gr = gb.result(sid)
        assert torch.equal(J, Jb) and torch.equal(g, gr) and torch.equal(uf, gb.u_final(sid)), k
        assert du is None or torch.equal(du, gb.du0(sid)), k
        keep.append((u0, th, J, g, uf, du))


def test_ensemble_graphs_follow_the_launch_shapes(nat):
    """An ensemble run again on the same buffers after its plan's transforms
    changed captures anew: the bits of solo solves of that plan."""
    from ns_solver_jax_differential_distributed_gb300.ensemble import Ensemble, SolveSpec
    plan, spec = nat.get_plan(64, L, torch.device("cuda")), spectral_u0(64, 8, 5)
    ens = Ensemble([SolveSpec(N=64, u0=spec, theta=(0.9, 0.4), nu=NU, dt=DT, scheme="upwind")], steps=40)
    u0, th = torch.from_numpy(spec).cuda(), torch.tensor([0.9, 0.4], device="cuda")
    old = plan.fft_radix()
    try:
        for radix in ((8, 8), (16, 16), (8, 16)):
            plan.set_fft_radix(*radix)
            u = ens.run()[1][0]
            us = nat.op_rollout(u0, th, 40, L, NU, DT, nat.SCHEME_IDS["upwind"], 0.5, 0.1, 1.0, True)[1]
            assert torch.equal(u, us), radix
    finally:
        plan.set_fft_radix(*old)
