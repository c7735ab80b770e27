"""Buffers the ABI takes at any float address -- the force field of a
projection step, the initial-state gradient -- give the results of aligned
ones at every kind of launch (resident, tiles of one and of four cells per
thread, row bands)."""
import ctypes
import math

import pytest
import torch

from ns_solver_jax_differential_distributed_gb300.workloads import spectral_u0

pytestmark = pytest.mark.gpu

L, NU, DT = 2 * math.pi, 1e-3, 5e-4
SIZES = [16, 64, 256, 1024]


@pytest.fixture(scope="module")
def nat(cuda_lib):
    from ns_solver_jax_differential_distributed_gb300 import _native
    return _native


def _shifted(x):
    """x (or its shape's zeros) one float past an aligned address."""
    y = torch.zeros(x.numel() + 1, device="cuda")[1:].view(x.shape)
    assert y.data_ptr() % 16 == 4
    return y.copy_(x)


@pytest.mark.parametrize("N", SIZES)
def test_projection_force(nat, N):
    u0 = torch.from_numpy(spectral_u0(N, min(8, N // 4), N)).cuda()
    f = torch.randn(2, N, N, device="cuda")
    plan, ph = nat.get_plan(N, L, torch.device("cuda")), nat.make_phys(L, NU, DT, "upwind", 0.5, 0.1, 1.0)
    ws = torch.empty(nat.lib().nsgb_rollout_workspace_bytes(plan.handle, 1), dtype=torch.uint8, device="cuda")
    outs = []
    for force in (f, _shifted(f)):
        out = torch.empty_like(u0)
        nat.call("nsgb_projector_step", plan.handle, ctypes.byref(ph), nat.ptr(u0), nat.ptr(force), nat.ptr(out),
                 nat.ptr(ws), ws.numel(), nat.stream_of(u0.device))
        outs.append(out)
    assert torch.equal(*outs)


@pytest.mark.parametrize("N", SIZES)
@pytest.mark.parametrize("steps", [1, 4])
def test_initial_state_gradient(nat, N, steps):
    from ns_solver_jax_differential_distributed_gb300.ensemble import GradientBatch
    u0 = torch.from_numpy(spectral_u0(N, min(8, N // 4), N)).cuda()
    th = torch.tensor([0.9, 0.4], device="cuda")
    J, g, _, du = nat.rollout_grad_raw(u0, th, steps, 3, L, NU, DT, 1, want_du0=True)
    s = nat.GradSession(u0, th, steps, 3, L, NU, DT, 1)
    s.forward()
    g2, du2 = torch.empty_like(th), _shifted(torch.zeros_like(u0))
    nat.call("nsgb_rollout_grad", s.plan.handle, ctypes.byref(s.ph), nat.ptr(u0), nat.ptr(th), 2, steps, 3,
             nat.GRAD_BACKWARD, None, None, nat.ptr(g2), nat.ptr(du2), nat.ptr(s.ws), s.ws.numel(),
             nat.stream_of(u0.device))
    assert torch.equal(g, g2) and torch.equal(du, du2)
    gb, du3 = GradientBatch(), _shifted(torch.zeros_like(u0))
    k = gb.add(u0, th, steps, 3, L, NU, DT, 1, want_du0=True)
    gb._solves[k]["member"].dJdu0 = du3.data_ptr()
    gb.run(2)
    assert torch.equal(g, gb.result(k)[1]) and torch.equal(du, du3)
