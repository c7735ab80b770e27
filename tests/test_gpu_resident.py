"""The resident kernel (a small grid's whole rollout or gradient in one cluster
launch): its fields equal the four-launch step's bit for bit (a plan whose
tile is not the default runs that one), its objective and theta sensitivities
equal the batched gradients' at the default tile bit for bit, at every size it
has, from one step up, with and without checkpoints and recomputed segments,
in both phases at once or one by one, on concurrent streams and inside a
caller's graph capture."""
import math

import pytest
import torch

from ns_solver_jax_differential_distributed_gb300.workloads import spectral_u0

pytestmark = pytest.mark.gpu

L, NU, DT = 2 * math.pi, 1e-3, 1e-3
SIZES = [32, 64, 128]


@pytest.fixture(scope="module")
def nat(cuda_lib):
    from ns_solver_jax_differential_distributed_gb300 import _native
    return _native


def _inputs(N, n_theta=3, seed=3):
    u0 = torch.from_numpy(spectral_u0(N, min(8, N // 4), seed + N)).cuda()
    return u0, torch.tensor([0.9, 0.4, 2e-3][:n_theta], device="cuda")


def _tiled(nat, N, fn):
    """fn() with the four-launch step: any tile but the resident kernel's."""
    plan = nat.get_plan(N, L, torch.device("cuda"))
    old, old_adj = plan.tiles(), plan.adjoint_tiles()
    assert old[:2] == (32, 8) and old_adj == (32, 8)
    plan.set_tiles(16, 8, old[2], old[3])
    try:
        out = fn()
        torch.cuda.synchronize()
        return out
    finally:
        plan.set_tiles(*old)
        plan.set_adjoint_tiles(*old_adj)


def _grad(nat, u0, th, steps, every, sch, **kw):
    return nat.rollout_grad_raw(u0, th, steps, every, L, NU, DT, sch, want_du0=True, own_workspace=True, **kw)


@pytest.mark.parametrize("N", SIZES)
@pytest.mark.parametrize("scheme", [0, 1])
def test_fields_equal_the_tiled_step(nat, N, scheme):
    u0, th = _inputs(N, 2 if scheme else 3)
    for steps in (1, 2, 3, 40):
        def roll():
            return nat.op_rollout(u0, th, steps, L, NU, DT, scheme, 0.5, 0.1, 1.0, True)
        J, u = roll()
        Jt, ut = _tiled(nat, N, roll)
        assert torch.equal(u, ut), (steps, (u - ut).abs().max().item())
        assert abs(float(J) - float(Jt)) <= 1e-6 * abs(float(Jt)) + 1e-9, (float(J), float(Jt))


@pytest.mark.parametrize("N", SIZES)
@pytest.mark.parametrize("scheme", ["central", "upwind"])
@pytest.mark.parametrize("steps,every", [(1, 1), (2, 2), (9, 1), (9, 4), (13, 12), (13, 50)])
def test_gradients_equal_tiled_and_batched(nat, N, scheme, steps, every):
    from ns_solver_jax_differential_distributed_gb300.ensemble import GradientBatch
    sch = nat.SCHEME_IDS[scheme]
    u0, th = _inputs(N)
    J, g, uf, du = _grad(nat, u0, th, steps, every, sch)
    Jt, gt, uft, dut = _tiled(nat, N, lambda: _grad(nat, u0, th, steps, every, sch))
    assert torch.equal(uf, uft) and torch.equal(du, dut)
    # in slices of five operations: J and dJ/dtheta bit for bit
    gb = GradientBatch()
    sid = gb.add(u0, th, steps, every, L, NU, DT, scheme, want_du0=True)
    gb.run(ops_per_call=5)
    Jb, gbt = gb.result(sid)
    assert torch.equal(J, Jb) and torch.equal(g, gbt) and torch.equal(du, gb.du0(sid)), (g, gbt)


@pytest.mark.parametrize("N", SIZES)
def test_single_steps_equal_the_tiled_step(nat, N):
    u0, th = _inputs(N, 2)
    for sch in (0, 1):
        def step():
            return nat.op_step(u0, th, 0.37, L, NU, DT, sch, 0.5, 0.1, 1.0)
        assert torch.equal(step(), _tiled(nat, N, step))


@pytest.mark.parametrize("N", SIZES)
@pytest.mark.parametrize("ops", [1, 2, 3, 7])
def test_sliced_gradients(nat, N, ops):
    """Slices that end in every kind of operation take up the state of the one
    before, members of unlike schedules, schemes and progress in one launch."""
    from ns_solver_jax_differential_distributed_gb300.ensemble import GradientBatch
    u0, th = _inputs(N)
    want, gb, ids = [], GradientBatch(), []
    for i, (steps, every) in enumerate([(7, 1), (7, 3), (8, 50), (9, 4), (1, 1)]):
        want.append(_grad(nat, u0, th, steps, every, i % 2))
        ids.append(gb.add(u0, th, steps, every, L, NU, DT, ["central", "upwind"][i % 2], want_du0=True,
                          want_u_final=True))
        gb.advance(ops)
    gb.run(ops_per_call=ops)
    for (J, g, uf, du), k in zip(want, ids):
        Jb, gbt = gb.result(k)
        assert torch.equal(J, Jb) and torch.equal(g, gbt)
        assert torch.equal(uf, gb.u_final(k)) and torch.equal(du, gb.du0(k))


def test_sliced_gradients_in_a_crowd(nat):
    """Too many solves for their clusters run tick by tick: a solve that goes
    from one way to the other and back keeps its bits."""
    from ns_solver_jax_differential_distributed_gb300.ensemble import GradientBatch
    u0, th = _inputs(128)
    gb = GradientBatch()
    first = gb.add(u0, th, 31, 5, L, NU, DT, "central", want_du0=True, want_u_final=True)
    gb.advance(13)  # forward steps, alone
    crowd = [gb.add(u0, th, 5, 5, L, NU, DT, "upwind") for _ in range(60)]
    gb.advance(11)  # tick by tick; the crowd of 15 operations goes on
    gb.advance(20)
    gb.run(ops_per_call=9)
    J, g, uf, du = _grad(nat, u0, th, 31, 5, 0)
    Jb, gbt = gb.result(first)
    assert torch.equal(J, Jb) and torch.equal(g, gbt)
    assert torch.equal(uf, gb.u_final(first)) and torch.equal(du, gb.du0(first))
    Jc, gc = _grad(nat, u0, th, 5, 5, 1)[:2]
    for k in crowd:
        Jb, gbt = gb.result(k)
        assert torch.equal(Jc, Jb) and torch.equal(gc, gbt)


def test_phases_one_by_one(nat):
    """Forward then backward (a differentiable rollout) equals one call."""
    u0, th = _inputs(64)
    for every in (1, 6):
        J, g, uf, du = _grad(nat, u0, th, 17, every, 1)
        s = nat.GradSession(u0, th, 17, every, L, NU, DT, 1)
        Js, ufs = s.forward()
        gs, dus = s.backward()
        assert torch.equal(J, Js) and torch.equal(uf, ufs) and torch.equal(g, gs) and torch.equal(du, dus)


def test_streams_and_capture(nat):
    """Solves of all sizes on several streams at once, and one recorded in a
    caller's graph, give the bits of solves one after another."""
    cases = [(N, sch) for N in SIZES for sch in (0, 1)] * 2

    def run(N, sch):
        u0, th = _inputs(N)
        return nat.op_rollout(u0, th, 60, L, NU, DT, sch, 0.5, 0.1, 1.0, True)
    alone = [run(*c) for c in cases]
    torch.cuda.synchronize()
    inputs = [_inputs(N) for N, _ in cases]
    streams = [torch.cuda.Stream() for _ in cases]
    outs = []
    for (N, sch), (u0, th), st in zip(cases, inputs, streams):
        st.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(st):
            outs.append(nat.op_rollout(u0, th, 60, L, NU, DT, sch, 0.5, 0.1, 1.0, True))
    torch.cuda.synchronize()
    for (J, u), (Ja, ua) in zip(outs, alone):
        assert torch.equal(J, Ja) and torch.equal(u, ua)
    N, sch = cases[-1]
    u0, th = inputs[-1]
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        nat.op_rollout(u0, th, 60, L, NU, DT, sch, 0.5, 0.1, 1.0, True)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        J, u = nat.op_rollout(u0, th, 60, L, NU, DT, sch, 0.5, 0.1, 1.0, True)
    J.fill_(0), u.fill_(0)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(J, alone[-1][0]) and torch.equal(u, alone[-1][1])


def test_non_finite_states_stay_non_finite(nat):
    u0, th = _inputs(64)
    u0[0, 5, 7] = float("nan")
    J, u = nat.op_rollout(u0, th, 12, L, NU, DT, 0, 0.5, 0.1, 1.0, True)
    Jt, ut = _tiled(nat, 64, lambda: nat.op_rollout(u0, th, 12, L, NU, DT, 0, 0.5, 0.1, 1.0, True))
    assert torch.isnan(J) and torch.isnan(Jt) and torch.equal(torch.isnan(u), torch.isnan(ut))
