"""The separate launches of small and middle grids, whose default shapes may run
resident instead: tiled stencils and adjoints of one and of four cells per
thread, split and whole transforms, graph chunks and captured gradients,
gradient batches by ticks and explicit forces on wide tiles -- in the
bounds-checking build, between guards, and replayed with inputs changed in
place."""
import ctypes
import math

import pytest
import torch

from tests.test_gpu_bounds_check import _fields, _phys, chk, ctx  # noqa: F401  (fixtures)
from tests.test_gpu_canary import Guarded
from ns_solver_jax_differential_distributed_gb300.workloads import spectral_u0

pytestmark = pytest.mark.gpu

L = 2 * math.pi
# N, stencil tile, adjoint tile, (rows, columns) per CTA, radix
SHAPES = [
    (16, (16, 8), (16, 8), (0, 0), (16, 16)),
    (64, (32, 8), (32, 8), (0, 0), (8, 8)),        # one cell per thread, default tile, separate launches
    (64, (16, 8), (32, 16), (2, 1), (16, 16)),
    (128, (32, 16), (16, 16), (0, 64), (16, 16)),  # whole butterflies in the columns
    (128, (128, 8), (64, 16), (0, 0), (16, 8)),
    (256, (64, 8), (64, 8), (0, 0), (16, 16)),     # defaults
    (256, (64, 16), (128, 8), (128, 32), (16, 16)),
    (512, (128, 8), (128, 8), (0, 0), (16, 16)),
]


def _shape(plan_calls, tile, adj, cta, radix):
    set_tiles, set_radix, set_adj = plan_calls
    set_radix(16, 16)
    set_tiles(tile[0], tile[1], *cta)
    set_radix(*radix)
    set_adj(*adj)


@pytest.mark.parametrize("scheme", ["central", "upwind"])
@pytest.mark.parametrize("N,tile,adj,cta,radix", SHAPES)
def test_in_bounds(ctx, N, tile, adj, cta, radix, scheme):  # noqa: F811
    C, st = ctx.C, ctx.st
    h = ctx.plan(N)
    _shape((lambda *a: ctx.ok(C.nsgb_plan_set_tiles(h, *a)), lambda *a: ctx.ok(C.nsgb_plan_set_fft_radix(h, *a)),
            lambda *a: ctx.ok(C.nsgb_plan_set_adjoint_tiles(h, *a))), tile, adj, cta, radix)
    n = ctypes.c_int(-1)
    ctx.ok(C.nsgb_plan_get_resident(h, 0, st, ctypes.byref(n)))
    assert n.value == 0
    u0, th = _fields(ctx, N)
    ph = _phys(ctx, scheme, 0.2 / N)
    steps, every = 21, 4
    uf, J, g, du0 = ctx.t((2, N, N)), ctx.t(()), ctx.t((3,)), ctx.t((2, N, N))
    ws = ctx.ws(C.nsgb_rollout_workspace_bytes(h, steps))
    ctx.ok(C.nsgb_rollout(h, ctypes.byref(ph), u0.data_ptr(), th.data_ptr(), 3, steps, uf.data_ptr(), J.data_ptr(),
                          ws.data_ptr(), ws.numel(), 1, st))
    gws = ctx.ws(C.nsgb_rollout_grad_workspace_bytes(h, 9, every))
    for _ in range(3):  # eager, captured, replayed
        ctx.ok(C.nsgb_rollout_grad(h, ctypes.byref(ph), u0.data_ptr(), th.data_ptr(), 3, 9, every, 3, J.data_ptr(),
                                   uf.data_ptr(), g.data_ptr(), du0.data_ptr(), gws.data_ptr(), gws.numel(), st))
    assert torch.isfinite(uf).all() and torch.isfinite(g).all() and torch.isfinite(du0).all()


@pytest.mark.parametrize("N", [64, 512, 1024])
def test_explicit_force_in_bounds(ctx, N):  # noqa: F811
    C, st, h = ctx.C, ctx.st, ctx.plan(N)
    u0, _ = _fields(ctx, N)
    force = ctx.t(None, fill=torch.randn(2, N, N, device="cuda"))
    out = ctx.t((2, N, N))
    ws = ctx.ws(C.nsgb_step_workspace_bytes(h))
    for scheme in ("central", "upwind"):
        ph = _phys(ctx, scheme, 0.2 / N)
        ctx.ok(C.nsgb_projector_step(h, ctypes.byref(ph), u0.data_ptr(), force.data_ptr(), out.data_ptr(),
                                     ws.data_ptr(), ws.numel(), st))
        assert torch.isfinite(out).all()


def test_gradient_batch_by_ticks_in_bounds(ctx):  # noqa: F811
    C, st, nat = ctx.C, ctx.st, ctx.nat
    ctx.ok(C.nsgb_plan_set_fft_radix(ctx.plan(64), 8, 16))
    cases = [(64, 9, 4, "upwind"), (256, 5, 2, "central"), (64, 3, 1, "central"), (256, 4, 50, "upwind"),
             (512, 3, 1, "upwind")]
    arr = (nat.GradMember * len(cases))()
    outs = []
    for m, (N, steps, every, scheme) in zip(arr, cases):
        u0, th = _fields(ctx, N)
        h = ctx.plan(N)
        m.plan, m.phys = h.value, _phys(ctx, scheme, 0.2 / N)
        m.u0, m.theta, m.theta_len, m.steps, m.every = u0.data_ptr(), th.data_ptr(), 3, steps, every
        J, g, du0 = ctx.t(()), ctx.t((3,)), ctx.t((2, N, N))
        outs += [J, g, du0]
        m.J, m.u_final, m.dJdtheta, m.dJdu0 = J.data_ptr(), None, g.data_ptr(), du0.data_ptr()
        m.state = ctx.ws(C.nsgb_rollout_grad_workspace_bytes(h, steps, every)).data_ptr()
        m.done_ops = 0
    ops = max(C.nsgb_grad_ops(s, e) for _, s, e, _ in cases)
    ws = ctx.ws(C.nsgb_grad_batch_workspace_bytes(len(cases), ops))
    ctx.ok(C.nsgb_grad_batch_advance(arr, len(cases), ops, ws.data_ptr(), ws.numel(), st))
    assert all(torch.isfinite(x).all() for x in outs)


@pytest.mark.parametrize("N,tile,adj,cta,radix", SHAPES)
def test_guards_and_replay(cuda_lib, N, tile, adj, cta, radix):
    """Buffers between guards; a gradient whose inputs change in place is
    replayed with the new ones."""
    from ns_solver_jax_differential_distributed_gb300 import _native as nat
    lib, st = nat.lib(), torch.cuda.current_stream().cuda_stream
    plan = nat.Plan(N, L, torch.device("cuda", torch.cuda.current_device()))
    _shape((plan.set_tiles, plan.set_fft_radix, plan.set_adjoint_tiles), tile, adj, cta, radix)
    assert plan.resident_clusters(True) == 0
    ph = nat.make_phys(L, 2e-3, 0.2 / N, "upwind")
    u0 = torch.from_numpy(spectral_u0(N, min(8, N // 4), 2)).cuda()
    th = torch.tensor([0.9, 0.4, 2e-3], device="cuda")
    steps, every = 9, 4

    def grad(ws, J, uf, g, du0):
        assert lib.nsgb_rollout_grad(plan.handle, ctypes.byref(ph), u0.data_ptr(), th.data_ptr(), 3, steps, every, 3,
                                     J.ptr(), uf.ptr(), g.ptr(), du0.ptr(), ws.ptr(), ws.nbytes, st) == 0
        torch.cuda.synchronize()
        return [x.inner.clone() for x in (uf, du0)] + [J.inner[:4].clone(), g.inner[:12].clone()]

    def bufs():
        return (Guarded(lib.nsgb_rollout_grad_workspace_bytes(plan.handle, steps, every)), Guarded(256),
                Guarded(8 * N * N), Guarded(256), Guarded(8 * N * N))
    same = bufs()
    first = grad(*same)
    for _ in range(2):  # captured, replayed
        assert all(torch.equal(a, b) for a, b in zip(first, grad(*same)))
    u0.mul_(0.75)
    th.copy_(torch.tensor([1.1, 0.5, 1e-3]))
    replayed = grad(*same)
    other = bufs()
    eager = grad(*other)
    assert all(torch.equal(a, b) for a, b in zip(replayed, eager))
    assert not torch.equal(replayed[0], first[0])
    ws = Guarded(lib.nsgb_rollout_workspace_bytes(plan.handle, 40))
    uf, J = Guarded(8 * N * N), Guarded(256)
    assert lib.nsgb_rollout(plan.handle, ctypes.byref(ph), u0.data_ptr(), th.data_ptr(), 3, 40, uf.ptr(), J.ptr(),
                            ws.ptr(), ws.nbytes, 1, st) == 0
    assert all(b.intact() for b in (*same, *other, ws, uf, J))
