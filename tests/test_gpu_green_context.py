"""Small grids on a stream that has a share of the device's SMs (a green
context): a resident launch's cluster of up to 16 CTAs may have no place there,
so solves run as separate launches, with the same bits."""
import ctypes
import math

import pytest
import torch

from ns_solver_jax_differential_distributed_gb300.workloads import spectral_u0

pytestmark = pytest.mark.gpu

L, NU, DT = 2 * math.pi, 1e-3, 1e-3


@pytest.fixture(scope="module")
def nat(cuda_lib):
    from ns_solver_jax_differential_distributed_gb300 import _native
    return _native


def _grad(nat, u0, th, steps, every, sch):
    return nat.rollout_grad_raw(u0, th, steps, every, L, NU, DT, sch, want_du0=True, own_workspace=True)


def _green_stream(sms):
    """(stream, closer) of a green context of about `sms` SMs, or None."""
    cu = ctypes.CDLL("libcuda.so.1")
    if not hasattr(cu, "cuGreenCtxStreamCreate"):
        return None
    dev = ctypes.c_int()
    res, part, rest = (ctypes.create_string_buffer(1024) for _ in range(3))
    n, desc, ctx, stream = ctypes.c_uint(1), ctypes.c_void_p(), ctypes.c_void_p(), ctypes.c_void_p()
    SM, DEFAULT_STREAM, NON_BLOCKING = 1, 1, 1
    ok = (cu.cuDeviceGet(ctypes.byref(dev), torch.cuda.current_device()) == 0
          and cu.cuDeviceGetDevResource(dev, res, SM) == 0
          and cu.cuDevSmResourceSplitByCount(part, ctypes.byref(n), res, rest, 0, sms) == 0
          and cu.cuDevResourceGenerateDesc(ctypes.byref(desc), part, 1) == 0
          and cu.cuGreenCtxCreate(ctypes.byref(ctx), desc, dev, DEFAULT_STREAM) == 0
          and cu.cuGreenCtxStreamCreate(ctypes.byref(stream), ctx, NON_BLOCKING, 0) == 0)
    if not ok:
        return None

    def close():
        cu.cuStreamDestroy_v2(stream)
        cu.cuGreenCtxDestroy(ctx)
    return stream.value, close


@pytest.mark.parametrize("N", [32, 128])
def test_streams_of_a_share_of_the_device_run_separate_launches(nat, N):
    u0 = torch.from_numpy(spectral_u0(N, min(8, N // 4), 3 + N)).cuda()
    th = torch.tensor([0.9, 0.4, 2e-3], device="cuda")
    plan = nat.get_plan(N, L, torch.device("cuda"))
    assert plan.resident_clusters(True) > 0
    J, g, uf, du = _grad(nat, u0, th, 7, 3, 1)
    Jr, ur = nat.op_rollout(u0, th, 40, L, NU, DT, 0, 0.5, 0.1, 1.0, True)
    st = nat.op_step(u0, th, 0.3, L, NU, DT, 0, 0.5, 0.1, 1.0)
    torch.cuda.synchronize()
    made = _green_stream(16)
    if made is None:
        pytest.skip("no green contexts here")
    handle, close = made
    try:
        assert plan.resident_clusters(True, handle) == 0
        with torch.cuda.stream(torch.cuda.ExternalStream(handle)):
            Jg, gg, ufg, dug = _grad(nat, u0, th, 7, 3, 1)
            Jrg, urg = nat.op_rollout(u0, th, 40, L, NU, DT, 0, 0.5, 0.1, 1.0, True)
            stg = nat.op_step(u0, th, 0.3, L, NU, DT, 0, 0.5, 0.1, 1.0)
        torch.cuda.synchronize()
    finally:
        torch.cuda.synchronize()
        close()
    for a, b in ((J, Jg), (g, gg), (uf, ufg), (du, dug), (Jr, Jrg), (ur, urg), (st, stg)):
        assert torch.equal(a, b)
