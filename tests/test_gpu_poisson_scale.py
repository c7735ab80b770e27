"""The Poisson multiplier over box lengths: the wavenumber table is scaled to
the range of the kernels' reciprocal (fft::host_wavenumbers), the column
pass's multiplier differs by size (N < 2048, N >= 2048, N = 8192), and radix 8
has its own launch bounds.  Against the spectral solve in float64."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _solve64(rhs, L):
    N = rhs.shape[0]
    k = 2 * math.pi * np.fft.fftfreq(N, L / N)
    kr = 2 * math.pi * np.fft.rfftfreq(N, L / N)
    k2 = k[:, None] ** 2 + kr[None, :] ** 2
    k2[0, 0] = np.inf
    return np.fft.irfft2(-np.fft.rfft2(rhs.astype(np.float64)) / k2, s=(N, N))


@pytest.mark.parametrize("radix", [16, 8])
@pytest.mark.parametrize("N,L", [(16, 1.0), (64, 1e-12), (128, 1e12), (1024, 3.0), (2048, 1e-9), (8192, 2 * math.pi)])
def test_multiplier_over_box_lengths(cuda_lib, N, L, radix):
    from ns_solver_jax_differential_distributed_gb300 import _native
    if radix == 8 and N == 8192:
        pytest.skip("1024 threads per column: beyond the column kernel's block")
    rhs = np.random.default_rng(N).standard_normal((N, N)).astype(np.float32)
    rhs -= rhs.mean()
    plan = _native.Plan(N, L, torch.device("cuda", torch.cuda.current_device()))
    plan.set_tiles(0, 0, 2, 1)
    plan.set_fft_radix(radix, radix)
    t = torch.from_numpy(rhs).cuda()
    p = torch.empty_like(t)
    ws = torch.empty(_native.lib().nsgb_poisson_workspace_bytes(plan.handle), dtype=torch.uint8, device="cuda")
    _native.call("nsgb_poisson", plan.handle, t.data_ptr(), p.data_ptr(), ws.data_ptr(), ws.numel(),
                 _native.stream_of(t.device))
    ref = _solve64(rhs, L)
    err = np.linalg.norm(p.double().cpu().numpy() - ref) / np.linalg.norm(ref)
    assert err < 2e-6 * max(1.0, math.log2(N) / 4), (N, L, radix, err)  # the bound of the other Poisson tests
