"""Radix-16 transforms by two threads per butterfly (small grids) round as whole
butterflies do, and the default transforms keep the bits that the solver's
results have had: an upwind gradient is not continuous in the last bits of the
forward states (a cell of |u| below them takes the other one-sided
difference), so another rounding order is another gradient.

The checksums are those of the solver when every transform was whole radix-16
butterflies; inputs are small integers, the same on every machine."""
import math
import zlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

L = 2 * math.pi
# N: CRC-32 of the Poisson solve, the final state and dJ/du0 of five upwind
# steps (checkpoints every two)
CRC = {
    16: (0x71b99cd0, 0x38a79e1b, 0xec9c8b4b),
    32: (0x1d74405c, 0x90d14ecd, 0x1442fe1f),
    64: (0x3cf745ba, 0xf49c8283, 0x5e3f765a),
    128: (0xe5169203, 0x1735c8a2, 0x1b3dedc9),
    256: (0xcc83703f, 0x422887dc, 0xa04bbfe6),
    512: (0x128d9d60, 0x5f127dd0, 0x0b4fb3c9),
    1024: (0xbe5f468c, 0x5c5bb7b4, 0x489734d8),
    2048: (0x5b943bfe, 0x3cf29b9c, 0xbc4518d3),
    4096: (0x82283c54, 0xdb87ea30, 0x05e751bf),
}


@pytest.fixture(scope="module")
def nat(cuda_lib):
    from ns_solver_jax_differential_distributed_gb300 import _native
    return _native


def _ints(N, comps, lo, hi, scale):
    rng = np.random.default_rng(N)
    a = rng.integers(lo, hi, size=(comps, N, N)).astype(np.float32) * np.float32(scale)
    return torch.from_numpy(a).cuda()


def results(nat, N):
    rhs = _ints(N, 1, -8, 9, 1.0)[0]
    u0 = _ints(N, 2, -64, 65, 2.0 ** -6)
    th = torch.tensor([0.75, 0.5, 2.0 ** -10], device="cuda")
    p = nat.op_poisson(rhs - rhs[0, 0], L)
    _, _, u, du0 = nat.rollout_grad_raw(u0, th, 5, 2, L, 2.0 ** -10, 2.0 ** -12, 1, want_du0=True)
    return p, u, du0


@pytest.mark.parametrize("N", sorted(CRC))
def test_default_results_keep_their_bits(nat, N):
    got = tuple(zlib.crc32(t.cpu().numpy().tobytes()) for t in results(nat, N))
    assert got == CRC[N], N


def test_largest_poisson_solve_keeps_its_bits(nat):
    rhs = _ints(8192, 1, -8, 9, 1.0)[0]
    assert zlib.crc32(nat.op_poisson(rhs - rhs[0, 0], L).cpu().numpy().tobytes()) == 0x83e2d3d9


@pytest.mark.parametrize("N,shape", [(128, (0, 64)), (256, (128, 32)), (256, (0, 32)), (256, (128, 0)), (512, (0, 16))])
def test_whole_butterflies_give_the_same_bits(nat, N, shape):
    """CTAs with no room for twice the threads run whole butterflies."""
    plan = nat.get_plan(N, L, torch.device("cuda"))
    assert plan.fft_radix() == (16, 16)
    want = [t.clone() for t in results(nat, N)]
    old = plan.tiles()
    try:
        plan.set_tiles(old[0], old[1], *shape)
        got = results(nat, N)
        torch.cuda.synchronize()
    finally:
        plan.set_tiles(*old)
    for a, b in zip(want, got):
        assert torch.equal(a, b)


def test_persistent_ensemble_equals_default_plans(nat):
    """The persistent launch runs whole radix-16 butterflies at every size."""
    from ns_solver_jax_differential_distributed_gb300 import ensemble
    specs = [ensemble.SolveSpec(N, _ints(N, 2, -64, 65, 2.0 ** -6).cpu().numpy(),
                                np.array([0.75, 0.5, 2.0 ** -10], np.float32), 2.0 ** -10, 2.0 ** -12, scheme, L)
             for N in (64, 128, 256, 512) for scheme in ("central", "upwind")]
    ens = ensemble.Ensemble(specs, steps=9, chunk=4)
    _, up = ens.run_persistent()
    up = [u.clone() for u in up]
    _, ur = ens.run()
    torch.cuda.synchronize()
    for s, a, b in zip(specs, up, ur):
        assert torch.equal(a, b), (s.N, s.scheme)


@pytest.mark.parametrize("N,count", [(256, 17), (512, 5)])
def test_large_batches_give_the_same_bits(nat, N, count):
    """Batches of more than a million cells run whole butterflies."""
    from ns_solver_jax_differential_distributed_gb300 import ensemble
    u0 = _ints(N, 2, -64, 65, 2.0 ** -6)
    th = np.array([0.75, 0.5, 2.0 ** -10], np.float32)
    for members in (1, count):
        ens = ensemble.Ensemble([ensemble.SolveSpec(N, u0.cpu().numpy(), th, 2.0 ** -10, 2.0 ** -12, "upwind", L)] *
                                members, steps=9, chunk=4)
        us = [u.clone() for u in ens.run()[1]]
        if members == 1:
            want = us[0]
        assert all(torch.equal(u, want) for u in us)
