"""The autotuner with fake timings: it comes back to a new plan's shapes, the
adjoint's among them, whenever whole solves are faster there, whatever the
stage timings said (as at the resident kernel's sizes), and it does not apply
shapes cached before the resident kernel."""
import json

import pytest

from ns_solver_jax_differential_distributed_gb300 import _native, autotune

DEFAULT = {"tiles": (32, 8, 16, 4), "radix": (16, 16), "adj": (32, 8)}


class FakePlan:
    def __init__(self, N=64, L=1.0, device="cpu"):
        self.N, self.L, self.device = N, L, device
        self._t, self._r, self._a = DEFAULT["tiles"], DEFAULT["radix"], DEFAULT["adj"]

    def tiles(self):
        return self._t

    def fft_radix(self):
        return self._r

    def adjoint_tiles(self):
        return self._a

    def set_tiles(self, tw=0, th=0, rows=0, cols=0):
        self._t = tuple(new or old for new, old in zip((tw, th, rows, cols), self._t))
        self._a = self._t[:2]  # as nsgb_plan_set_tiles does for a tile

    def set_fft_radix(self, rows=0, cols=0):
        self._r = (rows or self._r[0], cols or self._r[1])

    def set_adjoint_tiles(self, tw=0, th=0):
        self._a = (tw or self._a[0], th or self._a[1])

    @property
    def resident(self):
        return self._t[:2] == (32, 8) and self._r == (16, 16)


@pytest.fixture
def tuner(monkeypatch, tmp_path):
    """tune(winner, adj_winner): a tuning whose stage timings favour these."""
    monkeypatch.setattr(autotune, "_CACHE_PATH", str(tmp_path / "tiles.json"))
    monkeypatch.setattr(autotune.torch.cuda, "get_device_name", lambda d: "fake")
    monkeypatch.setattr(autotune.torch.cuda, "get_device_properties",
                        lambda d: type("P", (), {"multi_processor_count": 152})())
    monkeypatch.setattr(_native, "Plan", FakePlan)
    plan = FakePlan()
    monkeypatch.setattr(_native, "get_plan", lambda N, L, d: plan)

    def tune(winner, adj_winner, whole=1.0, force=True):
        monkeypatch.setattr(_native, "time_stages", lambda *a, **k: {
            "stencil": 1.0 if plan.tiles()[:2] == winner else 2.0, "rows_fwd": 1.0 / plan.fft_radix()[0],
            "rows_inv": 1.0, "cols": 1.0 / plan.fft_radix()[1]})
        monkeypatch.setattr(autotune, "_time_adjoint",
                            lambda *a, **k: 1.0 if plan.adjoint_tiles() == adj_winner else 2.0)
        monkeypatch.setattr(autotune, "_time_rollout", lambda *a, **k: whole if plan.resident else 2.0)
        monkeypatch.setattr(autotune, "_time_gradient", lambda *a, **k: (
            whole if plan.resident and plan.adjoint_tiles() == (32, 8) else 2.0), raising=False)
        return plan, autotune.tune(64, 1.0, "central", "cpu", reps=2, force=force)
    return tune


@pytest.mark.parametrize("winner,adj", [((16, 8), (16, 8)), ((64, 8), (16, 16)), ((32, 8), (16, 8)), ((32, 8), (32, 8))])
def test_default_shapes_win_as_a_whole(tuner, winner, adj):
    for _ in range(2):  # again from the tuned plan
        plan, best = tuner(winner, adj)
        assert plan.tiles()[:2] == (32, 8) and plan.fft_radix() == (16, 16)
        assert plan.adjoint_tiles() == (32, 8) == (best["adj_tw"], best["adj_th"])


def test_tuned_shapes_stay_where_they_win(tuner):
    plan, best = tuner((16, 8), (32, 16), whole=3.0)
    assert plan.tiles()[:2] == (16, 8) and plan.adjoint_tiles() == (32, 16) == (best["adj_tw"], best["adj_th"])


def test_shapes_cached_before_are_tuned_anew(tuner, tmp_path):
    old = {"tw": 16, "th": 8, "rows": 2, "cols": 1, "radix_rows": 16, "radix_cols": 16, "adj_tw": 16, "adj_th": 8}
    (tmp_path / "tiles.json").write_text(json.dumps({"fake|N=64|central": old}))
    assert not autotune.apply_cached(64, 1.0, "central", "cpu")
    plan, _ = tuner((16, 8), (16, 8), force=False)
    assert plan.resident and plan.adjoint_tiles() == (32, 8)
    assert autotune.apply_cached(64, 1.0, "central", "cpu")


@pytest.mark.gpu
@pytest.mark.parametrize("N", [32, 128])
def test_tune_small_grids(cuda_lib, tmp_path, monkeypatch, N):
    import math
    import torch
    from ns_solver_jax_differential_distributed_gb300.workloads import spectral_u0
    monkeypatch.setattr(autotune, "_CACHE_PATH", str(tmp_path / "tiles.json"))
    L, dev = 2 * math.pi, torch.device("cuda")
    plan = _native.get_plan(N, L, dev)
    old = (plan.tiles(), plan.fft_radix(), plan.adjoint_tiles())
    u0 = torch.from_numpy(spectral_u0(N, 8, 1)).cuda()
    th = torch.tensor([0.9, 0.4, 1e-3], device="cuda")
    _, _, u_ref, _ = _native.rollout_grad_raw(u0, th, 20, 1, L, 1e-3, 1e-3, 0)
    try:
        best = autotune.tune(N, L, "central", dev, reps=2, force=True)
        assert plan.tiles() == (best["tw"], best["th"], best["rows"], best["cols"])
        assert plan.fft_radix() == (best["radix_rows"], best["radix_cols"])
        assert plan.adjoint_tiles() == (best["adj_tw"], best["adj_th"])
        assert best["default"] == [*old[0], *old[1], *old[2]]
        _, _, u, _ = _native.rollout_grad_raw(u0, th, 20, 1, L, 1e-3, 1e-3, 0)
        assert float((u - u_ref).norm() / u_ref.norm()) < 1e-5
    finally:
        plan.set_tiles(old[0][0], old[0][1], 2, 1)
        plan.set_fft_radix(*old[1])
        plan.set_tiles(*old[0])
        plan.set_adjoint_tiles(*old[2])
